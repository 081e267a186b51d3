// What device.cuh needs to compile as host C++: the rounding intrinsics, as
// single operations that the compiler cannot fuse (device_source.py puts
// host forms in the place of the two approximate instructions).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <cfloat>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>
#include <tuple>
#include <vector>
#undef __device__
#undef __forceinline__
#undef __noinline__
#define __device__
#define __forceinline__ inline
#define __noinline__
static inline float one_op(float r) { asm("" : "+x"(r)); return r; }
static inline float __fmul_rn(float a, float b) { return one_op(a * b); }
static inline float __fadd_rn(float a, float b) { return one_op(a + b); }
static inline float __fsub_rn(float a, float b) { return one_op(a - b); }
static inline float __fdiv_rn(float a, float b) { return one_op(a / b); }
static inline float __fsqrt_rn(float a) { return one_op(std::sqrt(a)); }
template <class To, class From> static inline To bits(From f) { To t; std::memcpy(&t, &f, 4); return t; }
static inline float __int_as_float(int x) { return bits<float>(x); }
static inline float __uint_as_float(unsigned x) { return bits<float>(x); }
static inline int __float_as_int(float x) { return bits<int>(x); }
static inline unsigned __float_as_uint(float x) { return bits<unsigned>(x); }
static inline int __float2int_rz(float x) { return (int)x; }
static inline float rsqrtf(float x) { return 1.f / std::sqrt(x); }
static inline unsigned __umulhi(unsigned a, unsigned b) { return (unsigned)(((unsigned long long)a * b) >> 32); }
static inline void sincospif(float x, float* s, float* c) { *s = std::sin(x * 3.14159265f); *c = std::cos(x * 3.14159265f); }
template <class T> static inline T __ldg(const T* p) { return *p; }
// any reciprocal within 2 ulp, the bound the kernels count on
static inline float some_reciprocal(float x)
{
    const float r = 1.f / x;
    const unsigned h = bits<unsigned>(x) * 2654435761u >> 16;
    return std::isfinite(r) && r != 0.f ? bits<float>(bits<int>(r) + (int)(h % 5u) - 2) : r;
}
