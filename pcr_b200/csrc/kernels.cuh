// Wavefront stage kernels.  One iteration of the persistent wavefront is
//   schedule -> paths -> extend -> shadow -> status
// k_paths (paths.cuh) takes the queued paths, whose ray has been traced, and
// new camera paths, and follows each until it ends or its next ray has a
// triangle mesh to walk: then the path waits in the other queue, where
// k_extend walks it, as k_shadow does the shadow rays that meet the mesh.
// Paths on scenes without a mesh never wait, those of staged requests
// (Engine::route) after every vertex.  Every kernel loops over a device-side
// count, so a whole iteration (and several in a row) can be captured in one
// CUDA graph with no host round trip.  No kernel waits on another block or on
// the host: there is no spin anywhere.
#pragma once

#include <cub/block/block_scan.cuh>

#include "device.cuh"

namespace pcr {

struct EngineParams {
    int fill;          // refill target (paths in flight)
    int chunk;         // per-request issue chunk per refill
    int regen_every;   // refill cadence in iterations
    int wave;          // paths worth an iteration however long they are (0: no bound but `fill`)
};

// ------------------------------------------------------------------ schedule
// One block.  Decides how many new camera paths each active request gets
// this iteration: first up to `chunk` each (round-robin fairness), then the
// remaining free slots oldest-first.  Requests whose paths never wait
// (kReqFlat) share `fill` paths per iteration; the others share what the
// waiting paths leave of `fill`.
constexpr int kSchedThreads = 1024;

struct Share {
    long long mine, before, all;  // this thread's paths, those of the positions before it, everyone's
};

// Splits `slots` over the threads' remaining paths `rem`.
template <typename Scan>
__device__ __forceinline__ Share share_slots(typename Scan::TempStorage& tmp, long long rem, long long chunk, long long slots)
{
    // pass 1: up to chunk each, in active order
    long long w1 = rem < chunk ? rem : chunk;
    long long ex1, tot1;
    Scan(tmp).ExclusiveSum(w1, ex1, tot1);
    __syncthreads();
    long long g1 = slots - ex1;
    g1 = g1 < 0 ? 0 : (g1 > w1 ? w1 : g1);
    const long long left = slots - (tot1 < slots ? tot1 : slots);
    const long long rem2 = rem - g1;
    long long ex2, tot2;
    Scan(tmp).ExclusiveSum(rem2, ex2, tot2);
    __syncthreads();
    long long g2 = left - ex2;
    g2 = g2 < 0 ? 0 : (g2 > rem2 ? rem2 : g2);
    Share s;
    s.mine = g1 + g2;
    Scan(tmp).ExclusiveSum(s.mine, s.before, s.all);
    __syncthreads();
    return s;
}

// Paths are followed to their end, or to the mesh, within the iteration they
// start in, so their number alone does not bound an iteration, and cancels,
// admissions and results are seen between blocks of iterations.  The new paths
// of an iteration are cut to kVerticesPerSlot possible vertices per place of
// `fill`, with p.wave paths at least; where that cuts, every request gets an
// equal share first.  64: an iteration that is cut is mostly the tail of its
// few longest paths (1 M places, 6.3 M paths of depth 64 in a closed room,
// 16 shadow rays, with 16 / 32 / 64 vertices per place: 182 / 152 / 133 ms, a
// cancel seen after 24 / 52 / 123 ms; 290 ms when an iteration was one vertex).
constexpr long long kVerticesPerSlot = 64;
template <typename Scan>
__device__ __forceinline__ void limit_work(typename Scan::TempStorage& tmp, Share& s, long long cost, const EngineParams& p)
{
    __shared__ int s_most;
    if (p.wave <= 0) return;
    if (threadIdx.x == 0) s_most = 0;
    __syncthreads();
    const long long work = s.mine * cost;
    if (work > 0) atomicMax(&s_most, (int)cost);
    long long before, all;
    Scan(tmp).ExclusiveSum(work, before, all);
    __syncthreads();
    const long long wave = p.wave < p.fill ? p.wave : p.fill, least = wave * s_most;
    const long long budget = least > kVerticesPerSlot * p.fill ? least : kVerticesPerSlot * p.fill;
    if (all <= budget) return;
    const int n = __syncthreads_count(work > 0);
    const Share part = share_slots<Scan>(tmp, work, budget / n, budget);
    if (work > 0) s.mine = part.mine / cost;
    Scan(tmp).ExclusiveSum(s.mine, s.before, s.all);
    __syncthreads();
}

__global__ void __launch_bounds__(kSchedThreads) k_schedule(EngineView E, const EngineParams* P, int cur)
{
    typedef cub::BlockScan<long long, kSchedThreads, cub::BLOCK_SCAN_WARP_SCANS> Scan;
    __shared__ typename Scan::TempStorage tmp;
    Counters* C = E.cnt;
    const int tid = threadIdx.x;
    const int n_act = *E.n_active;
    int qn = C->queue_n[cur];
    if (qn > E.queue_cap) {  // never expected: k_paths guards every append
        qn = E.queue_cap;
        if (tid == 0) atomicOr(&C->status, 4);
    }
    const EngineParams p = *P;
    long long free_slots = (long long)p.fill - qn;
    if (free_slots < 0) free_slots = 0;
    if (p.regen_every > 1 && (C->iter % p.regen_every) != 0 && qn > 0) free_slots = 0;

    int slot = -1;
    bool flat = false;
    long long rem = 0, cost = 0;  // vertices that a path may have in the iteration, where that is more than one
    if (tid < n_act) {
        slot = E.active[tid];
        if (E.round_state[slot] == 1) {
            // an adaptive round ended last iteration and k_round kept
            // round_cnt pixels: open the next round, or finish the request
            DRequest& R = const_cast<DRequest&>(E.reqs[slot]);
            // a cancelled request opens no further round
            const int kept = (R.flags & kReqCancelled) ? 0 : E.round_cnt[slot];
            E.round_cnt[slot] = 0;
            E.round_state[slot] = 0;
            R.round_base = R.total;
            R.round += 1;
            R.total += (long long)kept * R.spp;
            if (kept == 0) {
                unsigned long long t;
                asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
                E.done_flag[slot] = 1;
                E.t_done[slot] = t;
            }
        }
        rem = E.reqs[slot].total - (long long)E.issued[slot];
        if (rem < 0) rem = 0;
        flat = (E.reqs[slot].flags & kReqFlat) != 0;
        if (!(E.reqs[slot].flags & kReqStaged)) cost = E.reqs[slot].depth;
    }
    Share q = {0, 0, 0}, w = {0, 0, 0};
    if (__syncthreads_or(!flat && rem > 0)) {
        q = share_slots<Scan>(tmp, flat ? 0 : rem, p.chunk, free_slots);
        limit_work<Scan>(tmp, q, cost, p);
    }
    if (__syncthreads_or(flat && rem > 0)) {
        w = share_slots<Scan>(tmp, flat ? rem : 0, p.chunk, p.fill);
        limit_work<Scan>(tmp, w, cost, p);
    }
    if (tid < n_act) {
        const long long g = q.mine + w.mine;
        E.give_base[tid] = (int)q.before;
        E.path_base[tid] = (int)w.before;
        E.give_start[tid] = (long long)E.issued[slot];
        if (g > 0) {
            if (E.issued[slot] == 0ull) {
                unsigned long long t;
                asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
                E.t_first[slot] = t;
            }
            E.issued[slot] += (unsigned long long)g;
        }
        E.outstanding[slot] = 0;  // k_extend counts the paths that wait
    }
    if (tid == 0) {
        C->n_rounds = 0;  // k_round of the last iteration has read the list
        C->new_n = (int)q.all;
        C->queue_n[cur] = qn;
        C->queue_n[cur ^ 1] = 0;
        C->shadow_n = 0;
        C->path_n = (int)w.all;
        C->next[0] = C->next[1] = C->next[2] = 0;
        C->paths += (unsigned long long)(q.all + w.all);
    }
}

// ------------------------------------------------------------------ spectral weights
// Per-channel XYZ weights of a path's wavelengths: w_k = cmf(lam_k) *
// (700-400)/yBarIntegral / N, so the pixel contribution of per-channel
// radiance c is sum_k c_k w_k = sum_k singleLambdaXYZ(lam_k, c_k) / N
// (code/Renderer.cpp:254-257, code/Includes/CIE.h:140-159).  Computed once
// per path at raygen; RGB mode passes the channels through.
struct XyzWeights {
    float3 w[4];
};

// The colour-matching functions tabulated every 1/kCmfPerNm nm over
// [kCmfLo, kCmfHi] (380..720 nm, wider than the 400..700 nm the hero
// wavelengths span) and read back with linear interpolation, so raygen
// evaluates four wavelengths per path without 28 exponentials.  Entries are
// the Wyman-Sloan-Shirley lobes (code/Includes/CIE.h:27-53, their float
// constants) evaluated in double at the exact grid wavelength, then rounded
// once; the lookup's fraction comes from one fused multiply-add of the exact
// difference lambda - kCmfLo, so the only error left is the interpolation's,
// below 2e-6 of each value.  In [kCmfXLo, kCmfXHi] x-bar's lobes cancel and
// the reference's own float evaluation (singleLambdaXYZ) carries rounding of
// up to 3e-5 of the result, which no smooth table follows; there x-bar is
// evaluated with the reference's float operations instead (xyz_weights).  Against the
// reference the result then stays below 1e-5 relative (1e-7 absolute near
// zero) over 380..720 nm.
constexpr float kCmfLo = 380.f, kCmfHi = 720.f, kCmfXLo = 495.f, kCmfXHi = 508.f;
constexpr int kCmfPerNm = 80;
constexpr int kCmfEntries = 340 * kCmfPerNm + 1;  // (kCmfHi - kCmfLo) * kCmfPerNm + 1
__device__ __forceinline__ double wyman_d(double l, float mu, float s1, float s2)
{
    const double t = (l < (double)mu) ? (l - (double)mu) * (double)s1 : (l - (double)mu) * (double)s2;
    return exp(-0.5 * t * t);
}
__global__ void k_cmf_table(float4* table)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kCmfEntries; i += gridDim.x * blockDim.x) {
        const double l = (double)kCmfLo + (double)i / (double)kCmfPerNm;
        const double x = (double)0.362f * wyman_d(l, 442.0f, 0.0624f, 0.0374f) +
                         (double)1.056f * wyman_d(l, 599.8f, 0.0264f, 0.0323f) -
                         (double)0.065f * wyman_d(l, 501.1f, 0.0490f, 0.0382f);
        const double y = (double)0.821f * wyman_d(l, 568.8f, 0.0213f, 0.0247f) +
                         (double)0.286f * wyman_d(l, 530.9f, 0.0613f, 0.0322f);
        const double z = (double)1.217f * wyman_d(l, 437.0f, 0.0845f, 0.0278f) +
                         (double)0.681f * wyman_d(l, 459.0f, 0.0385f, 0.0725f);
        table[i] = make_float4((float)x, (float)y, (float)z, 0.f);
    }
}
__device__ __forceinline__ float3 cmf_lut(const float4* __restrict__ table, float l)
{
    // l - kCmfLo is exact for l in [190, 760] (Sterbenz); fmaf rounds
    // d * kCmfPerNm - i once, so f carries no error from the product
    const float d = l - kCmfLo;
    const int i = min(max((int)floorf(d * (float)kCmfPerNm), 0), kCmfEntries - 2);
    const float f = fmaf(d, (float)kCmfPerNm, -(float)i);
    const float4 a = table[i], b = table[i + 1];
    return make_float3(a.x + (b.x - a.x) * f, a.y + (b.y - a.y) * f, a.z + (b.z - a.z) * f);
}
__device__ __forceinline__ bool in_cmf_x_window(float l) { return l >= kCmfXLo && l <= kCmfXHi; }

__device__ __noinline__ XyzWeights xyz_weights(bool spectral, const float* lam, int nch, float wN, float xyz_scale,
                                               const float4* cmf_table)
{
    XyzWeights W;
    if (!spectral) {
        W.w[0] = make_float3(1.f, 0.f, 0.f);
        W.w[1] = make_float3(0.f, 1.f, 0.f);
        W.w[2] = make_float3(0.f, 0.f, 1.f);
        W.w[3] = make_float3(0.f, 0.f, 0.f);
        return W;
    }
    const float s = xyz_scale * wN;
    int kx = -1;  // the wavelength in x-bar's exact window, if any
    for (int k = 0; k < 4; k++) {
        if (k < nch) {
            float3 c = cmf_lut(cmf_table, lam[k]);
            if (in_cmf_x_window(lam[k])) kx = k;
            W.w[k] = make_float3(c.x * s, c.y * s, c.z * s);
        } else {
            W.w[k] = make_float3(0.f, 0.f, 0.f);
        }
    }
    // a path's wavelengths lie 300/N nm apart (75 at N = 4) and the window is
    // 13 nm wide, so at most one of them is in it: one exact evaluation per
    // lane, outside the loop, keeps a warp from running it up to four times
    if (kx >= 0) {
        const float x = cmf_x(lam[kx]) * s;
        if (kx == 0) W.w[0].x = x;
        else if (kx == 1) W.w[1].x = x;
        else if (kx == 2) W.w[2].x = x;
        else W.w[3].x = x;
    }
    return W;
}
// Packed layout of the weights in the path queue (see PathQueue::w).
__device__ __forceinline__ void store_weights(const PathQueue& Q, int pos, const XyzWeights& W)
{
    Q.w[0][pos] = make_float4(W.w[0].x, W.w[0].y, W.w[0].z, W.w[1].x);
    Q.w[1][pos] = make_float4(W.w[1].y, W.w[1].z, W.w[2].x, W.w[2].y);
    Q.w[2][pos] = make_float4(W.w[2].z, W.w[3].x, W.w[3].y, W.w[3].z);
}
__device__ __forceinline__ XyzWeights load_weights(const PathQueue& Q, int pos)
{
    const float4 a = Q.w[0][pos], b = Q.w[1][pos], c = Q.w[2][pos];
    XyzWeights W;
    W.w[0] = make_float3(a.x, a.y, a.z);
    W.w[1] = make_float3(a.w, b.x, b.y);
    W.w[2] = make_float3(b.z, b.w, c.x);
    W.w[3] = make_float3(c.y, c.z, c.w);
    return W;
}
__device__ __forceinline__ XyzWeights rgb_weights()
{
    XyzWeights W;
    W.w[0] = make_float3(1.f, 0.f, 0.f);
    W.w[1] = make_float3(0.f, 1.f, 0.f);
    W.w[2] = make_float3(0.f, 0.f, 1.f);
    W.w[3] = make_float3(0.f, 0.f, 0.f);
    return W;
}

__device__ __forceinline__ float3 apply_xyz(const XyzWeights& W, float4 c)
{
    float3 s = make_float3(0.f, 0.f, 0.f);
    s.x += c.x * W.w[0].x; s.y += c.x * W.w[0].y; s.z += c.x * W.w[0].z;
    s.x += c.y * W.w[1].x; s.y += c.y * W.w[1].y; s.z += c.y * W.w[1].z;
    s.x += c.z * W.w[2].x; s.y += c.z * W.w[2].y; s.z += c.z * W.w[2].z;
    s.x += c.w * W.w[3].x; s.y += c.w * W.w[3].y; s.z += c.w * W.w[3].z;
    return s;
}

__device__ __forceinline__ float comp4(float4 v, int k) { return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w; }
__device__ __forceinline__ float4 mul4(float4 a, float4 b) { return make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w); }
__device__ __forceinline__ float4 rgb4(float4 c) { return make_float4(c.x, c.y, c.z, 0.f); }

// A material spectrum at the four carried wavelengths (Material::albedoAt /
// emissiveAt, code/Includes/Material.h:92-101).  Kept out of line: one copy
// of the sigmoid / table code instead of one per call site keeps k_paths'
// instruction footprint small.
__device__ __noinline__ float4 spec4(const DMaterial& m, int emissive, float4 lam)
{
    if (m.flags & (emissive ? kMatTabE : kMatTabA)) {
        const float* table = emissive ? m.tabE : m.tabA;
        return make_float4(spectrum_lerp<true>(table, lam.x), spectrum_lerp<true>(table, lam.y),
                           spectrum_lerp<true>(table, lam.z), spectrum_lerp<true>(table, lam.w));
    }
    const float4 fit = emissive ? m.efit : m.afit;
    const float4 v = make_float4(sigmoid_fit<true>(fit, lam.x), sigmoid_fit<true>(fit, lam.y), sigmoid_fit<true>(fit, lam.z),
                                 sigmoid_fit<true>(fit, lam.w));
    return emissive ? v : make_float4(v.x > 1.f ? 1.f : v.x, v.y > 1.f ? 1.f : v.y, v.z > 1.f ? 1.f : v.z, v.w > 1.f ? 1.f : v.w);
}

// ------------------------------------------------------------------ raygen
// Camera rays for the new paths (code/Renderer.cpp:190-239): pixel centre,
// jitter when aa > 1, hero wavelength and its stratified companions.
struct CameraPath {
    uint32_t pixel, sample;
    float3 d;
    float lambda0;
};

// 300 nm / n for n = 1..4 wavelengths (all exact)
__device__ __forceinline__ float wavelength_stride(int n)
{
    return n == 4 ? 75.f : (n == 3 ? 100.f : (n == 2 ? 150.f : 300.f));
}

// Pixel (returned) and local sample of a path number past 2^32.
__device__ __noinline__ uint32_t split_path(long long path, uint32_t per_pixel, uint32_t& q)
{
    const long long px = path / (long long)per_pixel;
    q = (uint32_t)(path - px * (long long)per_pixel);
    return (uint32_t)px;
}

// Path number `path` of request R; W receives the XYZ weights of a spectral
// path's wavelengths (left alone otherwise).
__device__ __forceinline__ CameraPath camera_path(const EngineView& E, const DRequest& R, long long path, float xyz_scale,
                                                  XyzWeights& W)
{
    CameraPath p;
    const bool adaptive = R.flags & kReqAdaptive;
    // adaptive round r: spp paths for each pixel still in the round's list
    const long long at = adaptive ? path - R.round_base : path;
    const uint32_t per = (uint32_t)(adaptive ? R.spp : R.paths_per_pixel);
    uint32_t q;
    if ((at >> 32) == 0) {
        p.pixel = (uint32_t)at / per;
        q = (uint32_t)at - p.pixel * per;
    } else {
        p.pixel = split_path(at, per, q);
    }
    if (adaptive) {
        // sample numbers r*spp.. as in the non-adaptive order
        p.pixel = (uint32_t)R.act[R.round & 1][p.pixel];
        p.sample = (uint32_t)R.round * (uint32_t)R.spp + q;
    } else if (R.local_spp == R.spp) {
        p.sample = q;
    } else {  // local sample q of a sample range
        const uint32_t round = q / (uint32_t)R.local_spp;
        p.sample = round * (uint32_t)(R.spp - R.local_spp) + (uint32_t)R.sample0 + q;
    }
    const int py = (int)(p.pixel / (uint32_t)R.width), px = (int)p.pixel - py * R.width;
    float jx = 0.f, jy = 0.f;
    if (R.aa > 1) {
        float4 j = rand4(R, p.pixel, p.sample / (uint32_t)R.spp, 0, 254u, 0);
        jx = j.x - 0.5f;
        jy = j.y - 0.5f;
    }
    float x = ((2 * (px + 0.5f + jx) / (float)R.width) - 1) * R.scale * R.aspect;
    float y = -((2 * (py + 0.5f + jy) / (float)R.height) - 1) * R.scale;
    float inv = rsqrtf(x * x + y * y + 1.f);
    p.d = make_float3(x * inv, y * inv, -inv);
    p.lambda0 = 0.f;
    if (R.flags & kReqSpectral) {
        float4 u = rand4(R, p.pixel, p.sample, 0, 255u, 0);
        p.lambda0 = 400.f + u.x * 300.f;
        const int nch = R.hero;
        // hero wavelength and its stratified companions (code/Renderer.cpp:227-239)
        float lam[4];
        const float span = 300.f, stride_l = wavelength_stride(nch);
        lam[0] = p.lambda0;
#pragma unroll
        for (int k = 1; k < 4; k++) {
            float l = lam[0] + stride_l * k;
            if (l > 700.f) l -= span;
            lam[k] = k < nch ? l : lam[0];
        }
        W = xyz_weights(true, lam, nch, 1.f / (float)nch, xyz_scale, E.cmf_table);
        const DScene& S = E.scenes[R.scene];
        if (S.emit_mat >= 0) {
            // emission of the scene's only emissive material, folded in
            const float4 e = spec4(E.mats[S.mat_base + S.emit_mat], 1, make_float4(lam[0], lam[1], lam[2], lam[3]));
            W.w[0] = f3mul(W.w[0], e.x);
            W.w[1] = f3mul(W.w[1], e.y);
            W.w[2] = f3mul(W.w[2], e.z);
            W.w[3] = f3mul(W.w[3], e.w);
        }
    }
    return p;
}

// Brings the next grid-stride record's line into L2 while this one is
// processed (no register cost; the record is read again when its turn comes).
__device__ __forceinline__ void prefetch_l2(const void* p)
{
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// ------------------------------------------------------------------ extend
// The trace kernels are latency-bound (dependent IEEE arithmetic, scattered
// scene loads): their register budget is capped at 64 per thread (blocks of
// up to 256, 4 per SM) so 32 or more warps stay resident per SM.
#ifndef PCR_TRACE_MIN_BLOCKS
#define PCR_TRACE_MIN_BLOCKS 4
#endif
#ifndef PCR_SHADOW_MIN_BLOCKS
#define PCR_SHADOW_MIN_BLOCKS PCR_TRACE_MIN_BLOCKS
#endif
constexpr int kTraceMaxBlock = 256, kTraceMinBlocks = PCR_TRACE_MIN_BLOCKS, kShadowMinBlocks = PCR_SHADOW_MIN_BLOCKS;

// Closest hit of the paths that wait in queue q: the BVH walk, bounded by the
// analytic hit.  Every ray here meets the mesh's box (others never wait), so
// warps walk with all lanes from the start.  kStaged: some of them are of
// staged requests, for which the analytic part is found here too.  Also counts
// each request's waiting paths.
template <bool kStaged>
__global__ void __launch_bounds__(kTraceMaxBlock, kTraceMinBlocks) k_extend(EngineView E, int q)
{
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int n = min(E.cnt->queue_n[q], E.queue_cap);
    const PathQueue Q = E.q[q];
    const int stride = gridDim.x * blockDim.x;
    for (int base = blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < n; base += stride) {
        const int i = base + lane, nx = i + stride;
        if (nx < n) { prefetch_l2(Q.o + nx); prefetch_l2(Q.d + nx); prefetch_l2(Q.id + nx); prefetch_l2(Q.hit + nx); }
        int slot = -1;
        if (i < n) {
            const int4 id = Q.id[i];
            slot = id.x;
            const DScene& S = E.scenes[id.w];
            const float3 o = xyz(Q.o[i]), d = xyz(Q.d[i]);
            const bool full = kStaged && (E.reqs[slot].flags & kReqStaged);
            float t = full ? FLT_MAX : Q.hit[i].x, u = 0.f, v = 0.f;
            uint32_t prim = kPrimNone;
            if (full) prim = scene_analytic<true>(S, o, d, t);
            const int tri = bvh4_closest<false>(S, o, d, t, u, v, nullptr);
            if (tri >= 0) prim = kPrimTri | (uint32_t)tri;
            if (full || tri >= 0) Q.hit[i] = make_float4(t, __uint_as_float(prim), u, v);
        }
        const unsigned same = __match_any_sync(kAll, slot);
        if (slot >= 0 && lane == __ffs(same) - 1)
            atomicAdd((unsigned long long*)&E.outstanding[slot], (unsigned long long)__popc(same));
        if (base >= n - stride) break;
    }
}

// ------------------------------------------------------------------ helpers

// Adds one sample's XYZ to a pixel's FP64 accumulator (device memory) with
// global-space reductions, which return nothing to the thread.
__device__ __forceinline__ void red_add(double* a, double v)
{
    asm volatile("red.global.add.f64 [%0], %1;" ::"l"(__cvta_generic_to_global(a)), "d"(v) : "memory");
}
__device__ __forceinline__ void add_xyz(double* acc, float3 c)
{
    red_add(acc + 0, (double)c.x);
    red_add(acc + 1, (double)c.y);
    red_add(acc + 2, (double)c.z);
}

// ------------------------------------------------------------------ shading steps
// The steps of one path vertex (code/Renderer.cpp:656-889 with samples = 1,
// the GPU's paths-per-pixel estimator).

// Wavelengths carried by a path (code/Renderer.cpp:227-239).
__device__ __forceinline__ float4 path_wavelengths(float l0, int single, int nHero)
{
    if (single) return make_float4(l0, l0, l0, l0);
    const float span = 300.f, stride_l = wavelength_stride(nHero);
    float l1 = l0 + stride_l * 1, l2 = l0 + stride_l * 2, l3 = l0 + stride_l * 3;
    if (l1 > 700.f) l1 -= span;
    if (l2 > 700.f) l2 -= span;
    if (l3 > 700.f) l3 -= span;
    return make_float4(l0, 1 < nHero ? l1 : l0, 2 < nHero ? l2 : l0, 3 < nHero ? l3 : l0);
}

// Hit point, outward normal (not yet turned towards the ray) and material
// (scene-local) of a hit.  kMesh: the scene may hold triangles.
struct Surface {
    float3 hit, N;
    int mi;
};
template <bool kMesh>
__device__ __forceinline__ Surface surface_at(const DScene& S, uint32_t prim, float t, float hu, float hv, float3 o, float3 d)
{
    Surface r;
    r.hit = make_float3(o.x + d.x * t, o.y + d.y * t, o.z + d.z * t);
    const uint32_t kind = prim & kPrimKindMask, pidx = prim & kPrimIndexMask;
    if (kind == kPrimSphere) {
        const float4 cr = S.spheres[pidx].c_r;
        float3 v = make_float3(r.hit.x - cr.x, r.hit.y - cr.y, r.hit.z - cr.z);
        r.N = f3mul(v, rsqrtf(f3dot(v, v)));
        r.mi = S.spheres[pidx].mat.x;
    } else if (!kMesh || kind == kPrimPlane) {
        const float4 na = S.planes[pidx].n_emit;
        r.N = make_float3(na.x, na.y, na.z);
        r.mi = __float_as_int(S.planes[pidx].o_mat.w);
    } else {
        const DTri& tr = S.tris[pidx];
        r.mi = __float_as_int(tr.e1_mat.w);
        if (__float_as_int(tr.e2_flags.w) & 1) {
            const float4 n0 = S.tri_n[pidx * 3], n1 = S.tri_n[pidx * 3 + 1], n2 = S.tri_n[pidx * 3 + 2];
            const float w = 1.f - hu - hv;
            float3 in = make_float3(n0.x * w + n1.x * hu + n2.x * hv, n0.y * w + n1.y * hu + n2.y * hv,
                                    n0.z * w + n1.z * hu + n2.z * hv);
            r.N = f3mul(in, rsqrtf(f3dot(in, in)));
        } else {
            r.N = xyz(S.tri_flatn[pidx]);
        }
    }
    return r;
}

// Mirror direction and origin.
__device__ __forceinline__ void reflect_at(float3 hit, float3 N, float3 d, float cosI, float3& o2, float3& d2)
{
    d2 = f3add(d, f3mul(N, 2.f * cosI));
    o2 = f3add(hit, f3mul(N, 1e-3f));
}

// Optics::dielectricBounce (code/Includes/Optics.h:59-82) with the coin u;
// returns whether the path reflects.  Its roundings are written out: left to
// the compiler, they would depend on the code around the call, and a path's
// directions with them.
__device__ __forceinline__ bool dielectric_bounce(float3 hit, float3 N, float3 d, float cosI, bool entering, float ior,
                                                  float u, float3& bo, float3& bd)
{
    const float n1 = entering ? 1.f : ior, n2 = entering ? ior : 1.f;
    const float eta = n1 / n2;
    const float e2 = __fmul_rn(eta, eta), s2 = fmaf(-cosI, cosI, 1.f);
    const float sinT2 = __fmul_rn(e2, s2);
    bool refl = sinT2 >= 1.f;
    if (!refl) {
        float F0 = (n1 - n2) / (n1 + n2);
        F0 *= F0;
        const float F = fmaf(1.f - F0, __powf(1.f - cosI, 5.f), F0);
        refl = u < F;
    }
    if (refl) {
        reflect_at(hit, N, d, cosI, bo, bd);
    } else {
        const float cosT = sqrtf(fmaf(-e2, s2, 1.f));
        const float k = fmaf(eta, cosI, -cosT);
        bd = make_float3(fmaf(d.x, eta, __fmul_rn(N.x, k)), fmaf(d.y, eta, __fmul_rn(N.y, k)),
                         fmaf(d.z, eta, __fmul_rn(N.z, k)));
        bo = f3sub(hit, f3mul(N, 1e-3f));
    }
    return refl;
}

// Optics::cauchyIor, for paths whose wavelengths may bend differently.
__device__ __forceinline__ float ior_at(const DMaterial& m, bool dispersion, float lambda)
{
    float ior = m.ior;
    if (dispersion) ior = m.ior + m.cauchyB * 1e4f / (lambda * lambda);
    return ior;
}

// Light sample s of a diffuse vertex: point, light normal and material.
struct LightSample {
    float3 P, Nl;
    int mat;
};
__device__ __forceinline__ LightSample sample_light(const DScene& S, const DRequest& R, uint32_t pixel, uint32_t sample,
                                                    uint32_t fork, uint32_t bounce, uint32_t s)
{
    LightSample r;
    const float4 rr = rand4(R, pixel, sample, fork, bounce, 1u + s);
    int pick = 0;
    if (S.n_lights > 1) {
        const float target = rr.x * S.total_light_area;
        float cum = 0.f;
        for (int l = 0; l < S.n_lights; l++) {
            cum += S.lights[l].total_area;
            if (target <= cum) { pick = l; break; }
        }
    }
    const DLight& L = S.lights[pick];
    if (L.kind == 0) {
        r.P = make_float3(L.o_mat.x + L.u.x * rr.y + L.v.x * rr.z, L.o_mat.y + L.u.y * rr.y + L.v.y * rr.z,
                          L.o_mat.z + L.u.z * rr.y + L.v.z * rr.z);
        r.Nl = xyz(L.n);
        r.mat = __float_as_int(L.o_mat.w);
    } else {
        const float4 r2 = rand4(R, pixel, sample, fork, bounce, 1000u + s);
        const float rt = rr.y * L.total_area;
        const float* cum = S.light_cum + L.tri_offset;
        int lo = 0, hi = L.tri_count;
        while (lo < hi) { int mid = (lo + hi) >> 1; if (cum[mid] < rt) lo = mid + 1; else hi = mid; }
        const int ti = lo < L.tri_count - 1 ? lo : L.tri_count - 1;
        const DTri& lt = S.light_tris[L.tri_offset + ti];
        float a = rr.z, b = r2.x;
        if (a + b > 1.f) { a = 1.f - a; b = 1.f - b; }
        r.P = make_float3(lt.v0_id.x + lt.e1_mat.x * a + lt.e2_flags.x * b,
                          lt.v0_id.y + lt.e1_mat.y * a + lt.e2_flags.y * b,
                          lt.v0_id.z + lt.e1_mat.z * a + lt.e2_flags.z * b);
        r.Nl = xyz(S.light_flatn[L.tri_offset + ti]);
        r.mat = __float_as_int(lt.e1_mat.w);
    }
    return r;
}

// Shadow segment from the shading point hc (which the lit-facing branch
// moves, code/Renderer.cpp:857, mutating operator+) to a light sample, and
// its geometry term G (0 when the sample adds nothing).
struct ShadowSegment {
    float3 so, wi;
    float d2, cosT, cosL, G;
};
__device__ __forceinline__ ShadowSegment shadow_segment(const LightSample& L, float3 N, float3& hc)
{
    ShadowSegment g;
    const float3 Li = f3sub(L.P, hc);
    g.d2 = f3dot(Li, Li);
    const float inv_d = rsqrtf(g.d2);
    g.wi = f3mul(Li, inv_d);
    g.cosT = fmaxf(0.f, f3dot(g.wi, N));
    if (g.cosT <= 0.f) g.so = f3sub(hc, f3mul(N, 1e-3f));
    else { hc = f3add(hc, f3mul(N, 1e-3f)); g.so = hc; }
    g.cosL = fmaxf(0.f, -f3dot(L.Nl, Li));
    g.G = g.cosT * g.cosL * (inv_d * inv_d);
    return g;
}
// The sample's factor: geometry term times the MIS weight when asked for.
__device__ __forceinline__ float shadow_factor(const DScene& S, const DRequest& R, const ShadowSegment& g)
{
    const float inv_pi = 1.f / 3.14159274f;
    float w = 1.f;
    if ((R.flags & kReqMIS) && g.cosL > 1e-6f) {
        const float pL = g.d2 / (g.cosL * S.total_light_area), pB = g.cosT * inv_pi;
        w = (pL * pL) / (pL * pL + pB * pB);
    }
    return g.G * w;
}

// Continuation of a diffuse vertex: Russian roulette and the cosine
// hemisphere.  Returns whether the path goes on; nd its direction and
// rr_scale its throughput factor.
__device__ __forceinline__ bool diffuse_bounce(const DRequest& R, uint32_t pixel, uint32_t sample, uint32_t fork, int bounce,
                                               bool last, bool spectral, float4 al, float3 N, float3& nd, float& rr_scale)
{
    const float4 r0 = rand4(R, pixel, sample, fork, (uint32_t)bounce, 0u);
    bool survive = !last;
    rr_scale = 1.f;
    if (survive && (R.flags & kReqRussian) && bounce >= 1) {
        float pr = spectral ? al.x : fmaxf(fmaxf(al.x, al.y), al.z);
        pr = fminf(0.95f, fmaxf(0.05f, pr));
        if (r0.w > pr) survive = false;
        else rr_scale = 1.f / pr;
    }
    if (survive) {
        float r1 = r0.x, r2 = r0.y;
        if ((R.flags & kReqStratified) && bounce == 0 && R.strata > 0) {
            const int sin_ = (int)sample % R.spp;
            const int sx = sin_ % R.strata, sy = (sin_ / R.strata) % R.strata;
            r1 = ((float)sx + r0.x) / (float)R.strata;
            r2 = ((float)sy + r0.y) / (float)R.strata;
        }
        nd = hemisphere(N, r1, r2);
    }
    return survive;
}

// ------------------------------------------------------------------ shadow
// The BVH part of the shadow test (code/Renderer.cpp:852-860) for the shadow
// rays that meet the mesh's box and that k_paths found lit otherwise: blocked
// by a hit in front of the bound and closer than lightDist2 - 1e-3 (compared
// in double, as the reference's double literal promotes it).  Lit samples add
// their XYZ contribution to the pixel's FP64 accumulator.  kStaged: some are of
// staged requests, which have the whole test here.
template <bool kStaged>
__global__ void __launch_bounds__(kTraceMaxBlock, kShadowMinBlocks) k_shadow(EngineView E)
{
    const int n = min(E.cnt->shadow_n, E.shadow_cap);
    const ShadowQueue SQ = E.sq;
    const int stride = gridDim.x * blockDim.x;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const int nx = i + stride;
        if (nx < n) { prefetch_l2(SQ.o + nx); prefetch_l2(SQ.d + nx); prefetch_l2(SQ.c + nx); if (!kStaged) prefetch_l2(SQ.bound + nx); }
        const float4 o = SQ.o[i];
        if (o.w >= 0.f) {
            const DScene& S = E.scenes[__float_as_int(SQ.c[i].w) >> 16];
            const float3 d = xyz(SQ.d[i]);
            float t, u, v;
            int query = kShadowWalk;
            if (kStaged && (E.reqs[__float_as_int(SQ.c[i].w) & 0xFFFF].flags & kReqStaged)) query = scene_blocked_analytic<true, true>(S, E.mats, xyz(o), d, o.w, t);
            else t = SQ.bound[i];
            if (query == kShadowWalk && bvh4_closest<false, true>(S, xyz(o), d, t, u, v, nullptr, (double)o.w - 1e-3) == -2)
                query = kShadowBlocked;
            if (query != kShadowBlocked) {
                // read after the walk, so that it holds no registers across it
                const float4 c = SQ.c[i];
                const int pixel = __float_as_int(SQ.d[i].w);
                add_xyz(E.reqs[__float_as_int(c.w) & 0xFFFF].accum + (size_t)pixel * 3, make_float3(c.x, c.y, c.z));
            }
        }
        if (i >= n - stride) break;
    }
}

// ------------------------------------------------------------------ status
// End of iteration: marks requests whose paths are all issued and retired.
__global__ void k_status(EngineView E, int next)
{
    Counters* C = E.cnt;
    const int n_act = *E.n_active;
    __shared__ int s_busy;
    if (threadIdx.x == 0) s_busy = 0;
    __syncthreads();
    unsigned long long now;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
    for (int r = threadIdx.x; r < n_act; r += blockDim.x) {
        const int slot = E.active[r];
        if (E.done_flag[slot]) continue;
        if (E.round_state[slot]) { s_busy = 1; continue; }
        const bool all_issued = (long long)E.issued[slot] >= E.reqs[slot].total;
        if (all_issued && E.outstanding[slot] == 0) {
            // a cancelled adaptive request opens no further round
            if ((E.reqs[slot].flags & (kReqAdaptive | kReqCancelled)) == kReqAdaptive) {
                E.round_state[slot] = 1;  // k_round, then the next k_schedule
                E.round_list[atomicAdd(&C->n_rounds, 1)] = slot;
                s_busy = 1;
            } else {
                E.done_flag[slot] = 1;
                E.t_done[slot] = now;
            }
        } else {
            s_busy = 1;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        C->idle = (s_busy == 0 && C->queue_n[next] == 0) ? 1 : 0;
        C->iter++;
    }
}

// ------------------------------------------------------------------ adaptive rounds
// End of an adaptive aa round (the GPU backends' per-pixel Welford loop,
// code/Gpu/Opengl/OpenglRenderer.cpp:1288-1383): each pixel of the round
// takes the mean of its spp paths, updates its running mean / M2, and stops
// after 4 or more rounds once every channel's relative variance
// M2/(taken-1) / (mean^2 + 0.01) is below 0.05, or after aa rounds.
// Stopped pixels write their mean to the accumulator (resolved with weight
// 1); the others reset it and move to the next round's list.
__global__ void k_round(EngineView E)
{
    const int n_rounds = E.cnt->n_rounds;
    const int lane = threadIdx.x & 31;
    for (int r = 0; r < n_rounds; r++) {
        const int slot = E.round_list[r];
        const DRequest& R = E.reqs[slot];
        const int n = (int)((R.total - R.round_base) / R.spp);
        const int* list = R.act[R.round & 1];
        int* next = R.act[(R.round & 1) ^ 1];
        const float inv = 1.f / (float)R.spp;
        const int stride = gridDim.x * blockDim.x;
        for (int base = blockIdx.x * blockDim.x; base < n; base += stride) {  // warp-uniform trips
            const int k = base + threadIdx.x;
            bool keep = false;
            int px = 0;
            if (k < n) {
                px = list[k];
                double* a = R.accum + (size_t)px * 3;
                const float3 c = make_float3((float)a[0] * inv, (float)a[1] * inv, (float)a[2] * inv);
                float4 m = R.welford[2 * (size_t)px], m2 = R.welford[2 * (size_t)px + 1];
                const float taken = m.w + 1.f;
                const float3 d1 = make_float3(c.x - m.x, c.y - m.y, c.z - m.z);
                m.x += d1.x / taken; m.y += d1.y / taken; m.z += d1.z / taken;
                const float3 d2 = make_float3(c.x - m.x, c.y - m.y, c.z - m.z);
                m2.x += d1.x * d2.x; m2.y += d1.y * d2.y; m2.z += d1.z * d2.z;
                m.w = taken;
                bool done = (int)taken >= R.aa;
                if (!done && taken >= 4.f) {
                    const float t1 = taken - 1.f;
                    const float rx = (m2.x / t1) / (m.x * m.x + 0.01f), ry = (m2.y / t1) / (m.y * m.y + 0.01f),
                                rz = (m2.z / t1) / (m.z * m.z + 0.01f);
                    done = fmaxf(fmaxf(rx, ry), rz) < 0.05f;
                }
                R.welford[2 * (size_t)px] = m;
                R.welford[2 * (size_t)px + 1] = m2;
                if (done) { a[0] = m.x; a[1] = m.y; a[2] = m.z; }
                else { a[0] = 0.0; a[1] = 0.0; a[2] = 0.0; keep = true; }
            }
            const unsigned km = __ballot_sync(0xffffffffu, keep);
            int b = 0;
            if (lane == 0 && km) b = atomicAdd(&E.round_cnt[slot], __popc(km));
            b = __shfl_sync(0xffffffffu, b, 0);
            if (keep) next[b + __popc(km & ((1u << lane) - 1u))] = px;
        }
    }
}

// ------------------------------------------------------------------ resolve
// Per-pixel mean -> linear sRGB (code/Renderer.cpp:300-302), then tone map
// and 8-bit quantise (code/Renderer.cpp:365-382) on the device.
__global__ void k_resolve(const double* __restrict__ acc, int npix, double inv_n, int spectral, int aces_tm,
                          float* __restrict__ hdr, unsigned char* __restrict__ rgb8, const int* status = nullptr,
                          int* status_host = nullptr)
{
    // (a copy of this one word would cost the call 9 us)
    if (status_host && blockIdx.x == 0 && threadIdx.x == 0) *status_host = *status;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < npix; i += gridDim.x * blockDim.x) {
        float3 c = make_float3((float)(acc[i * 3] * inv_n), (float)(acc[i * 3 + 1] * inv_n), (float)(acc[i * 3 + 2] * inv_n));
        if (spectral) c = xyz_to_srgb(c);
        if (hdr) { hdr[i * 3] = c.x; hdr[i * 3 + 1] = c.y; hdr[i * 3 + 2] = c.z; }
        if (rgb8) {
            float3 m = aces_tm ? make_float3(aces(c.x), aces(c.y), aces(c.z)) : make_float3(reinhard(c.x), reinhard(c.y), reinhard(c.z));
            rgb8[i * 3] = quantize(m.x);
            rgb8[i * 3 + 1] = quantize(m.y);
            rgb8[i * 3 + 2] = quantize(m.z);
        }
    }
}

// Tone map + quantise a linear sRGB image (the last step of k_resolve).
__global__ void k_tonemap(const float* __restrict__ hdr, int npix, int aces_tm, unsigned char* __restrict__ rgb8)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < npix; i += gridDim.x * blockDim.x) {
        const float3 c = make_float3(hdr[i * 3], hdr[i * 3 + 1], hdr[i * 3 + 2]);
        const float3 m = aces_tm ? make_float3(aces(c.x), aces(c.y), aces(c.z))
                                 : make_float3(reinhard(c.x), reinhard(c.y), reinhard(c.z));
        rgb8[i * 3] = quantize(m.x);
        rgb8[i * 3 + 1] = quantize(m.y);
        rgb8[i * 3 + 2] = quantize(m.z);
    }
}

// ------------------------------------------------------------------ denoise
// One pass of the 5x5 cross-bilateral on the 8-bit image (Denoise::
// bilateralRGB, code/Denoise.cpp:14-86, which runs two): spatial sigma 1.5
// px, colour sigma 10 levels, float arithmetic in the reference's order (no
// contraction), the weight's exponential taken in double and rounded once.
//
// A weight depends on the squared pixel distance (six values) and the squared
// colour distance, an integer, and rounds to zero from an exponent of 104 on:
// 6 x 20,900 weights (0.5 MB, L2-resident), tabulated once per context with
// the same operations, stand in for 25 double exponentials a pixel and pass
// (1280x720: 86 -> 43 us a pass; the byte loads of the window are left).
constexpr int kBilateralSums = 20900;  // colour distances up to an exponent of 104.5
constexpr int kBilateralEntries = 6 * kBilateralSums;
__device__ __forceinline__ int bilateral_row(int d2)  // of d2 = 0, 1, 2, 4, 5, 8
{
    return d2 < 3 ? d2 : (d2 == 4 ? 3 : (d2 == 5 ? 4 : 5));
}
__global__ void k_bilateral_table(float* __restrict__ table)
{
    using namespace ex;
    const float invSpatial2 = div(1.0f, mul(mul(2.0f, 1.5f), 1.5f));
    const float invColor2 = div(1.0f, mul(mul(2.0f, 10.0f), 10.0f));
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kBilateralEntries; i += gridDim.x * blockDim.x) {
        const int row = i / kBilateralSums;
        const int d2 = row < 3 ? row : (row == 3 ? 4 : (row == 4 ? 5 : 8));
        const float spatial = mul((float)d2, invSpatial2);
        const float color = mul((float)(i - row * kBilateralSums), invColor2);
        table[i] = (float)exp(-(double)add(spatial, color));
    }
}
__global__ void k_bilateral(const unsigned char* __restrict__ src, unsigned char* __restrict__ dst, int width,
                            int height, const float* __restrict__ table)
{
    using namespace ex;
    const int npix = width * height;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < npix; p += gridDim.x * blockDim.x) {
        const int y = p / width, x = p - y * width;
        const int cR = src[p * 3], cG = src[p * 3 + 1], cB = src[p * 3 + 2];
        float sumW = 0.f, sumR = 0.f, sumG = 0.f, sumB = 0.f;
        for (int dy = -2; dy <= 2; dy++) {
            const int ny = y + dy;
            if (ny < 0 || ny >= height) continue;
#pragma unroll
            for (int dx = -2; dx <= 2; dx++) {
                const int nx = x + dx;
                if (nx < 0 || nx >= width) continue;
                const int q = (ny * width + nx) * 3;
                const int nR = src[q], nG = src[q + 1], nB = src[q + 2];
                const int dR = nR - cR, dG = nG - cG, dB = nB - cB;
                const int c2 = dR * dR + dG * dG + dB * dB;
                if (c2 >= kBilateralSums) continue;  // weight zero: adds nothing
                const float w = table[bilateral_row(dx * dx + dy * dy) * kBilateralSums + c2];
                sumW = add(sumW, w);
                sumR = add(sumR, mul(w, (float)nR));
                sumG = add(sumG, mul(w, (float)nG));
                sumB = add(sumB, mul(w, (float)nB));
            }
        }
        if (sumW > 0.f) {
            dst[p * 3] = (unsigned char)fminf(255.f, add(div(sumR, sumW), 0.5f));
            dst[p * 3 + 1] = (unsigned char)fminf(255.f, add(div(sumG, sumW), 0.5f));
            dst[p * 3 + 2] = (unsigned char)fminf(255.f, add(div(sumB, sumW), 0.5f));
        } else {
            dst[p * 3] = src[p * 3];
            dst[p * 3 + 1] = src[p * 3 + 1];
            dst[p * 3 + 2] = src[p * 3 + 2];
        }
    }
}

// ------------------------------------------------------------------ parity kernels
__global__ void k_trace_rays(const DScene* scene, const DMaterial* mats, const float* __restrict__ rays, long long n,
                             int* mat, int* prim_out, float* t_out, int bvh_only, int* counts)
{
    const DScene& S = *scene;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float3 o = make_float3(rays[i * 6], rays[i * 6 + 1], rays[i * 6 + 2]);
        const float3 d = make_float3(rays[i * 6 + 3], rays[i * 6 + 4], rays[i * 6 + 5]);
        float t = FLT_MAX, u = 0.f, v = 0.f;
        if (bvh_only) {
            TraceCounts tc = {0, 0};
            int tri = counts ? bvh4_closest<true>(S, o, d, t, u, v, &tc) : bvh4_closest<false>(S, o, d, t, u, v, nullptr);
            prim_out[i] = tri >= 0 ? __float_as_int(S.tris[tri].v0_id.w) : -1;
            t_out[i] = tri >= 0 ? t : 0.f;
            if (counts) { counts[i * 2] = tc.nodes; counts[i * 2 + 1] = tc.tris; }
        } else {
            const uint32_t prim = scene_closest<true>(S, o, d, FLT_MAX, t, u, v);
            const uint32_t kind = prim & kPrimKindMask, pidx = prim & kPrimIndexMask;
            int mi = -1;
            uint32_t code = 0;
            if (kind == kPrimSphere) { mi = S.spheres[pidx].mat.x; code = kind | pidx; }
            else if (kind == kPrimPlane) { mi = __float_as_int(S.planes[pidx].o_mat.w); code = kind | pidx; }
            else if (kind == kPrimTri) {
                mi = __float_as_int(S.tris[pidx].e1_mat.w);
                code = kind | ((uint32_t)__float_as_int(S.tris[pidx].v0_id.w) & kPrimIndexMask);
            }
            mat[i] = mi;
            prim_out[i] = (int)code;
            t_out[i] = kind ? t : 0.f;
        }
    }
}

// The shadow test of k_shadow on caller rays (origin, unit direction) with
// their squared light distances: 1 when blocked.
__global__ void k_trace_shadow(const DScene* scene, const DMaterial* mats, const float* __restrict__ rays,
                               const float* __restrict__ dist2, long long n, int* blocked)
{
    const DScene& S = *scene;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float3 o = make_float3(rays[i * 6], rays[i * 6 + 1], rays[i * 6 + 2]);
        const float3 d = make_float3(rays[i * 6 + 3], rays[i * 6 + 4], rays[i * 6 + 5]);
        const float d2 = dist2[i];
        blocked[i] = scene_blocked(S, mats, o, d, d2) ? 1 : 0;
    }
}

__global__ void k_eval_stage(int what, const float* __restrict__ params, const float* __restrict__ in, long long n,
                             float* __restrict__ out, float xyz_scale, const float4* __restrict__ cmf_table)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        switch (what) {
        // (the form that renders use, over the wavelengths they carry)
        case 0: {
            const float4 fit = make_float4(params[0], params[1], params[2], params[3]);
            out[i] = in[i] >= 400.f && in[i] <= 700.f ? sigmoid_fit<true>(fit, in[i]) : sigmoid_fit<false>(fit, in[i]);
        } break;
        case 1:
            out[i] = in[i] >= 400.f && in[i] <= 700.f ? spectrum_lerp<true>(params, in[i]) : spectrum_lerp<false>(params, in[i]);
            break;
        case 2: { float3 c = cmf(in[i]); out[i * 3] = c.x; out[i * 3 + 1] = c.y; out[i * 3 + 2] = c.z; } break;
        case 3: {
            float3 c = cmf(in[i * 2]);
            float r = in[i * 2 + 1];
            out[i * 3] = r * c.x * xyz_scale; out[i * 3 + 1] = r * c.y * xyz_scale; out[i * 3 + 2] = r * c.z * xyz_scale;
        } break;
        case 4: { float3 c = xyz_to_srgb(make_float3(in[i * 3], in[i * 3 + 1], in[i * 3 + 2]));
                  out[i * 3] = c.x; out[i * 3 + 1] = c.y; out[i * 3 + 2] = c.z; } break;
        case 5: for (int k = 0; k < 3; k++) out[i * 3 + k] = reinhard(in[i * 3 + k]); break;
        case 6: for (int k = 0; k < 3; k++) out[i * 3 + k] = aces(in[i * 3 + k]); break;
        case 7: for (int k = 0; k < 3; k++) out[i * 3 + k] = (float)quantize(in[i * 3 + k]); break;
        case 8: {
            // the XYZ weight raygen stores for a one-wavelength path (the
            // colour-matching table), times the radiance: singleLambdaXYZ
            const float lam[4] = {in[i * 2], in[i * 2], in[i * 2], in[i * 2]};
            const XyzWeights W = xyz_weights(true, lam, 1, 1.f, xyz_scale, cmf_table);
            const float r = in[i * 2 + 1];
            out[i * 3] = r * W.w[0].x; out[i * 3 + 1] = r * W.w[0].y; out[i * 3 + 2] = r * W.w[0].z;
        } break;
        default: break;
        }
    }
}

}  // namespace pcr
