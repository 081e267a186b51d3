// The path kernel: raygen, analytic trace, shading and shadow rays.
#pragma once

#include "kernels.cuh"

namespace pcr {

// k_paths follows each path in one thread, vertex after vertex, with its state
// in registers: closest hit, shading, shadow rays, next direction.  On a scene
// without a mesh it goes on to the path's end.  Where a ray meets the mesh's
// box, the path waits in the queue for k_extend's walk and is taken up again in
// the next iteration; a shadow ray that would be lit but meets the box becomes
// a record for k_shadow.
//
// Why one kernel and not one per stage: a ray meets at most a few dozen quads
// and spheres outside the mesh, so that part of its trace is short, and what
// stages pass through memory outweighs it: 400 B of path and hit records per
// vertex and 96 B per shadow ray, besides three FP64 reductions per lit
// sample, and five launches per vertex of a path.  The BVH walk is left out
// because it needs its own registers and full warps: inlined here, six mesh
// renders took 48 ms instead of 28.
//
// A warp keeps its lanes filled: a lane whose path has ended takes a pending
// sub-path of a dispersive fork from the warp's stack, then a queued path, and
// when kPathRefill lanes wait (raygen costs about one vertex, so it is not run
// for a lane or two at a time), they take the next camera paths; queue and
// camera paths are numbered by one counter shared by the grid.
//
// The samples of a path are added up in double and go to the pixel's FP64
// accumulator when the path ends or waits.
//
// What bounds it: instruction fetch and issue (50 % of the issue slots used, 24
// of 32 lanes active; 16 warps per SM at 128 registers; waits for instructions
// are the most frequent stall, as warps are spread over 40 KB of hot code:
// 1, 2, 3, 4 blocks per SM take 1923, 1173, 950, 842 us, but 5 and 6 blocks at
// 96 and 80 registers 943 and 1034 us).  Cornell 256x256, 16 paths a pixel, 4
// vertices, 4 shadow rays: stages of a queue 4.39 ms, this kernel 0.84 ms.
// 64x64, one path a pixel: 240 -> 98 us.  Refilling at 4 / 12 / 24 / 32 dead
// lanes: 1015 / 947 / 909 / 900 us, 24 uneven renders 103.6 / 102.7 / 98.3 /
// 98.3 ms.  Barriers that keep the warps of a scheduler at the same vertex end
// the instruction waits but cost as much in barrier waits.
//
// With a mesh, against queue stages of one vertex each: bunny 320x320, 8 paths
// a pixel 4.97 -> 2.01 ms, 24 uneven renders 80.8 -> 75.6 ms; six renders half
// of them through a glass mesh, where most vertices wait, 22.4 -> 26.0 ms.
//
// Staged requests are those on scenes whose rays this kernel would trace by the
// exact tests (the estimates do not take the scene's quads), or whose shadow
// rays have to find the closest of the mesh's emissive triangles (and requests
// of few paths on mesh scenes, see Engine::route).  Such traces are long and
// leave lanes idle, which costs more at 16 warps per SM and inside this code
// than the stages' memory traffic.  So a path is followed for one vertex and
// waits: k_extend traces its next ray in full, and each of its shadow samples
// is a record for k_shadow.  Six batched renders with 4 (16) shadow rays, by
// stages of one vertex alone / traced here / staged: a Cornell box with a tilted
// quad 24.9 (63.7) / 32.7 (79.5) / 26.7 (66) ms, with 88 quads 71 (206) / 102 (316)
// / 75 (217) ms, with a mesh light 61 (197) / 112 (330) / 57 (191) ms; 256x256, 16
// paths a pixel, 4 shadow rays: 4.6 / 1.9 / 1.8, 9.4 / 6.5 / 4.8 and 7.5 / 7.2 / 3.7
// ms.  The rest of the difference in the first two: a warp appends its own
// paths, so neighbours lose each other sooner than where a block appends
// together (which takes k_shadow 3 % less and k_paths 3 to 8 % more).
constexpr int kPathBlock = 128;
#ifndef PCR_PATH_MIN_BLOCKS
#define PCR_PATH_MIN_BLOCKS 4
#endif
// (staged: 4, 5, 6, 7 blocks 8.8, 8.5, 8.4, 8.9 ms of the first batch above, 17.7,
// 17.1, 17.7, 19.8 ms with 16 shadow rays)
#ifndef PCR_STAGED_MIN_BLOCKS
#define PCR_STAGED_MIN_BLOCKS 5
#endif
#ifndef PCR_PATH_REFILL
#define PCR_PATH_REFILL 24
#endif
constexpr int kPathRefill = PCR_PATH_REFILL;
// A path forks at most once, into at most four sub-paths of which one stays
// in its lane; new camera paths are taken only when the stack is empty.  So
// pending entries + 3 x (lanes that may still fork) never exceed 3 x 32.
constexpr int kForkStack = 96;
constexpr int kForkWords = 14;
// Queued paths are taken up when this many lanes wait (a few loads each).
constexpr int kPathResume = 8;
// Shadow records are reserved per warp in chunks, one grid-wide atomic each; a
// warp takes a new chunk when fewer than kShadowLow are left, and marks what
// it leaves unused.  Records past the chunk are reserved one by one.
constexpr int kShadowChunk = 128, kShadowLow = 32;

struct PathWarp {
    float w[12][32];                     // XYZ weights of each lane's path
    uint32_t fork[kForkWords][kForkStack];  // pending sub-paths
    int pending;
    int shadow_next, shadow_end;         // the warp's chunk of shadow records
};

constexpr size_t kPathSmem = (kPathBlock / 32) * sizeof(PathWarp);

// The work of one k_paths launch for a single request (the plain method):
// `n` paths from number `first` on, in slot 0.
__global__ void k_one_request(EngineView E, DRequest r, long long first, int n)
{
    Counters* C = E.cnt;
    const_cast<DRequest*>(E.reqs)[0] = r;
    E.active[0] = 0;
    *E.n_active = 1;
    E.path_base[0] = 0;
    E.give_start[0] = first;
    C->path_n = n;
    C->next[0] = 0;
    C->paths += (unsigned long long)n;
    if (first == 0) {
        unsigned long long t;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        C->path_begin = t;
        C->path_end = 0;
    }
}

__device__ __forceinline__ XyzWeights lane_weights(const PathWarp& P, int lane)
{
    XyzWeights W;
    W.w[0] = make_float3(P.w[0][lane], P.w[1][lane], P.w[2][lane]);
    W.w[1] = make_float3(P.w[3][lane], P.w[4][lane], P.w[5][lane]);
    W.w[2] = make_float3(P.w[6][lane], P.w[7][lane], P.w[8][lane]);
    W.w[3] = make_float3(P.w[9][lane], P.w[10][lane], P.w[11][lane]);
    return W;
}
__device__ __forceinline__ void set_lane_weights(PathWarp& P, int lane, const XyzWeights& W)
{
    P.w[0][lane] = W.w[0].x; P.w[1][lane] = W.w[0].y; P.w[2][lane] = W.w[0].z;
    P.w[3][lane] = W.w[1].x; P.w[4][lane] = W.w[1].y; P.w[5][lane] = W.w[1].z;
    P.w[6][lane] = W.w[2].x; P.w[7][lane] = W.w[2].y; P.w[8][lane] = W.w[2].z;
    P.w[9][lane] = W.w[3].x; P.w[10][lane] = W.w[3].y; P.w[11][lane] = W.w[3].z;
}
// Only the hero wavelength is left.
__device__ __forceinline__ void single_lane_weights(PathWarp& P, int lane, float3 w)
{
    P.w[0][lane] = w.x; P.w[1][lane] = w.y; P.w[2][lane] = w.z;
#pragma unroll
    for (int k = 3; k < 12; k++) P.w[k][lane] = 0.f;
}

// BVH walk of a shadow ray in place, for a full shadow queue.
__device__ __noinline__ bool walk_blocked(const DScene& S, float3 o, float3 d, float bound, float d2)
{
    float u, v;
    return bvh4_closest<false, true>(S, o, d, bound, u, v, nullptr, (double)d2 - 1e-3) == -2;
}

// Reserves shadow records: the first one, or shadow_cap when none is left.
// (Past the cap the count grows by what is in flight at most, and shadow_cap
// stays far enough below 2^31 for that.)
__device__ __forceinline__ int shadow_slots(const EngineView& E, int count)
{
    int* next = &E.cnt->shadow_n;
    return __ldcg(next) < E.shadow_cap ? min(atomicAdd(next, count), E.shadow_cap) : E.shadow_cap;
}

// Marks the rest of the warp's chunk as unused.
__device__ __forceinline__ void close_shadow_chunk(const EngineView& E, const PathWarp& P, int lane)
{
    for (int k = P.shadow_next + lane; k < P.shadow_end; k += 32) E.sq.o[k] = make_float4(0.f, 0.f, 0.f, -1.f);
}

// Shadow records of a staged request's vertex: one per sample, those that add
// nothing marked as unused.  The lanes that come here together reserve them
// with one grid-wide atomic; where they do not fit (the fixed queue of
// pcr_render_noalloc), the vertices wait for the next iteration.  Without a
// mesh the lanes' records of a sample lie side by side (one contiguous run a
// store), over a BVH those of a vertex, which walk mostly the same nodes.
struct StagedRecords {
    int first, step, most;
    bool fit;
    __device__ __forceinline__ int at(int s) const { return first + s * step; }
    __device__ __forceinline__ void skip(const EngineView& E, int s) const
    {
        if (at(s) < E.shadow_cap) E.sq.o[at(s)] = make_float4(0.f, 0.f, 0.f, -1.f);
    }
};
__device__ __forceinline__ StagedRecords staged_records(const EngineView& E, int samples, bool mesh)
{
    const unsigned m = __activemask();
    const int lane = threadIdx.x & 31, leader = __ffs(m) - 1, casters = __popc(m);
    StagedRecords r;
    r.most = (int)__reduce_max_sync(m, (unsigned)samples);
    int at = 0;
    if (lane == leader) at = shadow_slots(E, r.most * casters);
    at = __shfl_sync(m, at, leader);
    r.fit = at + r.most * casters <= E.shadow_cap;
    const int rank = __popc(m & ((1u << lane) - 1u));
    const bool rows = __any_sync(m, mesh);
    r.first = at + (rows ? rank * r.most : rank);
    r.step = rows ? 1 : casters;
    return r;
}

// Whose paths a launch of k_paths follows (Engine::route): to their end, to the
// mesh, or staged.
constexpr int kFlatPaths = 0, kMeshPaths = 1, kStagedPaths = 2;

// Work of one launch: the paths of queue `cur` (kMesh), then the camera paths
// numbered over the active list: position r's start at base[r] and are the
// request's paths give_start[r], give_start[r] + 1, ...
template <int kPaths>
__global__ void __launch_bounds__(kPathBlock, kPaths == kStagedPaths ? PCR_STAGED_MIN_BLOCKS : PCR_PATH_MIN_BLOCKS)
k_paths(const __grid_constant__ EngineView E, int cur, float xyz_scale)
{
    extern __shared__ __align__(16) unsigned char s_paths[];
    PathWarp& P = reinterpret_cast<PathWarp*>(s_paths)[threadIdx.x >> 5];
    constexpr bool kMesh = kPaths != kFlatPaths, kStaged = kPaths == kStagedPaths;
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    Counters* C = E.cnt;
    const int* base = kMesh ? E.give_base : E.path_base;
    int* counter = &C->next[kPaths];
    // queued and camera paths of the other kind are left to its launch
    auto mine = [&](const DRequest& R) { return !kMesh || ((R.flags & kReqStaged) != 0) == kStaged; };
    const int queued = kMesh ? min(C->queue_n[cur], E.queue_cap) : 0;
    const int n = queued + (kMesh ? C->new_n : C->path_n), n_act = *E.n_active;
    // staged: all lanes at a time, from ranges of a few warps' worth each
    int refill = kStaged ? 32 : queued > 0 ? kPathResume : kPathRefill;
    const int take = n / (int)(gridDim.x * (kPathBlock / 32)) >= 512 ? 128 : 32;
    int own = 0, left = 0;
    if (lane == 0) P.pending = P.shadow_next = P.shadow_end = 0;
    __syncwarp();

    bool alive = false, more = n > 0;
    float3 o = make_float3(0.f, 0.f, 0.f), d = o;
    float4 tp = make_float4(0.f, 0.f, 0.f, 0.f);
    float lambda0 = 0.f;
    int meta = 0, slot = 0;
    uint32_t pixel = 0, sample = 0;
    bool traced = false;               // the ray's hit is known:
    uint32_t prim = kPrimNone;
    float t = 0.f, hu = 0.f, hv = 0.f;
    double ax = 0.0, ay = 0.0, az = 0.0;
    unsigned rays = 0, shadows = 0;
    auto flush = [&]() {
        if (ax != 0.0 || ay != 0.0 || az != 0.0) {
            double* acc = E.reqs[slot].accum + (size_t)pixel * 3;
            red_add(acc + 0, ax);
            red_add(acc + 1, ay);
            red_add(acc + 2, az);
            ax = ay = az = 0.0;
        }
    };

    // Next rays; a path whose ray waits for k_extend goes to the queue.
    auto trace = [&]() {
        bool wait = false;
        if (alive && !traced) {
            const DScene& S = E.scenes[E.reqs[slot].scene];
            rays++;
            t = FLT_MAX;
            if (kStaged) {
                wait = true;  // k_extend finds the hit
            } else {
                prim = scene_analytic<false>(S, o, d, t);
                if (kMesh) wait = mesh_may_hit(S, o, d, t);
            }
        }
        if (kMesh) {
            const unsigned m = __ballot_sync(kAll, wait);
            if (m) {
                int at = 0;
                if (lane == 0) at = atomicAdd(&C->queue_n[cur ^ 1], __popc(m));
                at = __shfl_sync(kAll, at, 0) + __popc(m & below);
                if (wait) {
                    flush();
                    alive = false;
                    if (at < E.queue_cap) {
                        const PathQueue& Q = E.q[cur ^ 1];
                        const DRequest& R = E.reqs[slot];
                        Q.o[at] = make_float4(o.x, o.y, o.z, lambda0);
                        Q.d[at] = make_float4(d.x, d.y, d.z, __int_as_float(meta));
                        Q.tp[at] = tp;
                        Q.id[at] = make_int4(slot, (int)pixel, (int)sample, R.scene);
                        if (!kStaged) Q.hit[at] = make_float4(t, __uint_as_float(prim), 0.f, 0.f);
                        if (R.flags & kReqSpectral) store_weights(Q, at, lane_weights(P, lane));
                    } else {
                        atomicOr(&C->status, 2);
                    }
                }
            }
        }
    };

    while (true) {
        if (kStaged) trace();
        // ---- refill
        unsigned dead = __ballot_sync(kAll, !alive);
        if (dead) {
            const int pending = P.pending;
            if (pending) {
                const int k = pending - 1 - __popc(dead & below);
                if (!alive && k >= 0) {
                    o = make_float3(__uint_as_float(P.fork[0][k]), __uint_as_float(P.fork[1][k]), __uint_as_float(P.fork[2][k]));
                    d = make_float3(__uint_as_float(P.fork[3][k]), __uint_as_float(P.fork[4][k]), __uint_as_float(P.fork[5][k]));
                    lambda0 = __uint_as_float(P.fork[6][k]);
                    const float f = __uint_as_float(P.fork[7][k]);
                    tp = make_float4(f, f, f, f);
                    single_lane_weights(P, lane, make_float3(__uint_as_float(P.fork[8][k]), __uint_as_float(P.fork[9][k]),
                                                             __uint_as_float(P.fork[10][k])));
                    pixel = P.fork[11][k];
                    sample = P.fork[12][k];
                    meta = (int)(P.fork[13][k] & 0xffffu);
                    slot = (int)(P.fork[13][k] >> 16);
                    alive = true;
                }
                __syncwarp();
                if (lane == 0) P.pending = max(0, pending - __popc(dead));
                __syncwarp();
                dead = __ballot_sync(kAll, !alive);
            }
            if (more && __popc(dead) >= refill) {
                int first = 0;
                if (kStaged) {
                    if (left == 0) {
                        if (lane == 0) own = atomicAdd(counter, take);
                        own = __shfl_sync(kAll, own, 0);
                        left = take;
                    }
                    first = own;
                    own += 32;
                    left -= 32;
                    more = own < n;
                } else {
                    if (lane == 0) first = atomicAdd(counter, __popc(dead));
                    first = __shfl_sync(kAll, first, 0);
                    more = first + __popc(dead) < n;
                }
                int i = first + __popc(dead & below);
                if (kMesh) {
                    const PathQueue& Q = E.q[cur];
                    if (kStaged && left > 0 && i + 32 < queued) {  // the warp's next paths
                        const int nx = i + 32;
                        prefetch_l2(Q.id + nx); prefetch_l2(Q.o + nx); prefetch_l2(Q.d + nx); prefetch_l2(Q.tp + nx);
                        prefetch_l2(Q.hit + nx);
                        prefetch_l2(Q.w[0] + nx); prefetch_l2(Q.w[1] + nx); prefetch_l2(Q.w[2] + nx);
                    }
                    if (!alive && i < queued) {
                        const int4 id = Q.id[i];
                        const DRequest& R = E.reqs[id.x];
                        if (mine(R)) {
                            const float4 o4 = Q.o[i], d4 = Q.d[i], h = Q.hit[i];
                            tp = Q.tp[i];
                            slot = id.x;
                            pixel = (uint32_t)id.y;
                            sample = (uint32_t)id.z;
                            o = xyz(o4);
                            d = xyz(d4);
                            lambda0 = o4.w;
                            meta = __float_as_int(d4.w);
                            t = h.x;
                            prim = __float_as_uint(h.y);
                            hu = h.z;
                            hv = h.w;
                            set_lane_weights(P, lane, (R.flags & kReqSpectral) ? load_weights(Q, i) : rgb_weights());
                            alive = traced = true;
                        }
                    }
                    if (!kStaged && first + __popc(dead) >= queued) refill = kPathRefill;
                    i -= queued;
                }
                if (!alive && i >= 0 && i < n - queued) {  // (negative: a queued path, perhaps of the other kind)
                    int lo = 0, hi = n_act - 1;
                    while (lo < hi) {  // last r with base[r] <= i: it has paths in this launch
                        const int mid = (lo + hi + 1) >> 1;
                        if (base[mid] <= i) lo = mid; else hi = mid - 1;
                    }
                    slot = E.active[lo];
                    const DRequest& R = E.reqs[slot];
                    if (mine(R)) {
                        XyzWeights W = rgb_weights();
                        const CameraPath p = camera_path(E, R, E.give_start[lo] + (i - base[lo]), xyz_scale, W);
                        set_lane_weights(P, lane, W);
                        pixel = p.pixel;
                        sample = p.sample;
                        o = make_float3(R.cam_x, R.cam_y, R.cam_z);
                        d = p.d;
                        lambda0 = p.lambda0;
                        tp = make_float4(1.f, 1.f, 1.f, 1.f);
                        meta = ((R.flags & kReqSpectral) ? R.hero : 4) << 12;
                        alive = true;
                    }
                }
            }
            if (!__any_sync(kAll, alive)) {
                if (more) continue;
                break;
            }
        }

        // ---- trace (staged: above, so that the lanes of paths that wait are
        // filled before the next vertex)
        if (!kStaged) trace();
        if (kPaths == kMeshPaths && P.shadow_end - P.shadow_next < kShadowLow) {  // shadow_next may lie past the end
            close_shadow_chunk(E, P, lane);
            __syncwarp();
            if (lane == 0) {
                const int at = shadow_slots(E, kShadowChunk);
                P.shadow_next = at;
                P.shadow_end = min(at + kShadowChunk, E.shadow_cap);
            }
            __syncwarp();
        }

        // ---- one vertex of each live path (staged: of those whose hit is known)
        if (alive && (!kStaged || traced)) {
            const DRequest& R = E.reqs[slot];
            const DScene& S = E.scenes[R.scene];
            alive = traced = false;
            if (prim != kPrimNone) {
                const int bounce = meta & 0xFF, fork = (meta >> 8) & 7, single = (meta >> 11) & 1, nHero = (meta >> 12) & 7;
                const bool spectral = (R.flags & kReqSpectral) != 0;
                const float4 lam4 = spectral ? path_wavelengths(lambda0, single, nHero) : make_float4(0.f, 0.f, 0.f, 0.f);
                const Surface sf = surface_at<kMesh>(S, prim, t, hu, hv, o, d);
                const float3 hit = sf.hit;
                float3 N = sf.N;
                const bool entering = f3dot(d, N) < 0.f;
                if (!entering) N = f3neg(N);
                const DMaterial& m = E.mats[S.mat_base + sf.mi];
                const bool last = bounce + 1 >= R.depth;
                if (m.flags & kMatEmissive) {
                    const float4 c = !spectral ? mul4(tp, rgb4(m.emissive))
                                   : S.emit_mat >= 0 ? tp : mul4(tp, spec4(m, 1, lam4));
                    const float3 e = apply_xyz(lane_weights(P, lane), c);
                    ax += (double)e.x;
                    ay += (double)e.y;
                    az += (double)e.z;
                } else if (m.flags & kMatMetallic) {
                    if (!last) {
                        const float cosI = -f3dot(d, N);
                        reflect_at(hit, N, d, cosI, o, d);
                        tp = mul4(tp, spectral ? spec4(m, 0, lam4) : rgb4(m.albedo));
                        meta++;
                        alive = true;
                    }
                } else if (m.flags & kMatTransparent) {
                    if (!last) {
                        const float cosI = -f3dot(d, N);
                        const bool dispersive = spectral && m.cauchyB != 0.f && !single && nHero > 1;
                        // fork: one sub-path per wavelength (code/Renderer.cpp:736-753);
                        // terminate: the hero wavelength's bounce alone
                        // (code/Gpu/Metal/MetalRenderer.mm:2143-2252)
                        const bool terminate = dispersive && (R.flags & kReqTerminate);
                        const bool disperse = dispersive && !terminate;
                        const int ways = disperse ? nHero : 1;
                        const float4 coins = rand4(R, pixel, sample, (uint32_t)fork, (uint32_t)bounce, 63u);
                        const float4 alg = spectral ? spec4(m, 0, lam4) : rgb4(m.albedo);
                        int at = 0;
                        if (disperse) at = atomicAdd(&P.pending, ways - 1);
                        float3 no = o, nd = d;
                        bool refl = false;
                        // the lane keeps sub-path 0, the last one computed
                        for (int k = ways - 1; k >= 0; k--) {
                            const float lk = comp4(lam4, k);
                            const float ior = ior_at(m, spectral && m.cauchyB != 0.f && (dispersive || single), lk);
                            refl = dielectric_bounce(hit, N, d, cosI, entering, ior, comp4(coins, k), no, nd);
                            if (k > 0 && at >= kForkStack) {
                                atomicOr(&C->status, 2);  // never expected, see kForkStack
                            } else if (k > 0) {
                                // sub-path k carries wavelength k alone
                                P.fork[0][at] = __float_as_uint(no.x);
                                P.fork[1][at] = __float_as_uint(no.y);
                                P.fork[2][at] = __float_as_uint(no.z);
                                P.fork[3][at] = __float_as_uint(nd.x);
                                P.fork[4][at] = __float_as_uint(nd.y);
                                P.fork[5][at] = __float_as_uint(nd.z);
                                P.fork[6][at] = __float_as_uint(lk);
                                P.fork[7][at] = __float_as_uint(comp4(tp, k) * comp4(alg, k));
                                P.fork[8][at] = __float_as_uint(P.w[3 * k][lane]);
                                P.fork[9][at] = __float_as_uint(P.w[3 * k + 1][lane]);
                                P.fork[10][at] = __float_as_uint(P.w[3 * k + 2][lane]);
                                P.fork[11][at] = pixel;
                                P.fork[12][at] = sample;
                                P.fork[13][at] = (uint32_t)((bounce + 1) | ((k + 1) << 8) | (1 << 11) | (nHero << 12)) |
                                                 ((uint32_t)slot << 16);
                                at++;
                            }
                        }
                        o = no;
                        d = nd;
                        if (disperse) {
                            const float f = tp.x * alg.x;
                            tp = make_float4(f, f, f, f);
                            meta = (bounce + 1) | (1 << 8) | (1 << 11) | (nHero << 12);
                            single_lane_weights(P, lane, make_float3(P.w[0][lane], P.w[1][lane], P.w[2][lane]));
                        } else {
                            tp = mul4(tp, alg);
                            meta++;
                            // a refraction ends the other wavelengths; the
                            // hero's share is scaled by their number so the
                            // estimate stays unbiased (a reflection does not
                            // depend on the wavelength and keeps them all)
                            if (terminate && !refl) {
                                const float h0 = tp.x * (float)nHero;
                                tp = make_float4(h0, h0, h0, h0);
                                meta |= 1 << 11;
                                single_lane_weights(P, lane, make_float3(P.w[0][lane], P.w[1][lane], P.w[2][lane]));
                            }
                        }
                        alive = true;
                    }
                } else {
                    // diffuse; the continuation starts at the hit moved once
                    // by 1e-3*N (the reference's mutating `hit + N * 1e-3`,
                    // code/Renderer.cpp:782 with samples = 1)
                    const float4 al = spectral ? spec4(m, 0, lam4) : rgb4(m.albedo);
                    float3 hc = f3add(hit, f3mul(N, 1e-3f));
                    StagedRecords rec;
                    bool postponed = false;
                    if (kStaged && S.total_light_area > 0.f) {
                        rec = staged_records(E, R.shadow, S.n_nodes > 0);
                        if (!rec.fit) {
                            // the path waits as it came, and its ray is traced again
                            for (int s = 0; s < rec.most; s++) rec.skip(E, s);
                            postponed = alive = true;
                            rays--;
                        }
                    }
                    if (!postponed) {
                        o = hc;
                        if (S.total_light_area > 0.f) {
                            const float inv_pi = 1.f / 3.14159274f;
                            const float scaleS = S.total_light_area * inv_pi / (float)R.shadow;
                            const float4 tpal = mul4(tp, al);
                            int cached = -1;
                            float3 V = make_float3(0.f, 0.f, 0.f);
                            if (spectral && S.emit_mat >= 0) {
                                // every light has the one emissive material, whose
                                // emission the weights already hold
                                V = f3mul(apply_xyz(lane_weights(P, lane), tpal), scaleS);
                                cached = S.emit_mat;
                            }
                            for (int s = 0; s < R.shadow; s++) {
                                const LightSample L = sample_light(S, R, pixel, sample, (uint32_t)fork, (uint32_t)bounce, (uint32_t)s);
                                const ShadowSegment g = shadow_segment(L, N, hc);
                                if (!(g.G > 0.f)) {
                                    if (kStaged) rec.skip(E, s);
                                    continue;
                                }
                                shadows++;
                                float bound = 0.f;
                                int query = kShadowWalk;
                                if (!kStaged) {
                                    query = scene_blocked_analytic<kMesh, false>(S, E.mats, g.so, g.wi, g.d2, bound);
                                    if (query == kShadowBlocked) continue;
                                }
                                if (L.mat != cached) {
                                    // product of this light material, once per vertex
                                    const DMaterial& lmat = E.mats[S.mat_base + L.mat];
                                    const float4 c = spectral ? mul4(tpal, spec4(lmat, 1, lam4)) : mul4(tpal, rgb4(lmat.emissive));
                                    V = f3mul(apply_xyz(lane_weights(P, lane), c), scaleS);
                                    cached = L.mat;
                                }
                                const float f = shadow_factor(S, R, g);
                                const float3 c = make_float3(V.x * f, V.y * f, V.z * f);
                                if (kMesh && query == kShadowWalk && (kStaged || mesh_may_hit(S, g.so, g.wi, bound))) {
                                    int at;
                                    if (kStaged) {
                                        at = rec.at(s);
                                    } else {
                                        at = atomicAdd(&P.shadow_next, 1);
                                        if (at >= P.shadow_end) at = shadow_slots(E, 1);
                                    }
                                    if (at < E.shadow_cap) {
                                        E.sq.o[at] = make_float4(g.so.x, g.so.y, g.so.z, g.d2);
                                        E.sq.d[at] = make_float4(g.wi.x, g.wi.y, g.wi.z, __int_as_float((int)pixel));
                                        E.sq.c[at] = make_float4(c.x, c.y, c.z, __int_as_float(slot | (R.scene << 16)));
                                        if (!kStaged) E.sq.bound[at] = bound;
                                        continue;
                                    }
                                    if (kStaged) continue;  // (they fit)
                                    if (walk_blocked(S, g.so, g.wi, bound, g.d2)) continue;
                                }
                                ax += (double)c.x;
                                ay += (double)c.y;
                                az += (double)c.z;
                            }
                            if (kStaged)
                                for (int s = R.shadow; s < rec.most; s++) rec.skip(E, s);
                        }
                        float3 nd;
                        float rr_scale;
                        if (diffuse_bounce(R, pixel, sample, (uint32_t)fork, bounce, last, spectral, al, N, nd, rr_scale)) {
                            d = nd;
                            tp = make_float4(tp.x * al.x * rr_scale, tp.y * al.y * rr_scale, tp.z * al.z * rr_scale,
                                             tp.w * al.w * rr_scale);
                            meta++;
                            alive = true;
                        }
                    }
                }
            }
            if (!alive) flush();
        }
        __syncwarp();
    }
    if (kPaths == kMeshPaths) close_shadow_chunk(E, P, lane);
    rays = __reduce_add_sync(kAll, rays);
    shadows = __reduce_add_sync(kAll, shadows);
    if (lane == 0 && (rays | shadows)) {  // a resumed path that ends at its vertex traced no ray
        atomicAdd(&C->rays, (unsigned long long)rays);
        atomicAdd(&C->shadow_rays, (unsigned long long)shadows);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long now;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
        atomicMax(&C->path_end, now);
    }
}

}  // namespace pcr
