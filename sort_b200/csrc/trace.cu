// Closest-hit and any-hit traversal of SORT-topology wide BVHs on sm_100a.
//
// The per-ray traversal restates Fbvh::GetIntersect
// (accel/fast_bvh.hpp:305-504, SIMD branch):
//   * root slab test against the enlarged scene box (scalar Intersect);
//   * a stack of (node, entry distance) pairs; a popped entry is skipped when
//     the current hit is nearer than its entry distance (strict <, line 343);
//   * a leaf tests its triangles in SIMD-lane packing order and keeps a hit only
//     when strictly nearer (simd/simd_triangle.h:359-369), so the first of equal
//     distances wins;
//   * an interior node's hit children are visited nearest first; equal distances
//     visit the higher child slot first (the 1-, 2- and >=3-hit cases of lines
//     416-455 all reduce to that order);
//   * any-hit returns at the first triangle hit (opaque early exit, 362-373).
// With FP32 child boxes and the same rounding, hits, distances and barycentrics
// are bit-identical to SORT's.
//
// The hot kernel is k_trace_walk over warp_walk.cuh: a ray per lane, leaves
// tested by eight lanes each, idle lanes refilled. Counting launches
// (sg_trace_stats) run Traversal, one ray per thread, whose node and triangle
// visits are SORT's one by one. Schedules change the order in which rays are
// taken, never a result: batch order, or the order of a coherence key (direction
// octant, origin cell, coarse direction), so that concurrent warps read the same
// nodes.
#include <cuda_runtime.h>

#include <mutex>
#include <vector>

#include "group_walk.cuh"
#include "prefix_sort.cuh"
#include "trace_kernels.h"
#include "traversal.cuh"
#include "warp_walk.cuh"

namespace sg {

// The counting launches' kernel: one ray per thread (`Traversal`). Q8 reads 8-bit nodes.
template <int W, bool ANY, int STACK, bool Q8>
__global__ void __launch_bounds__(128, 9) k_trace_stats(DevTree tr, DevRays rays, int64_t n,
                                                        int32_t* __restrict__ prim_out, float* __restrict__ t_out,
                                                        float* __restrict__ u_out, float* __restrict__ v_out,
                                                        uint8_t* __restrict__ occ_out, int* __restrict__ err,
                                                        unsigned long long* __restrict__ stats) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    Traversal<W, ANY, STACK, true, Q8, true> tv;
    uint2 stk_mem[STACK];
    tv.stk = stk_mem;
    if (tv.start(tr, rays, i))
        while (!tv.step(tr, err)) {
        }
    tv.finish(i, prim_out, t_out, u_out, v_out, occ_out, stats);
}

// Launch shape of k_trace_walk per tree form: blocks of 128 per SM (registers:
// 72 at 7 blocks hold the width-8 FP32 walk without a spill, 64 at 8 blocks the
// others but width 8 with 8-bit nodes, 12 bytes) and the idle lanes at which a warp
// takes new rays. Measured, same
// box, width 8: 7 blocks 2.54 / 2.10 ms on 4M diffuse / shadow rays (21M
// triangles), 8 blocks (88 bytes spilled) 2.98 / 2.25, 9 blocks 2.96 / 2.40.
// 8-bit nodes: 0.338 / 0.334 / 0.336 ms at 7 / 8 / 9 blocks on 700k rays.
// Width 4, 1M camera rays: 0.207 / 0.207 / 0.201 ms at 7 / 8 / 9 blocks.
// Refills at 4 / 10 / 16 / 24 / 28 / 32 idle lanes: diffuse 2.40 / 2.19 / 2.20 /
// 2.15 / 2.17 / 2.44 ms, shadow 2.29 / 2.09 / 2.09 / 2.05 / 2.05 / 2.13, camera
// (width 4) 0.215 / 0.192 / 0.184 / 0.178 / 0.178 / 0.180; a refill is a ray's
// setup at that many lanes, so it pays to wait. 8-bit nodes, whose visits cost
// more, 0.336 / 0.325 / 0.328 / 0.340 / 0.351 / 0.398.
template <int W, bool Q8>
struct WalkShape {
    static constexpr int kBlocks = W == 8 && !Q8 ? 7 : 8;
    static constexpr int kRefill = Q8 ? 12 : 24;
};

// Launch shape of k_trace_groups: blocks of 128 per SM (56 registers). A launch of at
// most a ray per group (18,944 rays on 148 SMs) over a width-8 tree takes it.
// k_trace_walk against it, us: diffuse rays, 5.2M triangles, 84.6 / 77.7 at 18,944
// rays, 94.6 / 92.0 at 26,000, 110 / 172 at 65,536; shadow 67.0 / 51.3, 91.4 / 66.4,
// 95.8 / 129; camera, 82k triangles, 32.9 / 30.8 at 18,944. A larger launch is bound
// by issue slots, of which this form takes more.
constexpr int kGroupBlocks = 8;

// Rays of a launch as its warps take them: one span of `span` rays per warp, or,
// with a counter, as many as the warp has idle lanes from the launch's counter,
// so that the whole GPU advances through the batch in order (neighbouring rays
// read the same nodes) and no warp ends much before the others.
struct TraceJob {
    const DevTree& tr;
    const DevRays& rays;
    const int32_t* order;
    int32_t* prim_out;
    float* t_out;
    float* u_out;
    float* v_out;
    uint8_t* occ_out;
    unsigned* counter;
    int next, end;  // rays left: the warp's span, or, with a counter, all of them until it has passed n

    __device__ __forceinline__ const DevTree& tree() const { return tr; }
    __device__ __forceinline__ bool more() const { return next < end; }
    __device__ __forceinline__ bool take(bool idle, unsigned mask, int lane, WalkShared* sh, RayState& r,
                                         const DevTree&) {
        if (counter) {
            unsigned b = 0;
            if (lane == 0) b = atomicAdd(counter, (unsigned)__popc(mask));
            b = __shfl_sync(kFullWarp, b, 0);
            next = b < (unsigned)end ? (int)b : end;
        }
        const int k = next + __popc(mask & ((1u << lane) - 1u));
        const bool got = idle && k < end;
        next += __popc(mask);
        if (!got) return false;
        const int i = order ? __ldg(order + k) : k;
        sh->ray[lane] = (uint32_t)i;
        r.o[0] = rays.ox[i];
        r.o[1] = rays.oy[i];
        r.o[2] = rays.oz[i];
        r.d[0] = rays.dx[i];
        r.d[1] = rays.dy[i];
        r.d[2] = rays.dz[i];
        r.tmin = rays.tmin[i];
        r.tmax = rays.tmax[i];
        return true;
    }
    __device__ __forceinline__ void put(bool fin, int lane, const WalkShared* sh) const {
        if (!fin) return;
        const uint32_t i = sh->ray[lane] & kWalkRayMask;
        const int32_t prim = sh->prim[lane];
        if (occ_out) {
            occ_out[i] = prim >= 0 ? 1 : 0;
            return;
        }
        prim_out[i] = prim;
        t_out[i] = sh->t[lane];
        if (u_out) u_out[i] = prim >= 0 ? sh->u[lane] : 0.0f;
        if (v_out) v_out[i] = prim >= 0 ? sh->v[lane] : 0.0f;
    }
};

constexpr int kMaxWalkRays = 1 << 30;  // per launch: ray indices of 30 bits
constexpr int kWalkSpan = 64;          // rays per warp of a large launch that has no counter
static_assert(kMaxWalkRays - 1 <= (int)kWalkRayMask, "a ray's index fits its shared word");

// Traces min(n, *n_dev) rays (n_dev may be null); with `order` set, the k-th ray
// taken is ray order[k]. slots: warps the GPU holds at once. Up to 32 rays per
// such warp each warp gets an equal share, so that a small batch spreads over
// every SM (a ray's chain of dependent loads is what a small launch waits for);
// beyond, warps take rays from `counter` (zero at launch) or by spans.
template <int W, bool ANY, int STACK, bool Q8>
__global__ void __launch_bounds__(kWalkThreads, WalkShape<W, Q8>::kBlocks)
    k_trace_walk(const __grid_constant__ DevTree tr, const __grid_constant__ DevRays rays, int n, int slots, int refill,
                 int32_t* __restrict__ prim_out, float* __restrict__ t_out, float* __restrict__ u_out,
                 float* __restrict__ v_out, uint8_t* __restrict__ occ_out, int* __restrict__ err,
                 const int* __restrict__ n_dev, const int32_t* __restrict__ order, unsigned* __restrict__ counter) {
    __shared__ WalkShared shared[kWalkWarps];
    const int lane = threadIdx.x & 31, warp = (int)blockIdx.x * kWalkWarps + (threadIdx.x >> 5);
    if (n_dev) n = min(n, *n_dev);
    int span = kWalkSpan;
    if (n <= slots * 32) {
        span = (n + slots - 1) / slots;
        counter = nullptr;
    }
    TraceJob job{tr, rays, order, prim_out, t_out, u_out, v_out, ANY ? occ_out : nullptr, counter, 0, n};
    if (!counter) {
        const int64_t first = (int64_t)warp * span;
        if (first >= n) return;
        job.next = (int)first;
        job.end = n - job.next < span ? n : job.next + span;
    }
    walk_rays<W, ANY, STACK, Q8, false>(job, shared + (threadIdx.x >> 5), lane, refill, err);
}

// Traces min(n, *n_dev) rays (n_dev may be null) with eight lanes per ray; up to a ray
// per warp each warp has one.
template <bool ANY, int STACK, bool Q8>
__global__ void __launch_bounds__(kWalkThreads, kGroupBlocks)
    k_trace_groups(const __grid_constant__ DevTree tr, const __grid_constant__ DevRays rays, int n,
                   int32_t* __restrict__ prim_out, float* __restrict__ t_out, float* __restrict__ u_out,
                   float* __restrict__ v_out, uint8_t* __restrict__ occ_out, int* __restrict__ err,
                   const int* __restrict__ n_dev) {
    __shared__ GroupStack<ANY, STACK> stacks[kBlockGroups];
    const int lane = threadIdx.x & 31, warp = (int)blockIdx.x * kWalkWarps + (threadIdx.x >> 5);
    const int ord = lane & (kGroupLanes - 1), g = lane / kGroupLanes;
    if (n_dev) n = min(n, *n_dev);
    const int warps = (int)gridDim.x * kWalkWarps;
    const int share = min(kWarpGroups, (n + warps - 1) / warps);  // groups of a warp that take rays
    int i = -1, next = g < share ? warp * share + g : n;
    GroupWalk<ANY, STACK, Q8> w;
    w.cur = kEmpty;
    for (;;) {
        const bool idle = w.cur == kEmpty && (i >= 0 || next < n);
        if (__any_sync(kFullWarp, idle)) {
            if (idle) {
                if (i >= 0) {
                    if constexpr (ANY) {
                        if (ord == 0) occ_out[i] = w.prim >= 0 ? 1 : 0;
                    } else {
                        if (ord == 0) prim_out[i] = w.prim;
                        if (ord == 1) t_out[i] = w.t;
                        if (ord == 2 && u_out) u_out[i] = w.u;
                        if (ord == 3 && v_out) v_out[i] = w.v;
                    }
                    i = -1;
                }
                if (next < n) {
                    i = next;
                    next += warps * share;
                    RayState r;
                    r.o[0] = rays.ox[i];
                    r.o[1] = rays.oy[i];
                    r.o[2] = rays.oz[i];
                    r.d[0] = rays.dx[i];
                    r.d[1] = rays.dy[i];
                    r.d[2] = rays.dz[i];
                    r.tmin = rays.tmin[i];
                    r.tmax = rays.tmax[i];
                    w.begin(tr, r);
                }
            }
        } else if (__all_sync(kFullWarp, w.cur == kEmpty)) {
            break;
        }
        w.step(tr.nodes, tr.tris, &stacks[(threadIdx.x >> 5) * kWarpGroups + g], lane, err);
    }
}

// Stream-ordered scratch of a launch (the sorted schedule's keys and order, the
// ray counter): one pool per device that keeps up to 1 GiB mapped between
// launches (NULL if it cannot be made).
static cudaMemPool_t trace_scratch_pool(int device) {
    static std::mutex lock;
    static std::vector<cudaMemPool_t> pools;
    std::lock_guard<std::mutex> g(lock);
    if (device < 0) return nullptr;
    if (pools.size() <= size_t(device)) pools.resize(size_t(device) + 1, nullptr);
    if (!pools[size_t(device)]) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        cudaMemPool_t pool = nullptr;
        if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) return nullptr;
        uint64_t keep = uint64_t(1) << 30;
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
        pools[size_t(device)] = pool;
    }
    return pools[size_t(device)];
}

// Launches k_trace_walk over n rays, with the launch's counter or without one, or
// k_trace_groups where there are few.
template <int W, bool ANY, int STACK, bool Q8>
static cudaError_t launch_walk(const TraceLaunch& L, const DevTree& tr, const DevRays& rays, int64_t n,
                               const int32_t* order, unsigned* counter, cudaStream_t s) {
    using Shape = WalkShape<W, Q8>;
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    const int slots = (sms < 1 ? 1 : sms) * Shape::kBlocks * kWalkWarps;
    if constexpr (W == 8) {
        const int group_warps = (sms < 1 ? 1 : sms) * kGroupBlocks * kWalkWarps;
        if (!order && n <= (int64_t)group_warps * kWarpGroups) {
            const int warps = n < group_warps ? (int)n : group_warps;
            k_trace_groups<ANY, STACK, Q8><<<(unsigned)((warps + kWalkWarps - 1) / kWalkWarps), kWalkThreads, 0, s>>>(
                tr, rays, (int)n, L.prim, L.t, L.u, L.v, L.occ, L.err, L.n_dev);
            return cudaGetLastError();
        }
    }
    const int refill = L.tuning.schedule == kSchedulePersistent ? L.tuning.refill_threshold : Shape::kRefill;
    // A large launch takes its rays from a counter: the caller's, or one from the
    // scratch pool (not while the stream is captured: a graph may be replayed
    // beside itself, and callers that asked for no scratch get none). Without the
    // memory for one the launch goes by spans, as those do: 2.68 against 2.15 ms
    // on 4M diffuse rays.
    char* scratch = nullptr;
    if (L.n_dev && (n > kMaxWalkRays || (!counter && n > (int64_t)slots * 32)))
        return cudaErrorInvalidValue;  // one launch, and its length is known on the device alone
    if (!counter && L.scratch && n > (int64_t)slots * 32) {
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(s, &cap) != cudaSuccess) {
            (void)cudaGetLastError();
            cap = cudaStreamCaptureStatusActive;
        }
        if (cap == cudaStreamCaptureStatusNone) {
            cudaMemPool_t pool = trace_scratch_pool(dev);
            if (pool && cudaMallocFromPoolAsync(reinterpret_cast<void**>(&scratch), 256, pool, s) == cudaSuccess) {
                counter = reinterpret_cast<unsigned*>(scratch);
            } else {
                (void)cudaGetLastError();
                scratch = nullptr;
            }
        }
    }
    for (int64_t a = 0; a < n && e == cudaSuccess; a += kMaxWalkRays) {
        const int m = (int)(n - a < kMaxWalkRays ? n - a : kMaxWalkRays);
        int64_t warps = slots;
        if (m <= slots * 32)
            warps = m < slots ? m : slots;
        else if (!counter)
            warps = (m + kWalkSpan - 1) / kWalkSpan;
        if (scratch && (e = cudaMemsetAsync(counter, 0, sizeof(unsigned), s)) != cudaSuccess) break;
        const DevRays r{rays.ox + a, rays.oy + a, rays.oz + a,   rays.dx + a,
                        rays.dy + a, rays.dz + a, rays.tmin + a, rays.tmax + a};
        k_trace_walk<W, ANY, STACK, Q8><<<(unsigned)((warps + kWalkWarps - 1) / kWalkWarps), kWalkThreads, 0, s>>>(
            tr, r, m, slots, refill, ANY ? nullptr : L.prim + a, ANY ? nullptr : L.t + a, L.u ? L.u + a : nullptr,
            L.v ? L.v + a : nullptr, ANY ? L.occ + a : nullptr, L.err, L.n_dev, order, counter);
        e = cudaGetLastError();
    }
    if (scratch) {
        const cudaError_t f = cudaFreeAsync(scratch, s);
        if (e == cudaSuccess) e = f;
    }
    return e;
}

// ---------------------------------------------------------------------------
// Sorted schedule (SG_SCHEDULE_SORTED): rays are taken in the order of a 30-bit
// coherence key, so that the rays in traversal at one time start near one another
// and head the same way.
// The key: direction octant (3 bits), the Morton code of the origin's cell on a
// 128^3 grid over the scene box (21 bits), then 2 bits per axis of direction.
//
// The order is a stable sort of the keys (equal keys keep batch order, which
// carries the input's own coherence: neighbouring pixels, neighbouring hit
// points), made by least-significant-digit radix passes of 10 bits over the
// whole key (three passes):
//  * k_sort_keys: key and batch index per ray (coalesced SoA reads);
//  * per pass, k_digit_count: a tile of 4,096 keys per block counts its digits
//    in shared memory and writes them digit-major (count[d * tiles + tile]);
//    scan_exclusive: prefix sums over those counts, so each (digit, tile)
//    knows where its run starts; k_digit_scatter: each warp owns a contiguous
//    512-key chunk of its tile, counts its digits, the block turns the counts
//    into per-warp starting places, and each warp writes its keys in order
//    (lanes of one digit ranked by __match_any_sync), which keeps the sort
//    stable;
//  * k_trace_walk with `order`: the k-th ray taken is ray order[k], and its
//    answer goes to that ray's own index, so results do not depend on the order.
constexpr int kKeyBits = 30;
constexpr int kSortBits = 30;  // top bits of the key that are sorted
using psort::kDigits;
using psort::kSortTile;
using psort::kSortThreads;
using psort::kSortItems;
static_assert(kSortBits % psort::kDigitBits == 0 && kSortBits <= kKeyBits, "whole digits of the key");

struct KeyGrid {
    float lo[3];
    float scale[3];  // 128 cells over the scene box's extent on each axis
};

__device__ __forceinline__ uint32_t spread7(uint32_t v) {  // bit b of v to bit 3b
    uint32_t r = 0;
#pragma unroll
    for (int b = 0; b < 7; ++b) r |= ((v >> b) & 1u) << (3 * b);
    return r;
}

// Key and batch index of every ray of a tile of kSortTile rays, and the tile's
// counts of the first pass's digit (as k_digit_count).
__global__ void __launch_bounds__(kSortThreads) k_sort_keys(DevRays rays, int64_t n, KeyGrid g, int shift, int tiles,
                                                            uint32_t* __restrict__ keys, int32_t* __restrict__ index,
                                                            uint32_t* __restrict__ count,
                                                            unsigned* __restrict__ counter) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *counter = 0;  // the traversal's
    __shared__ uint32_t hist[kDigits];
    for (int d = threadIdx.x; d < kDigits; d += kSortThreads) hist[d] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * kSortTile;
#pragma unroll 4
    for (int j = 0; j < kSortItems; ++j) {
        const int64_t i = base + j * kSortThreads + threadIdx.x;
        if (i >= n) continue;
        const float o[3] = {rays.ox[i], rays.oy[i], rays.oz[i]}, d[3] = {rays.dx[i], rays.dy[i], rays.dz[i]};
        uint32_t oct = 0, cell = 0, dir = 0;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            oct |= (d[a] < 0.0f ? 1u : 0u) << (2 - a);
            const float q = fminf(fmaxf((o[a] - g.lo[a]) * g.scale[a], 0.0f), 127.0f);  // NaN -> 0
            cell |= spread7((uint32_t)q) << (2 - a);
            const float e = fminf(fmaxf((d[a] + 1.0f) * 2.0f, 0.0f), 3.0f);
            dir |= ((uint32_t)e & 1u) << (2 - a) | (((uint32_t)e >> 1) & 1u) << (5 - a);
        }
        const uint32_t key = (oct << 27) | (cell << 6) | dir;
        keys[i] = key;
        index[i] = (int32_t)i;
        atomicAdd(&hist[(key >> shift) & (kDigits - 1)], 1u);
    }
    __syncthreads();
    for (int d = threadIdx.x; d < kDigits; d += kSortThreads) count[(size_t)d * tiles + blockIdx.x] = hist[d];
}

// The sorted schedule. Scratch (16 bytes per ray, 4 per (digit, tile) and the
// scan's) comes from the library's stream-ordered pool and is freed in stream
// order.
template <int W, bool ANY, int STACK, bool Q8>
static cudaError_t launch_sorted(const TraceLaunch& L, const DevTree& tr, const DevRays& rays, int64_t n,
                                 cudaStream_t s) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    cudaMemPool_t pool = trace_scratch_pool(dev);
    if (!pool) return cudaErrorMemoryAllocation;
    const int tiles = psort::sort_tiles(n);
    const size_t al = 256;
    auto up = [al](size_t b) { return ((b + al - 1) / al) * al; };
    const size_t b_ray = up(size_t(n) * 4), b_count = up(psort::sort_count_words(n) * 4),
                 b_scan = up(psort::sort_scan_words(n) * 4);
    char* base = nullptr;
    e = cudaMallocFromPoolAsync(reinterpret_cast<void**>(&base), 4 * b_ray + b_count + b_scan + al, pool, s);
    if (e != cudaSuccess) return e;
    uint32_t* keys[2] = {reinterpret_cast<uint32_t*>(base), reinterpret_cast<uint32_t*>(base + b_ray)};
    int32_t* idx[2] = {reinterpret_cast<int32_t*>(base + 2 * b_ray), reinterpret_cast<int32_t*>(base + 3 * b_ray)};
    uint32_t* count = reinterpret_cast<uint32_t*>(base + 4 * b_ray);
    uint32_t* scan = reinterpret_cast<uint32_t*>(base + 4 * b_ray + b_count);
    unsigned* counter = reinterpret_cast<unsigned*>(base + 4 * b_ray + b_count + b_scan);
    KeyGrid g;
    for (int a = 0; a < 3; ++a) {
        const float ext = tr.box_hi[a] - tr.box_lo[a];
        g.lo[a] = tr.box_lo[a];
        g.scale[a] = ext > 0.0f ? 128.0f / ext : 0.0f;
    }
    const int first = kKeyBits - kSortBits;
    k_sort_keys<<<tiles, kSortThreads, 0, s>>>(rays, n, g, first, tiles, keys[0], idx[0], count,
                                               counter);
    int cur = 0;
    if ((e = cudaGetLastError()) == cudaSuccess)
        e = psort::sort_pairs<uint32_t>(keys, idx, n, first, kKeyBits, count, scan, true, &cur, s);
    if (e == cudaSuccess) e = launch_walk<W, ANY, STACK, Q8>(L, tr, rays, n, idx[cur], counter, s);
    const cudaError_t f = cudaFreeAsync(base, s);
    return e != cudaSuccess ? e : f;
}

template <int W, bool ANY, int STACK, bool STATS>
static cudaError_t launch_stack(const TraceLaunch& L, const DevTree& tr, const DevRays& rays, int64_t n,
                                cudaStream_t s) {
    if (STATS) {
        const unsigned blocks = (unsigned)((n + 127) / 128);
        if (L.q8)
            k_trace_stats<W, ANY, STACK, true><<<blocks, 128, 0, s>>>(tr, rays, n, L.prim, L.t, L.u, L.v, L.occ, L.err,
                                                                      L.stats);
        else
            k_trace_stats<W, ANY, STACK, false><<<blocks, 128, 0, s>>>(tr, rays, n, L.prim, L.t, L.u, L.v, L.occ, L.err,
                                                                       L.stats);
        return cudaGetLastError();
    }
    // The automatic choice is batch order at every size: with lanes refilled and
    // leaves shared, a warp's rays need not be alike, and the sort costs more than
    // the cache lines it saves. Batch order against sorted, ms, 21M triangles, 4M
    // rays (1M rays): diffuse 2.19 / 2.50 (0.61 / 0.73), shuffled at random 2.52 /
    // 2.69 (0.70 / 0.80); camera 1.58 / 1.79, shuffled 2.33 / 2.50; shadow 2.09 /
    // 2.26, shuffled 2.44 / 2.50.
    if (L.tuning.schedule == kScheduleSorted && !L.n_dev && n >= (int64_t(1) << 16) && n <= kMaxWalkRays)
        return L.q8 ? launch_sorted<W, ANY, STACK, true>(L, tr, rays, n, s)
                    : launch_sorted<W, ANY, STACK, false>(L, tr, rays, n, s);
    return L.q8 ? launch_walk<W, ANY, STACK, true>(L, tr, rays, n, nullptr, L.counter, s)
                : launch_walk<W, ANY, STACK, false>(L, tr, rays, n, nullptr, L.counter, s);
}

template <int W, bool ANY, bool STATS>
static cudaError_t launch_w(const TraceLaunch& L, const DevTree& tr, const DevRays& rays, int64_t n, cudaStream_t s) {
    if (L.stack_need <= 64) return launch_stack<W, ANY, 64, STATS>(L, tr, rays, n, s);
    if (L.stack_need <= 128) return launch_stack<W, ANY, 128, STATS>(L, tr, rays, n, s);
    if (L.stack_need <= 256) return launch_stack<W, ANY, 256, STATS>(L, tr, rays, n, s);
    return cudaErrorInvalidValue;
}

template <bool STATS>
static cudaError_t launch_any_width(const TraceLaunch& L, const DevTree& tr, const DevRays& rays, int64_t n,
                                    cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    if (L.width == 8)
        return L.any ? launch_w<8, true, STATS>(L, tr, rays, n, s) : launch_w<8, false, STATS>(L, tr, rays, n, s);
    return L.any ? launch_w<4, true, STATS>(L, tr, rays, n, s) : launch_w<4, false, STATS>(L, tr, rays, n, s);
}

cudaError_t launch_trace_fp32(const TraceLaunch& L, const DevTree& tr, const DevRays& rays, int64_t n,
                              cudaStream_t s) {
    return L.stats ? launch_any_width<true>(L, tr, rays, n, s) : launch_any_width<false>(L, tr, rays, n, s);
}

}  // namespace sg
