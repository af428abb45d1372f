// Multi-scene batch traversal: one persistent kernel per group of batches that
// share a tree width, node format and query (closest / any hit) drains every
// batch of the group, whatever scene each one traces.
//
// The group's batches form one ray sequence (batch after batch, in table
// order). A warp claims as many consecutive rays of it as it has idle lanes,
// each lane finds its ray's batch by its position in that sequence, loads the
// ray from the batch's planes and traverses its batch's tree with the walk of
// the single-batch kernels (warp_walk.cuh), so every hit is the one
// sg_trace_closest / sg_trace_any returns for that batch alone. A warp refills
// once `refill` lanes are idle.
//
// Finished rays are written and counted against their batch when their warp
// refills (one atomic per batch and refill); the warp that counts a batch's
// last ray stamps the batch's completion time, which is thus the time its answers
// are written: a finished ray's wait for its warp's next refill is part of it. A
// run may carry a time budget: once it has passed, warps stop claiming rays, finish
// the ones they hold and the run reports the cut.
#include <cuda_runtime.h>

#include "batch_kernels.h"
#include "warp_walk.cuh"

namespace sg {

namespace {

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Largest k with batches[k].start <= idx (idx < the group's total, so that
// batch holds idx: empty batches share their start with the next one).
__device__ __forceinline__ int find_batch(const BatchDesc* __restrict__ bt, int count, int64_t idx, int hint) {
    const int64_t hs = __ldg(&bt[hint].start);
    if (idx >= hs && idx < hs + __ldg(&bt[hint].n)) return hint;
    int lo = 0, hi = count - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(&bt[mid].start) <= idx)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

// Counts the lanes whose answers were just written against their batches.
__device__ __forceinline__ void count_finished(bool fin, int b, const BatchArgs& a, int first, unsigned lane) {
    const unsigned fm = __ballot_sync(0xffffffffu, fin);
    if (fm == 0) return;
    const int leader = __ffs(fm) - 1;
    const int b0 = __shfl_sync(0xffffffffu, b, leader);
    const unsigned same = __ballot_sync(0xffffffffu, fin && b == b0);
    unsigned peers;
    if (same == fm)
        peers = fm;  // the usual case: one batch
    else
        peers = __match_any_sync(0xffffffffu, fin ? b : -1);
    if (fin && (unsigned)(__ffs(peers) - 1) == lane) {
        const unsigned long long c = (unsigned long long)__popc(peers);
        const unsigned long long old = atomicAdd(&a.remaining[first + b], 0ull - c);
        if (old == c) a.done_ns[first + b] = (long long)(global_ns() - a.state->start_ns);
    }
}

// The walk's shared state with, per lane, its ray's batch and index there.
struct BatchShared : WalkSharedMulti {
    int64_t index[32];
};

template <bool ANY>
struct BatchJob {
    const BatchArgs& a;
    const BatchDesc* __restrict__ bt;
    int first, count;
    int64_t total;
    long long budget;
    unsigned lanes;  // lanes that claim rays: a group of fewer rays than the grid has lanes is
                     // claimed in equal shares, one per warp, so that it spreads over every SM
    int b;           // this lane's batch within the group (its last one: the next search's hint)
    bool drained;    // warp-uniform: nothing left to claim

    __device__ __forceinline__ DevTree tree() const { return DevTree{}; }
    __device__ __forceinline__ bool more() const { return !drained; }
    __device__ __forceinline__ bool take(bool, unsigned mask, int lane, WalkSharedMulti* sh, RayState& r,
                                         DevTree& tr) {
        mask &= lanes;
        unsigned long long base = 0;
        if (lane == 0) {
            if (budget > 0 && (long long)(global_ns() - a.state->start_ns) > budget) {
                atomicOr(&a.state->status, kBatchBudgetCut);
                base = (unsigned long long)total;
            } else {
                base = atomicAdd(&a.state->counter[a.group], (unsigned long long)__popc(mask));
            }
        }
        base = __shfl_sync(kFullWarp, base, 0);
        if ((int64_t)base >= total || lanes != kFullWarp) drained = true;
        const int64_t idx = (int64_t)base + __popc(mask & ((1u << lane) - 1u));
        if (!((mask >> lane) & 1u) || idx >= total) return false;
        b = find_batch(bt, count, idx, b);
        const BatchDesc& d = bt[b];
        const int64_t stride = __ldg(&d.stride), j = idx - __ldg(&d.start);
        const float* p = d.rays + j;
        r.o[0] = __ldg(p);
        r.o[1] = __ldg(p + stride);
        r.o[2] = __ldg(p + 2 * stride);
        r.d[0] = __ldg(p + 3 * stride);
        r.d[1] = __ldg(p + 4 * stride);
        r.d[2] = __ldg(p + 5 * stride);
        r.tmin = __ldg(p + 6 * stride);
        r.tmax = __ldg(p + 7 * stride);
        tr = a.trees[__ldg(&d.tree)];
        sh->ray[lane] = 0;
        static_cast<BatchShared*>(sh)->index[lane] = j;
        return true;
    }
    __device__ __forceinline__ void put(bool fin, int lane, const WalkSharedMulti* sh) const {
        if (fin) {
            const BatchDesc& d = bt[b];
            const int64_t j = static_cast<const BatchShared*>(sh)->index[lane];
            const int32_t prim = sh->prim[lane];
            if constexpr (ANY) {
                d.occ[j] = prim >= 0 ? 1 : 0;
            } else {
                d.prim[j] = prim;
                d.t[j] = sh->t[lane];
                if (d.u) d.u[j] = prim >= 0 ? sh->u[lane] : 0.0f;
                if (d.v) d.v[j] = prim >= 0 ? sh->v[lane] : 0.0f;
            }
        }
        count_finished(fin, b, a, first, (unsigned)lane);
    }
};

// Blocks of 64 and 128: 896 resident threads per SM (72 registers), as k_trace_walk
// (20 bytes of the 8-bit width-8 walk spill); blocks of 256: three per SM, 768
// threads (80 registers). 24 batches of 4k .. 1M rays over five scenes (10k .. 2M
// triangles, width 8) take 1.01 ms; one ray per lane with every ray written and
// counted as it ends, 2.22.
template <int W, bool ANY, int STACK, int BLOCK, bool Q8>
__global__ void __launch_bounds__(BLOCK, 896 / BLOCK) k_trace_batches(const __grid_constant__ BatchArgs a) {
    __shared__ BatchShared shared[BLOCK / 32];
    const GroupDesc g = a.header->groups[a.group];
    if (g.count <= 0) return;
    const int64_t warps = (int64_t)gridDim.x * (BLOCK / 32), share = (g.total + warps - 1) / warps;
    const unsigned lanes = share < 32 ? (1u << share) - 1u : kFullWarp;
    BatchJob<ANY> job{a, a.batches + g.first, g.first, g.count, g.total, a.header->budget_ns, lanes, 0, false};
    walk_rays<W, ANY, STACK, Q8, true>(job, &shared[threadIdx.x >> 5], (int)(threadIdx.x & 31u), a.header->refill,
                                       &a.state->status);
}

__global__ void k_batch_begin(const RunHeader* __restrict__ h, const BatchDesc* __restrict__ batches,
                              RunState* __restrict__ st, unsigned long long* __restrict__ remaining,
                              long long* __restrict__ done_ns) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) {
        for (int g = 0; g < kMaxBatchGroups; ++g) st->counter[g] = 0;
        st->status = 0;
        st->start_ns = global_ns();
    }
    if (i < h->nbatches) {
        const int64_t n = batches[i].n;
        remaining[i] = (unsigned long long)n;
        done_ns[i] = n == 0 ? 0 : -1;
    }
}

template <int W, bool ANY, int STACK, int BLOCK, bool Q8>
cudaError_t launch_group(const BatchArgs& a, int grid, cudaStream_t s) {
    k_trace_batches<W, ANY, STACK, BLOCK, Q8><<<grid, BLOCK, 0, s>>>(a);
    return cudaGetLastError();
}

template <int W, bool ANY, int STACK, int BLOCK, bool Q8>
int group_occupancy() {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_trace_batches<W, ANY, STACK, BLOCK, Q8>, BLOCK, 0) !=
        cudaSuccess)
        return 0;
    return n;
}

template <int W, bool ANY, int STACK, int BLOCK, bool Q8>
BatchKernel make_kernel() {
    return BatchKernel{&launch_group<W, ANY, STACK, BLOCK, Q8>, &group_occupancy<W, ANY, STACK, BLOCK, Q8>};
}

template <int W, bool ANY, int STACK, bool Q8>
BatchKernel pick_block(int block) {
    if (block == 64) return make_kernel<W, ANY, STACK, 64, Q8>();
    if (block == 128) return make_kernel<W, ANY, STACK, 128, Q8>();
    if (block == 256) return make_kernel<W, ANY, STACK, 256, Q8>();
    return BatchKernel{nullptr, nullptr};
}

template <int W, bool ANY, bool Q8>
BatchKernel pick_stack(int stack, int block) {
    if (stack == 64) return pick_block<W, ANY, 64, Q8>(block);
    if (stack == 128) return pick_block<W, ANY, 128, Q8>(block);
    if (stack == 256) return pick_block<W, ANY, 256, Q8>(block);
    return BatchKernel{nullptr, nullptr};
}

template <int W>
BatchKernel pick_query(bool any, int stack, int block, bool q8) {
    if (any) return q8 ? pick_stack<W, true, true>(stack, block) : pick_stack<W, true, false>(stack, block);
    return q8 ? pick_stack<W, false, true>(stack, block) : pick_stack<W, false, false>(stack, block);
}

}  // namespace

BatchKernel batch_kernel(int width, bool any, int stack, int block, bool q8) {
    if (width == 8) return pick_query<8>(any, stack, block, q8);
    if (width == 4) return pick_query<4>(any, stack, block, q8);
    return BatchKernel{nullptr, nullptr};
}

cudaError_t launch_batch_begin(const RunHeader* header, const BatchDesc* batches, RunState* state,
                               unsigned long long* remaining, long long* done_ns, int max_batches, cudaStream_t s) {
    const int threads = 256;
    const int blocks = (max_batches + threads - 1) / threads;
    k_batch_begin<<<blocks < 1 ? 1 : blocks, threads, 0, s>>>(header, batches, state, remaining, done_ns);
    return cudaGetLastError();
}

}  // namespace sg
