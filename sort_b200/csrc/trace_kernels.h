// Host-side launch wrappers of the traversal kernels (implemented in trace.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "layout.h"

namespace sg {

constexpr int kScheduleThreadPerRay = 0;  // rays taken in batch order
constexpr int kSchedulePersistent = 1;    // the same, refilling at tuning.refill_threshold idle lanes
constexpr int kScheduleWhileWhile = 2;    // as 0
constexpr int kScheduleSpeculative = 3;   // as 0
constexpr int kScheduleSorted = 4;        // rays taken in the order of a coherence key
constexpr int kScheduleAuto = 5;          // batch order

struct TraceTuning {
    int schedule = kScheduleAuto;
    int refill_threshold = 8;  // persistent schedule: idle lanes of a warp that trigger a refill (1..32)
};

struct TraceLaunch {
    int width = 8;
    bool any = false;
    int stack_need = 1;  // depth * (width - 1) + 1, the deepest the stack can grow
    TraceTuning tuning;
    int32_t* prim = nullptr;
    float* t = nullptr;
    float* u = nullptr;
    float* v = nullptr;
    uint8_t* occ = nullptr;
    int* err = nullptr;
    unsigned long long* stats = nullptr;  // non-null: also accumulate SORT's traversal counters
    unsigned* counter = nullptr;  // zero when the launch starts: warps take rays from it (null: the launch finds its own)
    bool scratch = true;          // the launch may take stream-ordered scratch from the library's pool
    const int* n_dev = nullptr;   // if set, the batch is min(n, *n_dev), n <= 2^30; needs a counter (not in counting launches)
    bool q8 = false;             // interior nodes in the 8-bit format
};

cudaError_t launch_trace_fp32(const TraceLaunch& L, const DevTree& tr, const DevRays& rays, int64_t n,
                              cudaStream_t s);
}  // namespace sg
