// One wave of the wavefront path tracer (pt.cu): one or more samples for every
// pixel of a band, on caller-provided buffers. sg_pt_render_rows runs its waves
// on the render's own buffers; the render server (server.cpp) on its lanes'.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include <cstdint>

#include "pt_types.h"
#include "trace_kernels.h"

namespace sg {

// Waves sg_pt_render keeps in flight, each on its own buffers and streams.
constexpr int kInFlight = 2;

// Paths a wave of several samples holds at most: a small frame's samples share
// waves, because a wave of few paths is bound by its chain of dependent launches
// and by the latency of single rays, not by the work. One sample per wave against
// several: a 161x91 frame of 4 spp (four waves of 14,651 paths, or one of 58,604)
// 0.67 / 0.285 ms, 480x270 at 16 spp 6.03 / 2.16, a mix of 24 served renders
// (64x36 to 960x540, 1 to 16 spp) 28.7 / 12.9.
constexpr int64_t kWavePaths = int64_t(1) << 20;

// Paths a wave holds at most, and slots of a server's pool (serve_kernels.h): a
// shadow queue has two rays per path in eight planes, and the kernels find a place
// in it with an int. Larger frames go in several waves per sample.
constexpr int64_t kMaxWavePaths = int64_t(1) << 27;
static_assert(8 * (2 * kMaxWavePaths) - 1 <= INT32_MAX, "a place in the shadow queue's planes is an int");

// Samples per wave of a band of n pixels whose buffers hold cap paths.
inline int wave_samples(int64_t n, int64_t cap, int spp) {
    const int64_t most = (cap < kWavePaths ? cap : kWavePaths) / n;
    return most < 1 ? 1 : (most > spp ? spp : (int)most);
}

// Waves of `samples` samples each that spp samples take (any int: no sum of the two).
inline int wave_count(int spp, int samples) { return spp / samples + (spp % samples ? 1 : 0); }

// Queue lengths and ray counters of one bounce; bounce b uses entry b % 4 of the
// wave's kWaveCounts entries. Shading bounce b appends to entry b + 1 and clears
// entry b + 2, whose last users (bounce b - 2) are done, so that no memset or
// copy stands between two kernels.
struct WaveCount {
    int length;                  // extension rays
    int shadow;                  // shadow rays
    unsigned taken, shadow_taken;  // rays taken by the two traversals
};
constexpr int kWaveCounts = 4;

// A render of `pixels` pixels as waves: of `part` pixels (a frame too large for one
// wave goes in `parts` of them) and per_wave samples each, in_flight at once, each
// with its own set of buffers.
struct WavePlan {
    int part, parts, per_wave, in_flight;
    int64_t waves;
    size_t cap;    // paths of a set
    size_t bytes;  // of every set, and the ray totals
};
inline size_t wave_align(size_t x) { return (x + 255) & ~size_t(255); }
inline WavePlan wave_plan(int64_t pixels, int spp, int per_wave) {
    WavePlan w;
    w.part = (int)(pixels < kMaxWavePaths ? pixels : kMaxWavePaths);
    w.parts = (int)((pixels + w.part - 1) / w.part);
    w.per_wave = per_wave;
    w.waves = (int64_t)wave_count(spp, per_wave) * w.parts;
    w.in_flight = w.waves < kInFlight ? (int)w.waves : kInFlight;
    w.cap = (size_t)w.part * per_wave;
    const size_t cap = w.cap, scap = 2 * cap;
    // two extension queues (rays, paths), hits, the shadow queue (rays,
    // contributions), occlusion flags, throughput and radiance, shadow entries, counts
    const size_t set = 2 * (wave_align(cap * 32) + wave_align(cap * 4)) + 2 * wave_align(cap * 4) +
                       wave_align(scap * 32) + wave_align(scap * 12) + wave_align(scap) + wave_align(cap * 24) +
                       wave_align(cap * 8) + wave_align(kWaveCounts * sizeof(WaveCount));
    w.bytes = w.in_flight * set + wave_align(16);
    return w;
}

// The memory a scene's renders keep between them.
struct WaveBuffers {
    char* mem = nullptr;
    size_t bytes = 0;
    size_t most = SIZE_MAX;  // what samples sharing waves may take: less than what could not be had once
};

// Makes `buf` large enough for a render and says how it goes. Samples that share waves
// take up to 424 MB where a sample per wave takes 404 bytes per pixel, so beyond
// kAskBytes they get a sixteenth of the device's free memory at most and share by
// fewer where that, or what can be had, is less; the next render does not ask for it
// again, and the memory held is given up only for more, or where not even a sample per
// wave fits it. (Asking takes 70 to 100 us, a tenth of a small scene's first render.)
// Gpu: size_t free_bytes(), cudaError_t alloc(bytes, &mem), release(mem).
constexpr size_t kAskBytes = size_t(64) << 20;
template <class Gpu>
cudaError_t fit_wave_buffers(Gpu&& gpu, WaveBuffers& buf, int64_t pixels, int spp, WavePlan& plan) {
    for (int per_wave = wave_samples(pixels, kWavePaths, spp);; per_wave = (per_wave + 1) / 2) {
        plan = wave_plan(pixels, spp, per_wave);
        if (plan.bytes <= buf.bytes) return cudaSuccess;
        char* mem = nullptr;
        if (per_wave == 1) {
            if (buf.mem) gpu.release(buf.mem);
            buf.mem = nullptr;
            buf.bytes = 0;
            const cudaError_t e = gpu.alloc(plan.bytes, &mem);
            if (e != cudaSuccess) return e;
        } else {
            if (plan.bytes > buf.most) continue;
            if ((plan.bytes > kAskBytes && plan.bytes > gpu.free_bytes() / 16) ||
                gpu.alloc(plan.bytes, &mem) != cudaSuccess) {
                buf.most = plan.bytes - 1;
                continue;
            }
            if (buf.mem) gpu.release(buf.mem);
        }
        buf.mem = mem;
        buf.bytes = plan.bytes;
        return cudaSuccess;
    }
}

// Device buffers of a wave: two extension queues (8 floats per ray with stride
// cap, a path index per entry), the hits (cap each), the shadow queue (stride
// 2 * cap, three contribution planes) and its occlusion flags, per-path
// throughput and radiance (6 * cap floats) and the path's two shadow queue
// entries (2 * cap, -1: none), the counts and two ray totals (extension, shadow).
struct PtWave {
    float* qa_ray;
    int* qa_slot;
    float* qb_ray;
    int* qb_slot;
    float* sq_ray;
    float* sq_contrib;
    int32_t* hit_prim;
    float* hit_t;
    uint8_t* occ;
    float* thr;
    int* shadow_of;
    WaveCount* counts;  // kWaveCounts
    unsigned long long* totals;
    int cap;
    // Optional: a second stream on which each bounce's shadow rays run beside
    // the next bounce's extension rays, with two events for the hand-offs.
    cudaStream_t side;
    cudaEvent_t shaded, shadowed;
    // Optional: the radiance is added to the image only after `flush_after`
    // (the previous sample's addition, when samples run on several streams),
    // and `flush_done` is recorded after it.
    cudaEvent_t flush_after, flush_done;
};

// image[i] *= s for i < n (the 1/spp of a finished render), on stream st.
cudaError_t pt_scale(float* image, int64_t n, float s, cudaStream_t st);

// Samples sample .. sample + samples - 1 of pixels p0 .. p0 + n - 1 (n * samples
// <= w.cap) of a width x height frame: each pixel's radiance is added to
// image[3 * (p - p0) + c], sample after sample; nothing is zeroed or scaled.
// Every pixel draws the random numbers of its place in the frame, so waves over
// bands and over whole frames, of one sample or of several, give the same sums.
// `base` is the scene's launch (scene_launch), `tree` its tree.
cudaError_t pt_wave(const PtDev& dev, const TraceLaunch& base, const DevTree& tree, const Cam& cam, int width,
                    int height, int p0, int n, uint2 key, int sample, int samples, int max_depth, const PtWave& w,
                    float* image, cudaStream_t s);

}  // namespace sg
