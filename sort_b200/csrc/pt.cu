// Wavefront path tracer with SORT's PathTracing estimator (integrator/pathtracing.cpp:44-258).
//
// One wave traces one sample, of small frames several, for every pixel. Per bounce:
//   extend   closest-hit traversal of the compacted ray queue (trace.cu);
//   shade    for each hit: emission at the first vertex, next-event estimation
//            with both of EvaluateDirect's samples (integratormethod.cpp:100-192:
//            a light sample weighted by MIS against the BSDF, a BSDF sample that
//            hits the light weighted against the light), BSDF sampling of the
//            continuation, Russian roulette, all as PathTracing::li orders them;
//            shadow rays and the next rays are appended to compacted queues with
//            one atomic per warp;
//   shadow   any-hit traversal of the shadow queue;
//   accumulate  each path's unoccluded shadow contributions are added to its
//            radiance in a fixed order; at the end of the wave each path's
//            radiance is added to its pixel, sample after sample. Every sum has
//            one writer in a fixed order, so an image is bit-reproducible.
// Shading follows SORT's ScatteringEvent frame (scatteringevent.cpp:42-59) and
// BxDFs: Lambert (lambert.cpp:34-38), MicroFacetReflection with GGX and
// conductor Fresnel (microfacet.cpp:229-356, fresnel.h:119-130); the area light
// is SORT's AreaLight over a Quad (light/area.cpp, shape/quad.cpp), one-sided.
// Random numbers come from Philox4x32-10 (Salmon et al., SC'11), counter-based,
// keyed per render and indexed by (pixel, sample, bounce), so any schedule gives
// the same image. SORT draws from a Mersenne Twister seeded with the wall clock
// (core/rand.cpp:41-55), so images agree in distribution, not sample by sample.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "pt_common.cuh"
#include "pt_wave.h"
#include "scene_access.h"
#include "trace_kernels.h"

namespace sg {
namespace {

// A wave's paths: path p renders sample `sample` + p / n of frame pixel
// p0 + p % n (a band of whole rows starts at p0).
struct WavePixels {
    int p0, n;
    uint32_t sample;
    __device__ __forceinline__ int pixel(int p, uint32_t& smp) const {
        const int k = p < n ? 0 : p / n;
        smp = sample + (uint32_t)k;
        return p0 + (p - k * n);
    }
};

__global__ void k_generate(Cam cam, int width, int height, WavePixels px, int paths, uint2 key, Queue q, int cap,
                           float* __restrict__ thr, WaveCount* __restrict__ counts) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= paths) return;
    uint32_t sample;
    const int pixel = px.pixel(p, sample);
    put_ray(q.ray, cap, p, cam.eye, camera_dir(cam, width, height, pixel, key, sample), 0.0f, FLT_MAX);
    q.slot[p] = p;
    thr[p] = thr[cap + p] = thr[2 * cap + p] = 1.0f;          // throughput
    thr[3 * cap + p] = thr[4 * cap + p] = thr[5 * cap + p] = 0.0f;  // radiance of this sample
    if (p == 0) {
        counts[0] = WaveCount{paths, 0, 0, 0};
        counts[1] = WaveCount{0, 0, 0, 0};
    }
}

__global__ void k_shade(PtDev sc, uint2 key, WavePixels px, int bounce, int max_depth, Queue in, int cap,
                        WaveCount* __restrict__ counts, const int32_t* __restrict__ hit_prim,
                        const float* __restrict__ hit_t, Queue next, Queue shadow, int shadow_cap,
                        float* __restrict__ thr, int* __restrict__ shadow_of) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q == 0) counts[(bounce + 2) % kWaveCounts] = WaveCount{0, 0, 0, 0};
    if (q >= counts[bounce % kWaveCounts].length) return;
    const int p = in.slot[q];
    const int prim = hit_prim[q];
    Vertex v;
    if (prim >= 0) {
        const float3 o = f3(in.ray[q], in.ray[cap + q], in.ray[2 * cap + q]);
        const float3 d = f3(in.ray[3 * cap + q], in.ray[4 * cap + q], in.ray[5 * cap + q]);
        uint32_t sample;
        const int pixel = px.pixel(p, sample);
        v = shade_vertex(sc, key, (uint32_t)pixel, sample, bounce, max_depth, o, d, prim, hit_t[q],
                         f3(thr[p], thr[cap + p], thr[2 * cap + p]));
        if (v.emit) {
            thr[3 * cap + p] += v.Le.x;
            thr[4 * cap + p] += v.Le.y;
            thr[5 * cap + p] += v.Le.z;
        }
        if (v.new_T) {
            thr[p] = v.T.x;
            thr[cap + p] = v.T.y;
            thr[2 * cap + p] = v.T.z;
        }
    }
    const bool s1 = v.s1, s2 = v.s2, cont = v.cont;
    const float3 X = v.X, wi1 = v.wi1, wi2 = v.wi2, c1 = v.c1, c2 = v.c2, wi_next = v.wi_next;
    const float len1 = v.len1, t2 = v.t2;
    int* shadow_count = &counts[bounce % kWaveCounts].shadow;
    const int i1 = warp_append(shadow_count, s1);  // light-sample ray
    shadow_of[p] = i1;
    if (i1 >= 0) {
        put_ray(shadow.ray, shadow_cap, i1, X, wi1, 0.01f, len1 - 0.01f);
        shadow.contrib[i1] = c1.x;
        shadow.contrib[shadow_cap + i1] = c1.y;
        shadow.contrib[2 * shadow_cap + i1] = c1.z;
    }
    const int i2 = warp_append(shadow_count, s2);  // BSDF-sample ray
    shadow_of[cap + p] = i2;
    if (i2 >= 0) {
        put_ray(shadow.ray, shadow_cap, i2, X, wi2, 0.001f, t2 - 0.001f);
        shadow.contrib[i2] = c2.x;
        shadow.contrib[shadow_cap + i2] = c2.y;
        shadow.contrib[2 * shadow_cap + i2] = c2.z;
    }
    const int in_next = warp_append(&counts[(bounce + 1) % kWaveCounts].length, cont);
    if (in_next >= 0) {
        put_ray(next.ray, cap, in_next, X, wi_next, 0.0001f, FLT_MAX);
        next.slot[in_next] = p;
    }
}

// EvaluateDirect's two terms (light sample, then BSDF sample; an occluded or
// absent ray's is zero) are added to the path's radiance in SORT's order, for
// every path shaded this bounce. Adding two zeros would change nothing, so such
// paths are passed over. Also counts the bounce's rays.
__global__ void k_accumulate(Queue in, const WaveCount* __restrict__ count, const int* __restrict__ shadow_of,
                             const uint8_t* __restrict__ occ, const float* __restrict__ contrib, int shadow_cap,
                             float* __restrict__ thr, int cap, unsigned long long* __restrict__ totals) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q == 0) {  // waves of two samples may count at once
        atomicAdd(&totals[0], (unsigned long long)count->length);
        atomicAdd(&totals[1], (unsigned long long)count->shadow);
    }
    if (q >= count->length) return;
    const int p = in.slot[q];
    const int i1 = shadow_of[p], i2 = shadow_of[cap + p];
    const bool lit1 = i1 >= 0 && !occ[i1], lit2 = i2 >= 0 && !occ[i2];
    if (!lit1 && !lit2) return;
#pragma unroll
    for (int c = 0; c < 3; ++c)
        thr[(3 + c) * cap + p] +=
            (lit1 ? contrib[c * shadow_cap + i1] : 0.0f) + (lit2 ? contrib[c * shadow_cap + i2] : 0.0f);
}

// End of a wave: each pixel's sample radiances go into the image, sample after
// sample (one writer).
__global__ void k_flush(const float* __restrict__ thr, int cap, int n, int samples, float* __restrict__ image) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        float sum = image[3 * p + c];
        for (int k = 0; k < samples; ++k) sum += thr[(3 + c) * cap + k * n + p];
        image[3 * p + c] = sum;
    }
}

__global__ void k_scale(float* __restrict__ image, int n, float s) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) image[i] *= s;
}

__global__ void k_zero(float* __restrict__ image, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) image[i] = 0.0f;
}

}  // namespace
}  // namespace sg

struct sg_pt_scene {
    const sg_scene* scene = nullptr;
    int device = 0;
    float4* d_prim = nullptr;
    sg::PtMaterial* d_mats = nullptr;
    sg::PtLight light{};
    // Per-render buffers, grown on demand.
    sg::WaveBuffers buf;
    unsigned long long* d_totals = nullptr;  // rays traced by the last render: extension, shadow
    // kInFlight waves are in flight at once, each with its own buffers:
    // wave k runs on the caller's stream (k % kInFlight == 0) or on
    // extra[k % kInFlight], its shadow rays on side[k % kInFlight]
    // (pt_wave.h); the events order the hand-offs and the image additions.
    // Made by the first render.
    cudaStream_t extra[sg::kInFlight] = {};  // [0] unused: the caller's stream
    cudaStream_t side[sg::kInFlight] = {};
    cudaEvent_t shaded[sg::kInFlight] = {}, shadowed[sg::kInFlight] = {}, flushed[sg::kInFlight] = {};
    cudaEvent_t begun = nullptr;
};

extern "C" sg_status sg_pt_ray_counts(const sg_pt_scene* ps, int64_t* extension, int64_t* shadow, void* stream) {
    if (!ps || !extension || !shadow) return sg::set_error(SG_ERR_INVALID_ARGUMENT, "NULL argument");
    *extension = *shadow = 0;
    if (!ps->d_totals) return SG_OK;
    unsigned long long h[2] = {0, 0};
    cudaError_t e = cudaMemcpyAsync(h, ps->d_totals, sizeof(h), cudaMemcpyDeviceToHost, (cudaStream_t)stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize((cudaStream_t)stream);
    if (e != cudaSuccess) return sg::set_error(SG_ERR_CUDA, cudaGetErrorString(e));
    *extension = (int64_t)h[0];
    *shadow = (int64_t)h[1];
    return SG_OK;
}

namespace {

// The device's memory, as fit_wave_buffers asks for it.
struct RenderMemory {
    size_t free_bytes() const {
        size_t free = 0, total = 0;
        return cudaMemGetInfo(&free, &total) == cudaSuccess ? free : 0;
    }
    cudaError_t alloc(size_t bytes, char** mem) const {
        const cudaError_t e = cudaMalloc(mem, bytes);
        if (e == cudaErrorMemoryAllocation) (void)cudaGetLastError();  // the caller handles it; no launch check may see it
        return e;
    }
    void release(char* mem) const { cudaFree(mem); }
};

sg_status pt_fail(cudaError_t e) { return sg::set_error(SG_ERR_CUDA, cudaGetErrorString(e)); }

}  // namespace

namespace sg {

// Perspective pinhole, as the oracle harness builds SORT's PerspectiveCamera.
Cam make_camera(const float* camera, int width, int height) {
    Cam cam;
    const float3 eye = make_float3(camera[0], camera[1], camera[2]);
    float3 fwd = make_float3(camera[3] - eye.x, camera[4] - eye.y, camera[5] - eye.z);
    const float fl = std::sqrt(fwd.x * fwd.x + fwd.y * fwd.y + fwd.z * fwd.z);
    fwd = make_float3(fwd.x / fl, fwd.y / fl, fwd.z / fl);
    const float3 up = make_float3(camera[6], camera[7], camera[8]);
    float3 right = make_float3(fwd.y * up.z - fwd.z * up.y, fwd.z * up.x - fwd.x * up.z, fwd.x * up.y - fwd.y * up.x);
    const float rl = std::sqrt(right.x * right.x + right.y * right.y + right.z * right.z);
    right = make_float3(right.x / rl, right.y / rl, right.z / rl);
    const float3 upv = make_float3(right.y * fwd.z - right.z * fwd.y, right.z * fwd.x - right.x * fwd.z,
                                   right.x * fwd.y - right.y * fwd.x);
    cam.eye = eye;
    cam.fwd = fwd;
    cam.right = right;
    cam.up = upv;
    cam.half_h = std::tan(camera[9] * 3.14159265358979f / 180.0f * 0.5f);
    cam.half_w = cam.half_h * (float)width / (float)height;
    return cam;
}

sg_status pt_scene_parts(const sg_pt_scene* ps, PtDev* dev, const sg_scene** scene) {
    if (!ps || !dev || !scene) return set_error(SG_ERR_INVALID_ARGUMENT, "NULL path-tracing scene");
    *dev = PtDev{ps->d_prim, ps->d_mats, ps->light};
    *scene = ps->scene;
    return SG_OK;
}

}  // namespace sg

extern "C" sg_status sg_pt_create(const sg_scene* scene, const float* triangles, int64_t ntri, const int32_t* mat_of_tri,
                                  const float* materials, int32_t nmat, const float* light, sg_pt_scene** out) {
    if (!scene || !out || !light || (ntri > 0 && (!triangles || !mat_of_tri)) || nmat < 0 || (nmat > 0 && !materials))
        return sg::set_error(SG_ERR_INVALID_ARGUMENT, "bad path-tracing scene description");
    *out = nullptr;
    sg::TraceLaunch L;
    sg::DevTree tree;
    int device = 0;
    sg_status st = sg::scene_launch(scene, false, &L, &tree, &device);
    if (st != SG_OK) return st;
    std::vector<float4> prim((size_t)std::max<int64_t>(ntri, 1));
    for (int64_t i = 0; i < ntri; ++i) {
        const float* v = triangles + i * 9;
        // SORT's geometric normal, cross(v2 - v0, v1 - v0) normalised (simd_triangle.h:331)
        const float ax = v[6] - v[0], ay = v[7] - v[1], az = v[8] - v[2];
        const float bx = v[3] - v[0], by = v[4] - v[1], bz = v[5] - v[2];
        float nx = ay * bz - az * by, ny = az * bx - ax * bz, nz = ax * by - ay * bx;
        const float len = std::sqrt(nx * nx + ny * ny + nz * nz);
        if (len > 0.0f) {
            nx /= len;
            ny /= len;
            nz /= len;
        } else {
            nx = 0.0f;
            ny = 1.0f;
            nz = 0.0f;
        }
        const int32_t mid = mat_of_tri[i];
        if (mid >= nmat) return sg::set_error(SG_ERR_INVALID_ARGUMENT, "material index out of range");
        float w;
        std::memcpy(&w, &mid, 4);
        prim[(size_t)i] = make_float4(nx, ny, nz, w);
    }
    std::vector<sg::PtMaterial> mats((size_t)std::max(nmat, 1));
    for (int m = 0; m < nmat; ++m) {
        const float* q = materials + (size_t)m * 10;
        sg::PtMaterial pm{};
        pm.type = (int)q[0];
        if (pm.type != 0 && pm.type != 1) return sg::set_error(SG_ERR_INVALID_ARGUMENT, "unknown material type");
        for (int c = 0; c < 3; ++c) {
            pm.a[c] = q[1 + c];
            pm.k[c] = q[4 + c];
        }
        pm.rough = q[7];
        mats[(size_t)m] = pm;
    }
    auto* ps = new sg_pt_scene();
    ps->scene = scene;
    ps->device = device;
    for (int c = 0; c < 3; ++c) {
        ps->light.c[c] = light[c];
        ps->light.I[c] = light[5 + c];
    }
    ps->light.hx = light[3] * 0.5f;
    ps->light.hz = light[4] * 0.5f;
    ps->light.area = light[3] * light[4];
    int prev = -1;
    cudaGetDevice(&prev);
    cudaError_t e = cudaSetDevice(device);
    if (e == cudaSuccess) e = cudaMalloc(&ps->d_prim, prim.size() * sizeof(float4));
    if (e == cudaSuccess) e = cudaMalloc(&ps->d_mats, mats.size() * sizeof(sg::PtMaterial));
    if (e == cudaSuccess) e = cudaMemcpy(ps->d_prim, prim.data(), prim.size() * sizeof(float4), cudaMemcpyHostToDevice);
    if (e == cudaSuccess)
        e = cudaMemcpy(ps->d_mats, mats.data(), mats.size() * sizeof(sg::PtMaterial), cudaMemcpyHostToDevice);
    if (prev >= 0) cudaSetDevice(prev);
    if (e != cudaSuccess) {
        sg_pt_destroy(ps);
        return pt_fail(e);
    }
    *out = ps;
    return SG_OK;
}

extern "C" sg_status sg_pt_destroy(sg_pt_scene* ps) {
    if (!ps) return SG_OK;
    int prev = -1;
    cudaGetDevice(&prev);
    cudaSetDevice(ps->device);
    if (ps->d_prim) cudaFree(ps->d_prim);
    if (ps->d_mats) cudaFree(ps->d_mats);
    if (ps->buf.mem) cudaFree(ps->buf.mem);
    for (int k = 0; k < sg::kInFlight; ++k) {
        for (cudaStream_t t : {ps->extra[k], ps->side[k]})
            if (t) {
                cudaStreamSynchronize(t);
                cudaStreamDestroy(t);
            }
        for (cudaEvent_t ev : {ps->shaded[k], ps->shadowed[k], ps->flushed[k]})
            if (ev) cudaEventDestroy(ev);
    }
    if (ps->begun) cudaEventDestroy(ps->begun);
    if (prev >= 0) cudaSetDevice(prev);
    delete ps;
    return SG_OK;
}

namespace sg {

cudaError_t pt_scale(float* image, int64_t n, float s, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    if (n > int64_t(1) << 30) return cudaErrorInvalidValue;
    k_scale<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(image, (int)n, s);
    return cudaGetLastError();
}

cudaError_t pt_wave(const PtDev& dev, const TraceLaunch& base_in, const DevTree& tree, const Cam& cam, int width,
                    int height, int p0, int n, uint2 key, int sample, int samples, int max_depth, const PtWave& w,
                    float* image, cudaStream_t s) {
    if (n <= 0 || samples <= 0 || (int64_t)n * samples > w.cap || w.cap > kMaxWavePaths) return cudaErrorInvalidValue;
    const int cap = w.cap, scap = 2 * w.cap;
    const int paths = n * samples;
    TraceLaunch base = base_in;
    base.tuning.schedule = kScheduleThreadPerRay;  // queue lengths live on the device
    Queue qa{w.qa_ray, w.qa_slot, nullptr}, qb{w.qb_ray, w.qb_slot, nullptr};
    const Queue sq{w.sq_ray, nullptr, w.sq_contrib};
    const WavePixels px{p0, n, (uint32_t)sample};
    const int threads = 256;
    const int blocks = (paths + threads - 1) / threads;
    cudaError_t e = cudaSuccess;
    Queue* cur = &qa;
    Queue* nxt = &qb;
    auto closest = [&](const Queue* q, WaveCount* count) {
        DevRays r{q->ray,           q->ray + cap,     q->ray + 2 * cap, q->ray + 3 * cap,
                  q->ray + 4 * cap, q->ray + 5 * cap, q->ray + 6 * cap, q->ray + 7 * cap};
        TraceLaunch Lc = base;
        Lc.any = false;
        Lc.prim = w.hit_prim;
        Lc.t = w.hit_t;
        Lc.n_dev = &count->length;
        Lc.counter = &count->taken;
        return launch_trace_fp32(Lc, tree, r, (int64_t)paths, s);
    };
    // Shadow rays of bounce `cur` and its paths' radiance on stream t.
    auto shadows = [&](const Queue* q, WaveCount* count, cudaStream_t t) {
        DevRays sr{sq.ray,            sq.ray + scap,     sq.ray + 2 * scap, sq.ray + 3 * scap,
                   sq.ray + 4 * scap, sq.ray + 5 * scap, sq.ray + 6 * scap, sq.ray + 7 * scap};
        TraceLaunch La = base;
        La.any = true;
        La.occ = w.occ;
        La.n_dev = &count->shadow;
        La.counter = &count->shadow_taken;
        cudaError_t r = launch_trace_fp32(La, tree, sr, 2 * (int64_t)paths, t);
        if (r != cudaSuccess) return r;
        k_accumulate<<<blocks, threads, 0, t>>>(*q, count, w.shadow_of, w.occ, sq.contrib, scap, w.thr, cap, w.totals);
        return cudaGetLastError();
    };
    k_generate<<<blocks, threads, 0, s>>>(cam, width, height, px, paths, key, *cur, cap, w.thr, w.counts);
    if ((e = closest(cur, &w.counts[0])) != cudaSuccess) return e;
    for (int bounce = 0; bounce < max_depth; ++bounce) {
        WaveCount* count = &w.counts[bounce % kWaveCounts];
        k_shade<<<blocks, threads, 0, s>>>(dev, key, px, bounce, max_depth, *cur, cap, w.counts, w.hit_prim, w.hit_t,
                                           *nxt, sq, scap, w.thr, w.shadow_of);
        if (!w.side) {
            if ((e = shadows(cur, count, s)) != cudaSuccess) return e;
        } else {
            // The shadow rays of this bounce go to the side stream and run
            // beside the next bounce's extension rays; the next shading (which
            // reuses the shadow queue and the path state) waits for them.
            if ((e = cudaEventRecord(w.shaded, s)) != cudaSuccess ||
                (e = cudaStreamWaitEvent(w.side, w.shaded, 0)) != cudaSuccess ||
                (e = shadows(cur, count, w.side)) != cudaSuccess ||
                (e = cudaEventRecord(w.shadowed, w.side)) != cudaSuccess)
                return e;
        }
        std::swap(cur, nxt);  // the next queue becomes the current one
        if (bounce + 1 < max_depth && (e = closest(cur, &w.counts[(bounce + 1) % kWaveCounts])) != cudaSuccess)
            return e;
        if (w.side && (e = cudaStreamWaitEvent(s, w.shadowed, 0)) != cudaSuccess) return e;
    }
    if (w.flush_after && (e = cudaStreamWaitEvent(s, w.flush_after, 0)) != cudaSuccess) return e;
    k_flush<<<(n + threads - 1) / threads, threads, 0, s>>>(w.thr, cap, n, samples, image);
    if (w.flush_done && (e = cudaEventRecord(w.flush_done, s)) != cudaSuccess) return e;
    return cudaGetLastError();
}

}  // namespace sg

extern "C" sg_status sg_pt_render(sg_pt_scene* ps, const float* camera, int32_t width, int32_t height, int32_t spp,
                                  int32_t max_depth, uint64_t seed, float* image, void* stream) {
    return sg_pt_render_rows(ps, camera, width, height, 0, height, spp, max_depth, seed, image, stream);
}

extern "C" sg_status sg_pt_render_rows(sg_pt_scene* ps, const float* camera, int32_t width, int32_t height,
                                       int32_t row_begin, int32_t row_end, int32_t spp, int32_t max_depth,
                                       uint64_t seed, float* image, void* stream) {
    if (!ps || !camera || !image || width <= 0 || height <= 0 || spp <= 0 || max_depth <= 0)
        return sg::set_error(SG_ERR_INVALID_ARGUMENT, "bad render arguments");
    if ((int64_t)width * height > (int64_t)1 << 28) return sg::set_error(SG_ERR_LIMIT, "image too large");
    if (row_begin < 0 || row_end > height || row_begin >= row_end)
        return sg::set_error(SG_ERR_INVALID_ARGUMENT, "bad row range");
    const int P = width * (row_end - row_begin);  // pixels of the band
    const int p0 = width * row_begin;
    sg::TraceLaunch base;
    sg::DevTree tree;
    int device = 0;
    sg_status st = sg::scene_launch(ps->scene, false, &base, &tree, &device);
    if (st != SG_OK) return st;
    base.tuning.schedule = sg::kScheduleThreadPerRay;  // queue lengths live on the device
    int prev = -1;
    cudaGetDevice(&prev);
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) return pt_fail(e);
    struct Restore {
        int dev;
        ~Restore() {
            if (dev >= 0) cudaSetDevice(dev);
        }
    } restore{prev};
    cudaStream_t s = (cudaStream_t)stream;

    ps->d_totals = nullptr;  // until this render's buffers stand
    sg::WavePlan plan;
    if ((e = sg::fit_wave_buffers(RenderMemory{}, ps->buf, P, spp, plan)) != cudaSuccess) return pt_fail(e);
    const int part = plan.part, parts = plan.parts, per_wave = plan.per_wave, in_flight = plan.in_flight;
    const int64_t waves = plan.waves;
    const size_t cap = plan.cap, scap = 2 * cap;
    char* b = ps->buf.mem;
    auto take = [&](size_t bytes) {
        char* r = b;
        b += sg::wave_align(bytes);
        return r;
    };
    bool made = true;
    for (int k = 0; k < sg::kInFlight; ++k) {
        for (cudaStream_t* t : {&ps->extra[k], &ps->side[k]})
            if (t != &ps->extra[0])
                made = made && (*t || cudaStreamCreateWithFlags(t, cudaStreamNonBlocking) == cudaSuccess);
        for (cudaEvent_t* ev : {&ps->shaded[k], &ps->shadowed[k], &ps->flushed[k]})
            made = made && (*ev || cudaEventCreateWithFlags(ev, cudaEventDisableTiming) == cudaSuccess);
    }
    made = made && (ps->begun || cudaEventCreateWithFlags(&ps->begun, cudaEventDisableTiming) == cudaSuccess);
    if (!made) return sg::set_error(SG_ERR_CUDA, "render streams and events");
    sg::PtWave w[sg::kInFlight] = {};
    for (int k = 0; k < in_flight; ++k) {
        w[k].qa_ray = (float*)take(cap * 32);
        w[k].qa_slot = (int*)take(cap * 4);
        w[k].qb_ray = (float*)take(cap * 32);
        w[k].qb_slot = (int*)take(cap * 4);
        w[k].hit_prim = (int32_t*)take(cap * 4);
        w[k].hit_t = (float*)take(cap * 4);
        w[k].sq_ray = (float*)take(scap * 32);
        w[k].sq_contrib = (float*)take(scap * 12);
        w[k].occ = (uint8_t*)take(scap);
        w[k].thr = (float*)take(cap * 24);    // throughput and radiance per path
        w[k].shadow_of = (int*)take(cap * 8);  // two shadow queue entries per path
        w[k].counts = (sg::WaveCount*)take(sg::kWaveCounts * sizeof(sg::WaveCount));
        w[k].cap = (int)cap;
        w[k].side = ps->side[k];
        w[k].shaded = ps->shaded[k];
        w[k].shadowed = ps->shadowed[k];
        w[k].flush_done = ps->flushed[k];
    }
    unsigned long long* totals = (unsigned long long*)take(16);  // rays traced: extension, shadow
    if ((size_t)(b - ps->buf.mem) > plan.bytes) return sg::set_error(SG_ERR_INTERNAL, "render buffer layout overflow");
    for (sg::PtWave& x : w) x.totals = totals;
    ps->d_totals = totals;
    if ((e = cudaMemsetAsync(totals, 0, 16, s)) != cudaSuccess) return pt_fail(e);

    const sg::Cam cam = sg::make_camera(camera, width, height);
    const uint2 key = make_uint2((uint32_t)seed, (uint32_t)(seed >> 32));
    sg::PtDev dev{ps->d_prim, ps->d_mats, ps->light};
    const int threads = 256;
    const int img_n = 3 * P;
    sg::k_zero<<<(img_n + threads - 1) / threads, threads, 0, s>>>(image, img_n);
    // The other streams start after everything the caller put on `stream`.
    if ((e = cudaEventRecord(ps->begun, s)) != cudaSuccess) return pt_fail(e);
    for (int k = 1; k < sg::kInFlight; ++k)
        if ((e = cudaStreamWaitEvent(ps->extra[k], ps->begun, 0)) != cudaSuccess) return pt_fail(e);
    for (int64_t k = 0; k < waves; ++k) {
        const int set = int(k % sg::kInFlight), first = int(k / parts) * per_wave, from = int(k % parts) * part;
        sg::PtWave& ws = w[set];
        ws.flush_after = k > 0 ? ps->flushed[(k - 1) % sg::kInFlight] : nullptr;  // image sums in order
        const cudaStream_t on = set ? ps->extra[set] : s;
        if ((e = sg::pt_wave(dev, base, tree, cam, width, height, p0 + from, std::min(part, P - from), key, first,
                             std::min(per_wave, spp - first), max_depth, ws, image + 3 * (int64_t)from, on)) !=
            cudaSuccess)
            return pt_fail(e);
    }
    // Every stream's work is done before the scale: the last addition closes
    // the chain, and every other stream's last wave precedes it.
    if ((e = cudaStreamWaitEvent(s, ps->flushed[(waves - 1) % sg::kInFlight], 0)) != cudaSuccess) return pt_fail(e);
    sg::k_scale<<<(img_n + threads - 1) / threads, threads, 0, s>>>(image, img_n, 1.0f / (float)spp);
    if ((e = cudaGetLastError()) != cudaSuccess) return pt_fail(e);
    return SG_OK;
}
