// Warp-cooperative wide-BVH traversal: the closest-hit / any-hit walk of the
// hot kernels.
//
// Restates Fbvh::GetIntersect (accel/fast_bvh.hpp:305-504, SIMD branch) ray by
// ray: the visit order, the culling, the leaf order and the rounding of every
// operation that decides a hit are those of Traversal (traversal.cuh), so the
// hits, distances and barycentrics are the same bits.
//
// What bounds it and why it has this form. A ray visits about 13.7 nodes and
// 3.3 leaves of 5.8 triangles (21M triangles, OBVH, diffuse rays), and with one
// ray per lane from start to end the lanes of a warp part ways: 14 lanes are busy
// in a node visit, 5 in a leaf, a leaf runs as long as its largest, and 32 rays take
// 26.0k warp instructions at 7.7 lanes. Here:
//  * a leaf is tested by eight lanes at once, whichever lanes own the rays, so
//    one round of instructions tests four leaves (35 rounds per 32 rays in place
//    of 20 leaf steps of up to 8 triangles each); the rays' triangle-test
//    constants and nearest hits lie in shared memory for that;
//  * a leaf reached in a step is tested in the same step;
//  * lanes whose ray is finished take new rays together once enough of them are
//    idle, so the node visits run with 25 lanes;
//  * a node's children go through packed FP32 pairs, one 32-byte load per plane,
//    and the two nearest hits stay in registers (a push is a predicated store).
// That issues 11.5k instructions per 32 rays at 24.6 lanes (shadow rays 10.2k at
// 25.9). Issue slots are then 60% busy and the L1 data pipe is at 73% of its peak
// (shadow 83%: a divergent 32-byte load per plane and lane, 48 bytes per
// triangle), with 4.7 warps waiting on loads per issue (5.8); DRAM is at 2%.
// One ray per lane against this form, one box: 4,194,304 diffuse rays, 21M triangles,
// 3.93 ms in sorted order, 2.15 in batch order; as many shadow rays 3.61 / 2.05;
// 1,048,576 camera rays, 82k triangles, width 4, 0.255 / 0.176; 700,001 diffuse rays,
// 1.3M triangles, 8-bit nodes 0.744 / 0.323.
// Slower forms: a second round's triangles fetched ahead (52 bytes spilled,
// 2.99 ms on the diffuse rays against 2.66), every hit but the nearest pushed and
// sorted on the stack (2.98), the 1/d and -o/d pairs kept doubled in registers
// (2.78), child references loaded after the box tests (3.2 against 3.18).
#pragma once

#include <cuda_runtime.h>

#include <type_traits>

#include "trace_common.cuh"

namespace sg {

constexpr unsigned kFullWarp = 0xffffffffu;
constexpr int kWalkThreads = 128;            // threads per block of the kernels over walk_rays
constexpr int kWalkWarps = kWalkThreads / 32;
constexpr uint32_t kWalkRayMask = (1u << 30) - 1u;  // ray index in WalkShared::ray
constexpr int kLeafLanes = 8;                // lanes that test one leaf's triangles at once
constexpr int kRoundLeaves = 32 / kLeafLanes;  // leaves tested at once
static_assert(kLeafLanes <= kPadSlots, "a leaf's lanes may read past its last slot");

// -0.0 twice, in constant memory so that the compiler cannot see the value:
// fma(a, b, -0) is then a product rounded once, packed, that cannot be
// contracted with the addition after it (mul.rn.f32x2 followed by add.rn.f32x2
// is contracted, which changed 2 of 524,288 hits against SORT).
static __constant__ float2 c_neg_zero2 = {-0.0f, -0.0f};

typedef unsigned long long f32x2;  // two floats, the first in the low half

__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// 32 bytes of a node: one sector, one load.
struct Load32 {
    f32x2 w[4];
};
__device__ __forceinline__ Load32 load32(const char* p) {
    Load32 r;
    asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];"
        : "=l"(r.w[0]), "=l"(r.w[1]), "=l"(r.w[2]), "=l"(r.w[3])
        : "l"(p));
    return r;
}

// The traversal stack: entries in the thread's local memory, addressed by
// their local-space address, so that a push is one predicated store and one
// predicated add (written as C++ the compiler branches around each push).
__device__ __forceinline__ void stack_put(uint32_t at, int32_t ref, float d) {
    asm volatile("st.local.v2.b32 [%0], {%1, %2};" ::"r"(at), "r"(ref), "f"(d));
}
__device__ __forceinline__ void stack_get(uint32_t at, int32_t& ref, float& d) {
    asm volatile("ld.local.v2.b32 {%0, %1}, [%2];" : "=r"(ref), "=f"(d) : "r"(at));
}
__device__ __forceinline__ void stack_get(uint32_t at, int32_t& ref) {
    asm volatile("ld.local.b32 %0, [%1];" : "=r"(ref) : "r"(at));
}

// tri_test (trace_common.cuh) in two parts, for a ray given by its shared
// record: the same operations on the same values; the axes are permuted with
// two predicates, and nothing branches.
struct TriEdges {
    float e0, e1, e2, y0, y1, y2;  // edge functions; the vertices' coordinates on the major axis
};
// Whether the edge functions are all >= 0 or all <= 0 (a NaN among them may
// pass; the distance test then fails).
__device__ __forceinline__ bool walk_tri_edges(const float4& c0, float sz, uint32_t ly, const float4& a,
                                               const float4& b, const float4& c, TriEdges& e) {
    const bool y0 = ly == 0, y1 = ly == 1;  // y = 0: x, z = 2, 1; y = 1: 0, 2; y = 2: 1, 0
    auto perm = [&](const float4& p, float& x, float& y, float& z) {
        x = __fsub_rn(y0 ? p.z : (y1 ? p.x : p.y), c0.x);
        y = __fsub_rn(y0 ? p.x : (y1 ? p.y : p.z), c0.y);
        z = __fsub_rn(y0 ? p.y : (y1 ? p.z : p.x), c0.z);
    };
    float ax, az, bx, bz, cx, cz;
    perm(a, ax, e.y0, az);
    perm(b, bx, e.y1, bz);
    perm(c, cx, e.y2, cz);
    ax = __fadd_rn(__fmul_rn(e.y0, c0.w), ax);
    az = __fadd_rn(__fmul_rn(e.y0, sz), az);
    bx = __fadd_rn(__fmul_rn(e.y1, c0.w), bx);
    bz = __fadd_rn(__fmul_rn(e.y1, sz), bz);
    cx = __fadd_rn(__fmul_rn(e.y2, c0.w), cx);
    cz = __fadd_rn(__fmul_rn(e.y2, sz), cz);
    e.e0 = __fsub_rn(__fmul_rn(bx, cz), __fmul_rn(bz, cx));
    e.e1 = __fsub_rn(__fmul_rn(cx, az), __fmul_rn(cz, ax));
    e.e2 = __fsub_rn(__fmul_rn(ax, bz), __fmul_rn(az, bx));
    return fminf(fminf(e.e0, e.e1), e.e2) >= 0.0f || fmaxf(fmaxf(e.e0, e.e1), e.e2) <= 0.0f;
}
// Distance and barycentrics of a triangle whose edges passed.
__device__ __forceinline__ bool walk_tri_hit(const TriEdges& e, bool pass, float sy, float tmin, float tmax, float& t,
                                             float& u, float& v) {
    const float det = __fadd_rn(e.e0, __fadd_rn(e.e1, e.e2));
    const float rcp_det = __frcp_rn(pass ? det : 1.0f);
    t = __fmul_rn(e.e0, __fmul_rn(e.y0, sy));
    t = __fadd_rn(__fmul_rn(e.e1, __fmul_rn(e.y1, sy)), t);
    t = __fadd_rn(__fmul_rn(e.e2, __fmul_rn(e.y2, sy)), t);
    t = __fmul_rn(t, rcp_det);
    u = __fmul_rn(e.e1, rcp_det);
    v = __fmul_rn(e.e2, rcp_det);
    return pass && det != 0.0f && t > tmin && t <= tmax;
}

// One warp's shared state, indexed by the lane that owns the ray.
struct WalkShared {
    float4 c0[32];   // origin x, y, z in the ray's permuted frame, shear x
    float4 c1[32];   // shear z, shear y, tmin, tmax
    uint2 queue[32];  // leaves of this step: first slot, owner lane | major axis << 5
    float t[32], u[32], v[32];  // the nearest hit so far (t: FLT_MAX before the first)
    int32_t prim[32];           // its primitive, -1: no hit yet (any-hit: 0 after one)
    uint32_t ray[32];           // the caller's index of the ray | major axis << 30
};
// The same where the rays of one warp may belong to different trees.
struct WalkSharedMulti : WalkShared {
    const float4* tris[32];
};

template <int W, bool ANY, int STACK, bool Q8, bool MULTI = false>
struct WarpWalk {
    using Shared = typename std::conditional<MULTI, WalkSharedMulti, WalkShared>::type;
    // Any-hit entries are a reference alone: nothing is culled before the first hit.
    using Slot = typename std::conditional<ANY, int32_t, uint2>::type;
    static constexpr uint32_t kSlot = sizeof(Slot);

    float rcp[3], od[3];  // 1/d and -o/d of each axis
    float tmin;
    float lim;    // min(tmax, nearest hit so far): entries beyond it are culled
    int32_t cur;   // entry to process: interior node (>= 0), leaf (< -1), kEmpty: the ray is finished
    uint32_t sp;   // local address past the top of the stack

    __device__ __forceinline__ bool active() const { return cur != kEmpty; }

    // Takes ray r: ray setup, root test, the shared record. stack: the local
    // address of the lane's stack.
    __device__ __forceinline__ void begin(const DevTree& tr, RayState& r, Shared* sh, int lane, uint32_t stack) {
        ray_setup(r);
        tmin = r.tmin;
        // SORT culls an entry whose distance lies beyond the current hit when it
        // is popped (fast_bvh.hpp:343); the hit only gets nearer, so such a child
        // need not be pushed: lim is part of the slab test. A pushed entry is
        // never beyond tmax, so culling with lim is culling with the hit.
        lim = r.tmax > FLT_MAX ? FLT_MAX : r.tmax;
        sp = stack;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            rcp[a] = r.rcp[a];
            od[a] = r.od[a];
        }
        sh->c0[lane] = make_float4(r.ox, r.oy, r.oz, r.sx);
        sh->c1[lane] = make_float4(r.sz, r.sy, r.tmin, r.tmax);
        sh->t[lane] = FLT_MAX;
        sh->prim[lane] = -1;
        sh->ray[lane] |= (uint32_t)r.ly << 30;
        if constexpr (MULTI) sh->tris[lane] = tr.tris;
        const float f0 = root_intersect(r, tr.box_lo, tr.box_hi);
        cur = f0 >= 0.0f && !(FLT_MAX < f0) ? tr.root : kEmpty;
    }

    // Next entry that is not culled; the ray is finished when there is none.
    __device__ __forceinline__ void pop(uint32_t stack) {
        for (;;) {
            if (sp == stack) {
                cur = kEmpty;
                return;
            }
            sp -= kSlot;
            if constexpr (ANY) {
                stack_get(sp, cur);
                if (cur != kEmpty) return;
            } else {
                float d;
                stack_get(sp, cur, d);
                if (!(lim < d) && cur != kEmpty) return;
            }
        }
    }

    // Near and far planes of the node's children on axis a, two children per
    // register pair. 8-bit nodes: each bound decodes to fl(origin + q * 2^e)
    // (layout.h, quantize.cpp), a box containing SORT's.
    struct Planes {
        f32x2 n[W / 2], f[W / 2];
    };
    struct Q8Head {
        Load32 a, b;
    };
    __device__ __forceinline__ void load_axis(const char* __restrict__ p, const Q8Head& h, int a, Planes& q) const {
        if constexpr (Q8) {
            float org[4];
            unpack2(h.a.w[0], org[0], org[1]);
            unpack2(h.a.w[1], org[2], org[3]);
            const uint32_t eb = __float_as_uint(org[3]);
            const float sc = __uint_as_float(((eb >> (8 * a)) & 0xffu) << 23);
            const f32x2 s2 = pack2(sc, sc), o2 = pack2(org[a], org[a]), bias = pack2(-8388608.0f, -8388608.0f);
            uint32_t lo[2], hi[2];
            if constexpr (W == 8) {
                const f32x2 l = a == 0 ? h.a.w[2] : (a == 1 ? h.b.w[0] : h.b.w[2]);
                const f32x2 u = a == 0 ? h.a.w[3] : (a == 1 ? h.b.w[1] : h.b.w[3]);
                lo[0] = (uint32_t)l;
                lo[1] = (uint32_t)(l >> 32);
                hi[0] = (uint32_t)u;
                hi[1] = (uint32_t)(u >> 32);
            } else {
                const f32x2 x = a == 0 ? h.a.w[2] : (a == 1 ? h.a.w[3] : h.b.w[0]);
                lo[0] = lo[1] = (uint32_t)x;
                hi[0] = hi[1] = (uint32_t)(x >> 32);
            }
            const bool flip = rcp[a] < 0.0f;
#pragma unroll
            for (int g = 0; g < W / 4; ++g) {
                const uint32_t nw = flip ? hi[g] : lo[g], fw = flip ? lo[g] : hi[g];
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    auto byte2 = [](uint32_t w, int b) {  // 2^23 + two bytes
                        return pack2(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7540u | (unsigned)b)),
                                     __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7540u | (unsigned)(b + 1))));
                    };
                    q.n[2 * g + k] = fma2(add2(byte2(nw, 2 * k), bias), s2, o2);
                    q.f[2 * g + k] = fma2(add2(byte2(fw, 2 * k), bias), s2, o2);
                }
            }
        } else {
            constexpr int kPlane = W * 4;  // bytes
            const int off = (int)(__float_as_uint(rcp[a]) >> 31) * kPlane;  // the upper plane where 1/d < 0
            const char* pn = p + 2 * a * kPlane + off;
            const char* pf = p + 2 * a * kPlane + (kPlane - off);
            if constexpr (W == 8) {
                const Load32 l = load32(pn), u = load32(pf);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    q.n[k] = l.w[k];
                    q.f[k] = u.w[k];
                }
            } else {
                const ulonglong2 l = __ldg(reinterpret_cast<const ulonglong2*>(pn));
                const ulonglong2 u = __ldg(reinterpret_cast<const ulonglong2*>(pf));
                q.n[0] = l.x;
                q.n[1] = l.y;
                q.f[0] = u.x;
                q.f[1] = u.y;
            }
        }
        const f32x2 nz = pack2(c_neg_zero2.x, c_neg_zero2.y), rc = pack2(rcp[a], rcp[a]), o = pack2(od[a], od[a]);
#pragma unroll
        for (int k = 0; k < W / 2; ++k) {
            q.n[k] = add2(fma2(q.n[k], rc, nz), o);
            q.f[k] = add2(fma2(q.f[k], rc, nz), o);
        }
    }

    // Interior node `cur`: box-tests the children (the arithmetic of
    // slab_near_far), pushes all hits but the nearest and makes that one `cur`
    // (SORT's order: nearest first, equal distances higher slot first); pops
    // when no child is hit.
    __device__ __forceinline__ void node(const float4* __restrict__ nodes, uint32_t stack, float tmax) {
        constexpr int kBytes = 16 * (Q8 ? (W == 8 ? kQ8F4W8 : kQ8F4W4) : NodeShape<W>::kF4);
        constexpr int kChild = 16 * (Q8 ? (W == 8 ? 4 : 3) : 6 * (W / 4));  // byte offset of child[0]
        const char* p = reinterpret_cast<const char*>(nodes) + (size_t)(uint32_t)cur * kBytes;
        Q8Head h;
        if constexpr (Q8) {
            h.a = load32(p);
            h.b = load32(p + 32);
        }
        int32_t ch[W];
        if constexpr (W == 8) {
            const Load32 c = load32(p + kChild);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                ch[2 * k] = (int32_t)(uint32_t)c.w[k];
                ch[2 * k + 1] = (int32_t)(uint32_t)(c.w[k] >> 32);
            }
        } else if constexpr (Q8) {
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                ch[2 * k] = (int32_t)(uint32_t)h.b.w[2 + k];
                ch[2 * k + 1] = (int32_t)(uint32_t)(h.b.w[2 + k] >> 32);
            }
        } else {
            const int4 c = __ldg(reinterpret_cast<const int4*>(p + kChild));
            ch[0] = c.x;
            ch[1] = c.y;
            ch[2] = c.z;
            ch[3] = c.w;
        }
        float d[W], x[W];  // entry and exit distance
        {
            Planes q;
            load_axis(p, h, 0, q);
#pragma unroll
            for (int k = 0; k < W / 2; ++k) {
                unpack2(q.n[k], d[2 * k], d[2 * k + 1]);
                unpack2(q.f[k], x[2 * k], x[2 * k + 1]);
            }
        }
#pragma unroll
        for (int a = 1; a < 3; ++a) {
            Planes q;
            load_axis(p, h, a, q);
#pragma unroll
            for (int k = 0; k < W / 2; ++k) {
                float n[2], f[2];
                unpack2(q.n[k], n[0], n[1]);
                unpack2(q.f[k], f[0], f[1]);
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const int j = 2 * k + c;
                    d[j] = a == 1 ? fmaxf(fmaxf(d[j], n[c]), tmin) : fmaxf(d[j], n[c]);
                    x[j] = a == 1 ? fminf(fminf(x[j], f[c]), lim) : fminf(x[j], f[c]);
                }
            }
        }
        // The two nearest hits so far stay in registers (r1, then r2): a visit
        // mostly hits one or two children, so it mostly makes one store at most.
        int32_t r1 = kEmpty, r2 = kEmpty;
        if constexpr (ANY) {
            // Before the first hit nothing is culled, so any order finds the
            // same answer: descend into the lowest hit slot, push the others.
            if (d[W - 1] <= x[W - 1]) r1 = ch[W - 1];
#pragma unroll
            for (int j = W - 2; j >= 0; --j)
                asm volatile(
                    "{\n\t.reg .pred P, S;\n\t"
                    "setp.le.f32 P, %3, %4;\n\t"
                    "setp.ne.and.s32 S, %2, -1, P;\n\t"
                    "@S st.local.b32 [%0], %2;\n\t"
                    "@S add.u32 %0, %0, 4;\n\t"
                    "@P mov.b32 %2, %1;\n\t"
                    "@P mov.b32 %1, %5;\n\t}"
                    : "+r"(sp), "+r"(r1), "+r"(r2)
                    : "f"(d[j]), "f"(x[j]), "r"(ch[j]));
            asm volatile(
                "{\n\t.reg .pred S;\n\t"
                "setp.ne.s32 S, %1, -1;\n\t"
                "@S st.local.b32 [%0], %1;\n\t"
                "@S add.u32 %0, %0, 4;\n\t}"
                : "+r"(sp)
                : "r"(r2));
            cur = r1;
            if (r1 == kEmpty) pop(stack);
        } else {
            if (!(tmin > -1.0f)) {
                // fast_bvh.hpp:438-453: with three or more hits (those beyond the
                // current hit among them) only distances > -1 are taken.
                float exits[W];
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    Planes q;
                    load_axis(p, h, a, q);
#pragma unroll
                    for (int k = 0; k < W / 2; ++k) {
                        float f[2];
                        unpack2(q.f[k], f[0], f[1]);
                        exits[2 * k] = fminf(a ? exits[2 * k] : tmax, f[0]);
                        exits[2 * k + 1] = fminf(a ? exits[2 * k + 1] : tmax, f[1]);
                    }
                }
                int hits = 0;
#pragma unroll
                for (int j = 0; j < W; ++j) hits += d[j] <= exits[j] ? 1 : 0;
                if (hits >= 3) {
#pragma unroll
                    for (int j = 0; j < W; ++j)
                        if (!(d[j] > -1.0f)) d[j] = __int_as_float(0x7fffffff);  // NaN: no hit
                }
            }
            // A later child at an equal distance is the nearer one (SORT visits
            // the higher slot first); whatever drops out of the two is pushed.
            const uint32_t sp0 = sp;
            const float inf = __int_as_float(0x7f800000);
            float d1 = inf, d2 = inf;
            if (d[0] <= x[0]) {
                r1 = ch[0];
                d1 = d[0];
            }
#pragma unroll
            for (int j = 1; j < W; ++j)
                if (j == 1)
                    asm volatile(
                        "{\n\t.reg .pred P, Q;\n\t"
                        "setp.le.f32 P, %4, %5;\n\t"
                        "setp.le.and.f32 Q, %4, %1, P;\n\t"
                        "@P mov.b32 %2, %6;\n\t"
                        "@P mov.f32 %3, %4;\n\t"
                        "@Q mov.b32 %2, %0;\n\t"
                        "@Q mov.f32 %3, %1;\n\t"
                        "@Q mov.b32 %0, %6;\n\t"
                        "@Q mov.f32 %1, %4;\n\t}"
                        : "+r"(r1), "+f"(d1), "+r"(r2), "+f"(d2)
                        : "f"(d[j]), "f"(x[j]), "r"(ch[j]));
                else
                    asm volatile(
                        "{\n\t.reg .pred P, Q, R, S;\n\t.reg .b32 r;\n\t.reg .f32 t;\n\t"
                        "setp.le.f32 P, %5, %6;\n\t"          // the child's box is hit
                        "setp.le.and.f32 Q, %5, %2, P;\n\t"   // it is the nearest
                        "setp.le.and.f32 R, %5, %4, P;\n\t"   // it is one of the two nearest
                        "setp.ne.and.s32 S, %3, -1, P;\n\t"   // one of the three is pushed
                        "selp.b32 r, %3, %7, R;\n\t"
                        "selp.f32 t, %4, %5, R;\n\t"
                        "@S st.local.v2.b32 [%0], {r, t};\n\t"
                        "@S add.u32 %0, %0, 8;\n\t"
                        "@R mov.b32 %3, %7;\n\t"
                        "@R mov.f32 %4, %5;\n\t"
                        "@Q mov.b32 %3, %1;\n\t"
                        "@Q mov.f32 %4, %2;\n\t"
                        "@Q mov.b32 %1, %7;\n\t"
                        "@Q mov.f32 %2, %5;\n\t}"
                        : "+r"(sp), "+r"(r1), "+f"(d1), "+r"(r2), "+f"(d2)
                        : "f"(d[j]), "f"(x[j]), "r"(ch[j]));
            // Four or more hits: the pushed ones by decreasing distance, equal
            // distances lowest slot first (they were pushed in slot order).
            for (uint32_t k = sp0 + kSlot; (int32_t)(sp - k) > 0; k += kSlot) {
                int32_t r, pr;
                float t, pt;
                stack_get(k, r, t);
                uint32_t q = k;
                while (q != sp0) {
                    stack_get(q - kSlot, pr, pt);
                    if (!(pt < t)) break;
                    stack_put(q, pr, pt);
                    q -= kSlot;
                }
                if (q != k) stack_put(q, r, t);
            }
            asm volatile(
                "{\n\t.reg .pred S;\n\t"
                "setp.ne.s32 S, %1, -1;\n\t"
                "@S st.local.v2.b32 [%0], {%1, %2};\n\t"
                "@S add.u32 %0, %0, 8;\n\t}"
                : "+r"(sp)
                : "r"(r2), "f"(d2));
            cur = r1;
            if (r1 == kEmpty) pop(stack);
        }
    }

    // Tests up to four pending leaves' next eight triangles (whole warp): lane
    // l of eight takes triangle l of leaf base + lane / 8. Per leaf the hits
    // are taken in lane order, each only if strictly nearer, which is SORT's
    // order and rule (simd/simd_triangle.h:359-369). again: this lane's leaf
    // goes on past these slots.
    __device__ __forceinline__ void round(const float4* __restrict__ tris, Shared* sh, int lane, int base, int cnt,
                                          bool& again) {
        const int k = base + lane / kLeafLanes, ord = lane & (kLeafLanes - 1);
        const bool live = k < cnt;
        const uint2 leaf = sh->queue[live ? k : cnt - 1];
        const int src = (int)(leaf.y & 31u);
        const float4* tb = tris;
        if constexpr (MULTI) tb = sh->tris[src];
        const float4* q = tb + 3 * (size_t)(leaf.x + (uint32_t)ord);
        const float4 a = __ldg(q), b = __ldg(q + 1), c = __ldg(q + 2);
        const float4 c0 = sh->c0[src], c1 = sh->c1[src];
        TriEdges e;
        bool pass = walk_tri_edges(c0, c1.x, leaf.y >> 5, a, b, c, e) && live;
        const unsigned ends = __ballot_sync(kFullWarp, __float_as_int(b.w) != 0) >> (lane & ~(kLeafLanes - 1)) & 0xffu;
        const unsigned before = (1u << ord) - 1u;
        pass = pass && (ends & before) == 0;
        if (__any_sync(kFullWarp, pass)) {
            float t, u, v;
            bool hit = walk_tri_hit(e, pass, c1.y, c1.z, c1.w, t, u, v) && t < sh->t[src];
            // One hit of each leaf at a time, in lane order.
            for (;;) {
                const unsigned hm = __ballot_sync(kFullWarp, hit);
                if (hm == 0) break;
                if (hit && (hm >> (lane & ~(kLeafLanes - 1)) & before) == 0) {
                    hit = false;
                    if constexpr (ANY) {
                        sh->prim[src] = 0;
                    } else if (t < sh->t[src]) {
                        sh->t[src] = t;
                        sh->u[src] = u;
                        sh->v[src] = v;
                        sh->prim[src] = __float_as_int(a.w);
                    }
                }
                __syncwarp();
                if constexpr (ANY) break;
            }
        }
        unsigned on = __ballot_sync(kFullWarp, live && ord == 0 && ends == 0);
        for (; on; on &= on - 1u) again |= __shfl_sync(kFullWarp, src, __ffs(on) - 1) == lane;
    }

    // Leaf step of the whole warp: lanes with a leaf in `cur`. Eight lanes test
    // a leaf's next eight triangles, four leaves at a time, whichever lanes own
    // them; lanes whose ray is finished help.
    __device__ __forceinline__ void leaves(const float4* __restrict__ tris, uint32_t stack, Shared* sh, int lane) {
        bool leaf = cur < kEmpty;
        unsigned pend = __ballot_sync(kFullWarp, leaf);
        if (pend == 0) return;
        do {
            const int cnt = __popc(pend);
            if (leaf)
                sh->queue[__popc(pend & ((1u << lane) - 1u))] =
                    make_uint2((uint32_t)cur & 0x7fffffffu, (uint32_t)lane | sh->ray[lane] >> 30 << 5);
            __syncwarp();
            bool again = false;
            for (int base = 0; base < cnt; base += kRoundLeaves) round(tris, sh, lane, base, cnt, again);
            __syncwarp();
            leaf = again && !(ANY && sh->prim[lane] == 0);
            if (leaf) cur += kLeafLanes;
            pend = __ballot_sync(kFullWarp, leaf);
        } while (pend);
        if (cur < kEmpty) {
            if constexpr (ANY) {
                if (sh->prim[lane] == 0) {
                    cur = kEmpty;
                    return;
                }
            } else {
                lim = fminf(lim, sh->t[lane]);
            }
            pop(stack);
        }
    }

    // One step of the whole warp: every lane at an interior node visits it, then
    // every lane at a leaf tests it (also one reached in this step).
    __device__ __forceinline__ void step(const float4* __restrict__ nodes, const float4* __restrict__ tris,
                                         uint32_t stack, Shared* sh, int lane, int* __restrict__ err) {
        if (cur >= 0) {
            if (sp - stack > (STACK - W) * kSlot) {  // cannot happen when STACK >= depth*(W-1)+1; reported, never overrun
                atomicOr(err, 1);
                cur = kEmpty;
            } else {
                node(nodes, stack, sh->c1[lane].w);
            }
        }
        __syncwarp();
        leaves(tris, stack, sh, lane);
    }
};

// Traverses every ray that `job` hands out, one warp's share. A lane whose ray
// is finished keeps its answer until at least `refill` lanes are idle; then the
// idle lanes write their answers and take new rays together, so that neither
// runs for a lane or two at a time.
//   tree()         the rays' tree (MULTI: any value, take sets each lane's)
//   bool more()    whether rays are left to take (the whole warp, one answer)
//   bool take(idle, mask, lane, sh, r, tr)
//                  the whole warp, `mask` its idle lanes: an idle lane's next ray
//                  into r, its index into sh->ray[lane]; false when none is left
//   void put(fin, lane, sh)
//                  the whole warp: lanes with fin set write their ray's answer
template <int W, bool ANY, int STACK, bool Q8, bool MULTI, class Job>
__device__ __forceinline__ void walk_rays(Job& job, typename WarpWalk<W, ANY, STACK, Q8, MULTI>::Shared* sh, int lane,
                                          int refill, int* __restrict__ err) {
    using Walk = WarpWalk<W, ANY, STACK, Q8, MULTI>;
    typename Walk::Slot stk[STACK];
    const uint32_t stack = (uint32_t)__cvta_generic_to_local(stk);
    Walk w;
    w.cur = kEmpty;
    bool held = false;  // this lane holds a finished, unwritten answer or a ray in traversal
    typename std::conditional<MULTI, DevTree, const DevTree&>::type tr = job.tree();
    for (;;) {
        const unsigned idle = __ballot_sync(kFullWarp, !w.active());
        if (idle == kFullWarp || (__popc(idle) >= refill && job.more())) {
            const bool fin = held && !w.active();
            job.put(fin, lane, sh);
            if (fin) held = false;
            if (job.more()) {
                RayState r;
                if (job.take(!w.active(), idle, lane, sh, r, tr)) {
                    w.begin(tr, r, sh, lane, stack);
                    held = true;
                }
                __syncwarp();
                if (__ballot_sync(kFullWarp, w.active()) == 0) continue;
            } else if (idle == kFullWarp) {
                break;
            }
        }
        w.step(tr.nodes, tr.tris, stack, sh, lane, err);
    }
}

}  // namespace sg
