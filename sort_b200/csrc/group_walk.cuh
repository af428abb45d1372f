// Closest-hit / any-hit walk of small launches over width-8 trees: eight lanes per ray.
//
// The visit order, the culling, the leaf order and the rounding of every operation
// that decides a hit are those of WarpWalk (warp_walk.cuh), so the results are the
// same bits. A launch of few rays waits for one ray's chain of dependent visits, so
// the chain is what this form shortens: lane j of a group tests child j of the node
// (or triangle j of the leaf), a child's place in the visit order is the count of
// the children before it, all pushes are one store and a pop looks at eight entries
// at once. What is left of the chain is loads: each visit waits for its node, each
// leaf for its triangles (prefetching the pushed children: 0.96 to 1.00x).
// WarpWalk against this form, us, with L2 warm: 4,099 camera rays, 82k triangles,
// 28.7 / 24.6; 4,096 diffuse rays, 5.2M triangles, 60.4 / 52.9; 16,384 diffuse
// 92.3 / 80.3, shadow 70.2 / 51.3; 16,384 diffuse, 8-bit nodes, 90.2 / 67.7. Width 4,
// where half of a group's lanes idle at a node, gained nothing (9,472 diffuse rays
// 80.1 / 82.0, camera 30.8 / 30.8) and has no such form.
#pragma once

#include <cuda_runtime.h>

#include "trace_common.cuh"
#include "warp_walk.cuh"

namespace sg {

constexpr int kGroupLanes = kLeafLanes;           // lanes per ray
constexpr int kWarpGroups = 32 / kGroupLanes;     // rays of a warp
constexpr int kBlockGroups = kWalkThreads / kGroupLanes;

// Traversal stack of one group.
template <bool ANY, int STACK>
struct GroupStack {
    int32_t ref[STACK];
    float d[ANY ? 1 : STACK];
};

template <bool ANY, int STACK, bool Q8>
struct GroupWalk {
    static constexpr int W = 8;  // of the tree; a child per lane
    float rcp[3], od[3];
    float ox, oy, oz, sx, sy, sz;  // origin in the permuted frame, shear
    float tmin, tmax, lim;
    int ly;
    float t, u, v;  // the nearest hit so far
    int32_t prim;
    int32_t cur;    // entry to process; kEmpty: the ray is finished
    int sp;         // entries on the stack

    __device__ __forceinline__ void begin(const DevTree& tr, RayState& r) {
        ray_setup(r);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            rcp[a] = r.rcp[a];
            od[a] = r.od[a];
        }
        ox = r.ox;
        oy = r.oy;
        oz = r.oz;
        sx = r.sx;
        sy = r.sy;
        sz = r.sz;
        ly = r.ly;
        tmin = r.tmin;
        tmax = r.tmax;
        lim = r.tmax > FLT_MAX ? FLT_MAX : r.tmax;
        t = FLT_MAX;
        u = v = 0.0f;
        prim = -1;
        sp = 0;
        const float f0 = root_intersect(r, tr.box_lo, tr.box_hi);
        cur = f0 >= 0.0f && !(FLT_MAX < f0) ? tr.root : kEmpty;
    }

    // Child `ord` of the node: its reference, entry and exit distance (the exit
    // without the ray's end).
    __device__ __forceinline__ int32_t child(const float4* __restrict__ nodes, int ord, float& d, float& x) const {
        constexpr int kBytes = 16 * (Q8 ? kQ8F4W8 : NodeShape<W>::kF4);
        constexpr int kChild = 16 * (Q8 ? 4 : 6 * (W / 4));
        const char* p = reinterpret_cast<const char*>(nodes) + (size_t)(uint32_t)cur * kBytes;
        float n[3], f[3];
        if constexpr (Q8) {
            const float4 h = __ldg(reinterpret_cast<const float4*>(p));
            const float org[3] = {h.x, h.y, h.z};
            const uint32_t eb = __float_as_uint(h.w);
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const unsigned char* b = reinterpret_cast<const unsigned char*>(p) + 16 + 2 * a * W + ord;
                const int off = (int)(__float_as_uint(rcp[a]) >> 31) * W;
                const float sc = __uint_as_float(((eb >> (8 * a)) & 0xffu) << 23);
                n[a] = __fmaf_rn((float)__ldg(b + off), sc, org[a]);
                f[a] = __fmaf_rn((float)__ldg(b + (W - off)), sc, org[a]);
            }
        } else {
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const float* b = reinterpret_cast<const float*>(p) + 2 * a * W + ord;
                const int off = (int)(__float_as_uint(rcp[a]) >> 31) * W;
                n[a] = __ldg(b + off);
                f[a] = __ldg(b + (W - off));
            }
        }
        const int32_t ch = __ldg(reinterpret_cast<const int32_t*>(p + kChild) + ord);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            n[a] = __fadd_rn(__fmul_rn(n[a], rcp[a]), od[a]);
            f[a] = __fadd_rn(__fmul_rn(f[a], rcp[a]), od[a]);
        }
        d = fmaxf(fmaxf(fmaxf(n[0], n[1]), tmin), n[2]);
        x = fminf(fminf(f[0], f[1]), f[2]);
        return ch;
    }

    // One step of the whole warp: groups at an interior node visit it, then groups
    // at a leaf test it (also one reached in this step), then those without an
    // entry take the next one that is not culled.
    __device__ __forceinline__ void step(const float4* __restrict__ nodes, const float4* __restrict__ tris,
                                         GroupStack<ANY, STACK>* stk, int lane, int* __restrict__ err) {
        const int ord = lane & (kGroupLanes - 1), g0 = lane & ~(kGroupLanes - 1);
        const unsigned before = (1u << ord) - 1u;
        auto group = [&](bool p) { return __ballot_sync(kFullWarp, p) >> g0 & 0xffu; };
        bool need = false;
        bool at_node = cur >= 0;
        if (at_node && sp > STACK - W) {  // cannot happen when STACK >= depth*(W-1)+1; reported, never overrun
            if (ord == 0) atomicOr(err, 1);
            cur = kEmpty;
            at_node = false;
        }
        if (__any_sync(kFullWarp, at_node)) {
            float d = 0.0f, x = 0.0f;
            int32_t ch = kEmpty;
            bool box = false;
            if (at_node) {
                ch = child(nodes, ord, d, x);
                box = d <= fminf(x, tmax);
            }
            bool hit = box && d <= fminf(x, lim) && ch != kEmpty;
            if constexpr (!ANY) {
                // fast_bvh.hpp:438-453: with three or more hits (those beyond the
                // current hit among them) only distances > -1 are taken.
                if (__any_sync(kFullWarp, at_node && !(tmin > -1.0f)))
                    if (__popc(group(box)) >= 3 && !(d > -1.0f)) hit = false;
            }
            const unsigned hm = group(hit);
            const int hits = __popc(hm);
            int rank = __popc(hm & before);  // any-hit: slot order
            if constexpr (!ANY) {
                // Nearest first, equal distances higher slot first.
                if (__any_sync(kFullWarp, hits > 1)) {
                    rank = 0;
#pragma unroll
                    for (int s = 1; s < W; ++s) {
                        const float o = __shfl_xor_sync(kFullWarp, d, s);
                        const int other = ord ^ s;
                        if ((hm >> other & 1u) && (o < d || (o == d && other > ord))) ++rank;
                    }
                }
            }
            const unsigned nearest = group(hit && rank == 0);
            const int32_t next = __shfl_sync(kFullWarp, ch, g0 + (nearest ? __ffs(nearest) - 1 : 0));
            if (hit && rank > 0) {
                const int at = sp + hits - 1 - rank;
                stk->ref[at] = ch;
                if constexpr (!ANY) stk->d[at] = d;
            }
            if (at_node) {
                if (hits) {
                    sp += hits - 1;
                    cur = next;
                } else {
                    need = true;
                }
            }
        }
        bool leaf = cur < kEmpty;
        if (__any_sync(kFullWarp, leaf)) {
            uint32_t first = (uint32_t)cur & 0x7fffffffu;
            const float4 c0 = make_float4(ox, oy, oz, sx);
            bool more = leaf;
            do {
                float4 a = make_float4(0, 0, 0, 0), b = a, c = a;
                if (more) {
                    const float4* q = tris + 3 * (size_t)(first + (uint32_t)ord);
                    a = __ldg(q);
                    b = __ldg(q + 1);
                    c = __ldg(q + 2);
                }
                TriEdges e;
                bool pass = walk_tri_edges(c0, sz, (uint32_t)ly, a, b, c, e) && more;
                const unsigned ends = group(__float_as_int(b.w) != 0);
                pass = pass && (ends & before) == 0;
                if (__any_sync(kFullWarp, pass)) {
                    float tt, uu, vv;
                    const bool hit = walk_tri_hit(e, pass, sy, tmin, tmax, tt, uu, vv) && tt < t;
                    if constexpr (ANY) {
                        if (group(hit)) prim = 0;
                    } else {
                        // The hits in lane order, each only if strictly nearer
                        // (simd/simd_triangle.h:359-369): the nearest, lowest lane first.
                        float m = hit ? tt : FLT_MAX;
#pragma unroll
                        for (int s = 1; s < kGroupLanes; s *= 2) m = fminf(m, __shfl_xor_sync(kFullWarp, m, s));
                        const unsigned win = group(hit && tt == m);
                        const int src = g0 + (win ? __ffs(win) - 1 : 0);
                        const float wt = __shfl_sync(kFullWarp, tt, src), wu = __shfl_sync(kFullWarp, uu, src),
                                    wv = __shfl_sync(kFullWarp, vv, src);
                        const int32_t wp = __float_as_int(__shfl_sync(kFullWarp, a.w, src));
                        if (win) {
                            t = wt;
                            u = wu;
                            v = wv;
                            prim = wp;
                        }
                    }
                }
                more = more && ends == 0 && !(ANY && prim == 0);
                first += kGroupLanes;
            } while (__any_sync(kFullWarp, more));
            if (leaf) {
                if (ANY && prim == 0)
                    cur = kEmpty;
                else
                    need = true;
                lim = fminf(lim, t);
            }
        }
        __syncwarp();  // pushed entries are read by the group's other lanes
        while (__any_sync(kFullWarp, need)) {
            const int at = sp - 1 - ord;
            int32_t ref = kEmpty;
            bool ok = need && at >= 0;
            if (ok) {
                ref = stk->ref[at];
                if constexpr (!ANY) ok = !(lim < stk->d[at]);
            }
            const unsigned m = group(ok);
            const int k = m ? __ffs(m) - 1 : 0;
            const int32_t next = __shfl_sync(kFullWarp, ref, g0 + k);
            if (need) {
                if (m) {
                    cur = next;
                    sp -= k + 1;
                    need = false;
                } else {
                    sp -= kGroupLanes;
                    if (sp <= 0) {
                        sp = 0;
                        cur = kEmpty;
                        need = false;
                    }
                }
            }
        }
        __syncwarp();  // read entries may be overwritten
    }
};

}  // namespace sg
