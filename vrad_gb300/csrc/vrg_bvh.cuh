// vrg_bvh.cuh -- walking the four-wide hierarchy (bvhbuild.cpp).
//
// A node is 64 bytes: four boxes of one byte per bound, and the children's
// words.  Divergent lanes read nodes at the load pipe's data rate, so the
// bytes of a node are what a step costs (full floats, 112 bytes: 350 us for
// 2^20 lines in 12,300 triangles with that pipe 87 % busy).  Every plane is
// moved outwards by the walk's slab bound (ray_slack): a hit of the exact test
// lies within it of its triangle, so no leaf that holds one is skipped and the
// answers are those of testing every triangle.
#pragma once

#include <cuda_runtime.h>

#include "vrg_device.h"
#include "vrg_trace.cuh"

namespace vrg {

__device__ __forceinline__ float box_rcp(float d) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    return r;
}

// A ray against boxes: per axis the reciprocal direction and the origin's
// distance to a plane that the ray enters or leaves by, moved by the slab.
//
// bvh_step multiplies the reciprocal by up to 2^23 steps of a node, a 60th of
// the scene's scale at most, and that has to stay finite: an infinity of the
// wrong sign closes every box.  So no component counts as less than 2^-28 of
// the largest.  A hit inside the scene is at most scale + |origin| away along
// the largest axis, so this moves it sideways by less than a thousandth of the
// slab.  A direction too short or too long for the rest (the product is then
// 2^120 at most) gets no number for its reciprocal: it passes every box, and the
// exact tests decide alone.
struct BoxRay {
    float inv[3], in[3], out[3];
    uint32_t neg;  // bit a: the direction's a component is negative
};
__device__ __forceinline__ BoxRay box_ray(const SceneGeom &g, const Ray &ray, float slack) {
    BoxRay r;
    const float o[3] = {ray.ox, ray.oy, ray.oz}, d[3] = {ray.dx, ray.dy, ray.dz};
    const float most = fmaxf(fabsf(d[0]), fmaxf(fabsf(d[1]), fabsf(d[2])));
    const bool fits = most >= fmaxf(g.scale * 0x1p-75f, 0x1p-90f) && most <= 0x1p60f;
    const float least = most * 0x1p-28f;
    r.neg = 0u;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const bool neg = signbit(d[a]);
        r.neg |= (neg ? 1u : 0u) << a;
        r.inv[a] = fits ? box_rcp(fabsf(d[a]) < least ? copysignf(least, d[a]) : d[a]) : __int_as_float(0x7fc00000);
        const float sd = neg ? -slack : slack;
        r.in[a] = -sd - o[a];
        r.out[a] = sd - o[a];
    }
    return r;
}

// A direction of no length meets no triangle: the quotient that the exact test
// takes is infinite or no number.
__device__ __forceinline__ bool has_direction(const Ray &ray) {
    return ray.dx != 0.0f || ray.dy != 0.0f || ray.dz != 0.0f;
}

// 2^23 + byte c of w, as a float.
__device__ __forceinline__ float byte_float(uint32_t w, int c) {
    return __uint_as_float(__byte_perm(w, 0x4b000000u, 0x7540u | (uint32_t)c));
}

// One step through inner node `cur`: the nearest child the ray meets on
// [t0, t1] becomes `cur` (its entry t in `at`) and the others are stacked with
// theirs; false when it meets none.  A plane q steps from the node's origin is
// met at t = (2^23 + q) * (step * inv) + k, whose rounding is a step at most.
// Without ORDER the children go in any order and their entries are not kept.
template <bool ORDER>
__device__ __forceinline__ bool bvh_step(const BvhView &bv, const BoxRay &rp, float t0, float t1, uint2 *stk, int &sp,
                                         uint32_t &cur) {
    const float4 *np = bv.nodes + 4 * (size_t)cur;
    const float4 h = __ldg(np);
    const uint4 b0 = __ldg(reinterpret_cast<const uint4 *>(np + 1)), b1 = __ldg(reinterpret_cast<const uint4 *>(np + 2)),
                b2 = __ldg(reinterpret_cast<const uint4 *>(np + 3));
    const float step[3] = {__uint_as_float(b2.z), __uint_as_float(b2.w), h.w}, org[3] = {h.x, h.y, h.z};
    const uint32_t lo[3] = {b0.x, b0.z, b1.x}, hi[3] = {b0.y, b0.w, b1.y}, word[4] = {b1.z, b1.w, b2.x, b2.y};
    float s[3], kin[3], kout[3];
    uint32_t win[3], wout[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const bool neg = (rp.neg >> a) & 1u;
        s[a] = step[a] * rp.inv[a];
        const float m = -8388608.0f * s[a];
        kin[a] = __fmaf_rn(org[a] + rp.in[a], rp.inv[a], m);
        kout[a] = __fmaf_rn(org[a] + rp.out[a], rp.inv[a], m);
        win[a] = neg ? hi[a] : lo[a];
        wout[a] = neg ? lo[a] : hi[a];
    }
    uint32_t next = kBvhNone;
    float at = kInf;
#pragma unroll
    for (int c = 0; c < 4; c++) {
        const float tn = fmaxf(fmaxf(fmaxf(__fmaf_rn(byte_float(win[0], c), s[0], kin[0]),
                                           __fmaf_rn(byte_float(win[1], c), s[1], kin[1])),
                                     __fmaf_rn(byte_float(win[2], c), s[2], kin[2])), t0);
        const float tf = fminf(fminf(fminf(__fmaf_rn(byte_float(wout[0], c), s[0], kout[0]),
                                           __fmaf_rn(byte_float(wout[1], c), s[1], kout[1])),
                                     __fmaf_rn(byte_float(wout[2], c), s[2], kout[2])), t1);
        if (!ORDER) {
            if (tn <= tf) {
                if (next != kBvhNone) stk[sp++] = make_uint2(next, 0u);
                next = word[c];
            }
        } else if (tn <= tf) {
            const bool nearer = tn < at;
            if (next != kBvhNone) {
                stk[sp] = make_uint2(nearer ? next : word[c], __float_as_uint(nearer ? at : tn));
                sp++;
            }
            if (nearer || next == kBvhNone) {
                next = word[c];
                at = tn;
            }
        }
    }
    cur = next;
    return next != kBvhNone;
}

// The next stacked node that can still hold the answer; false when there is
// none.
__device__ __forceinline__ bool bvh_pop(const uint2 *stk, int &sp, float best_t, uint32_t &cur) {
    while (sp > 0) {
        sp--;
        const uint2 e = stk[sp];
        if (__uint_as_float(e.y) > best_t) continue;
        cur = e.x;
        return true;
    }
    return false;
}

// Tests a leaf's triangles; true when the walk ends here.
template <int MODE, int OPT>
__device__ __forceinline__ bool bvh_leaf(const DevScene &s, const BvhView &bv, const Ray &ray, float tmin, float tmax,
                                         int32_t skip, float any_limit, uint32_t word, int32_t &best, float &best_t) {
    const size_t first = (size_t)bv.base + bvh_leaf_first(word);
    const uint32_t cnt = bvh_leaf_count(word);
    for (uint32_t i = 0; i < cnt; i++)
        if (tri_test<MODE, OPT>(s, ray, tmin, tmax, skip, any_limit, __ldg(s.leaf_planes + first + i), first + i, best, best_t))
            return true;
    return false;
}

// A whole walk; returns the hit triangle's index (-1 for none) and its t.
template <int MODE, int OPT>
__device__ __forceinline__ int32_t bvh_trace(const DevScene &s, const BvhView &bv, const Ray &ray, float slack,
                                             float tmin, float tmax, int32_t skip, float any_limit, float *t_out) {
    int32_t best = -1;
    float best_t = kInf;
    uint2 stk[kBvhStack];
    if (bv.nodes && tmin <= tmax && has_direction(ray)) {
        const BoxRay rp = box_ray(s.g, ray, slack);
        uint32_t cur = 0u;
        int sp = 0;
        for (;;) {
            bool more;
            if (cur & kBvhLeafBit) {
                if (bvh_leaf<MODE, OPT>(s, bv, ray, tmin, tmax, skip, any_limit, cur, best, best_t)) break;
                more = false;
            } else {
                more = bvh_step<MODE == kClosest>(bv, rp, tmin, fminf(tmax, best_t), stk, sp, cur);
            }
            if (!more && !bvh_pop(stk, sp, best_t, cur)) break;
        }
    }
    *t_out = best_t;
    return best;
}

}  // namespace vrg
