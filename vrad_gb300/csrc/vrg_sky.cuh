// vrg_sky.cuh -- sky maps: what the 162 sky directions meet in a scene,
// looked up instead of walked.  Layout in vrg_device.h (SkyView), built by
// skymap.cu.
#pragma once

#include <cuda_runtime.h>

#include "anorms_table.h"
#include "vrg_device.h"
#include "vrg_trace.cuh"

namespace vrg {

// The 162 sky directions (one copy per translation unit).
static __constant__ float c_anorms[kNumAnorms * 3] = VRG_ANORMS_INIT;

// Cell and depth of a point in direction j's map; false outside the map,
// where no triangle is.  Coordinates round to integers by adding 1.5 * 2^23
// (the cell coordinates are stored half a cell low, so that rounding to the
// nearest finds the cell): the margins of the bounds cover both roundings.
__device__ __forceinline__ int round_bits(float v) {
    return (int)(__float_as_uint(v + 12582912.0f) - 0x4b400000u);
}

__device__ __forceinline__ bool sky_cell(const SkyView &sv, int j, float px, float py, float pz, uint32_t &cell,
                                         int &depth) {
    const float4 gu = __ldg(sv.dirs + 3 * j), gv = __ldg(sv.dirs + 3 * j + 1), gd = __ldg(sv.dirs + 3 * j + 2);
    const float cu = __fmaf_rn(gu.x, px, __fmaf_rn(gu.y, py, __fmaf_rn(gu.z, pz, gu.w)));
    const float cv = __fmaf_rn(gv.x, px, __fmaf_rn(gv.y, py, __fmaf_rn(gv.z, pz, gv.w)));
    depth = round_bits(__fmaf_rn(gd.x, px, __fmaf_rn(gd.y, py, __fmaf_rn(gd.z, pz, gd.w))));
    const int iu = round_bits(cu), iv = round_bits(cv);
    if ((uint32_t)iu >= (uint32_t)sv.n || (uint32_t)iv >= (uint32_t)sv.n) return false;
    cell = (uint32_t)((j * sv.n + iv) * sv.n + iu);
    return true;
}

// The line of direction j from p, in a cell whose bounds do not decide it:
// the closest hit among the cell's triangles by the exact test.  Every
// triangle that could decide the line is in the list, except that in a
// kSkyPast cell a line from before the sky that hits neither sky nor what lies
// around it ends at the covering triangle.
__device__ __forceinline__ bool sky_list_occluded(const DevScene &s, const SkyView &sv, int j, float px, float py,
                                                  float pz) {
    uint32_t cell = 0;
    int depth;
    if (!sky_cell(sv, j, px, py, pz, cell, depth)) return false;
    const uint32_t bound = __ldg(sv.bound + cell);
    const uint2 info = __ldg(sv.info + cell);
    const uint32_t cnt = info.y & ~kSkyCellFlag;
    // where no opaque triangle reaches past the sky every accepted hit occludes
    const float any_limit = (info.y & kSkyCellFlag) ? 0.0f : kInf;
    const Line L = make_line(px, py, pz, radd(px, rmul(c_anorms[3 * j], kMaxTraceLength)),
                             radd(py, rmul(c_anorms[3 * j + 1], kMaxTraceLength)),
                             radd(pz, rmul(c_anorms[3 * j + 2], kMaxTraceLength)));
    const Ray ray{L.ox, L.oy, L.oz, L.dx, L.dy, L.dz};
    int32_t best = -1;
    float best_t = kInf;
    for (uint32_t i = 0; i < cnt; i++) {
        const uint2 e = __ldg(sv.pool + info.x + i);
        if ((int)e.y < depth) break;  // this triangle and the rest lie behind p
        const size_t k = e.x;
        if (tri_test<kSkyOcc, kOptSign>(s, ray, 0.0f, L.len, -1, any_limit, __ldg(s.leaf_planes + k), k, best, best_t))
            return true;
    }
    if (best < 0) return (bound & kSkyPast) && depth <= (int)((bound & ~kSkyPast) >> 16) * 2;
    return (__ldg(&s.tri_ids[best]) & kTraceIdSky) == 0;
}

// Cosine-weighted share of the sky directions that reach the sky from p with
// normal n (sums in direction order, as the walk adds them); -1 when no
// direction faces the normal.  A line is decided by its cell's two depths
// where they can (96 % of the lines of the 4,096-face room: 32 bits read
// instead of a walk); the rest test the cell's triangles, 2.6 on average.
// kSkyGroup directions go at a time so that their loads overlap.  Issue-bound:
// 90 warp instructions per direction, two thirds of the issue slots busy.  The
// room's gather takes 3.3 ms instead of 16.3 (2.1 of them in here; 15.4 by
// the walk), with 152 x 152 cells per direction.
constexpr int kSkyGroup = 6;
static_assert(kNumAnorms % kSkyGroup == 0, "whole groups of directions");

__device__ __forceinline__ float sky_fraction(const DevScene &s, const SkyView &sv, float px, float py, float pz,
                                              float nx, float ny, float nz, uint32_t &rays) {
    float sw = 0.0f, sum = 0.0f;
    for (int j0 = 0; j0 < kNumAnorms; j0 += kSkyGroup) {
        float w[kSkyGroup];
        int depth[kSkyGroup];
        uint32_t bound[kSkyGroup];
#pragma unroll
        for (int i = 0; i < kSkyGroup; i++) {
            const int j = j0 + i;
            w[i] = dot3r(nx, ny, nz, c_anorms[3 * j], c_anorms[3 * j + 1], c_anorms[3 * j + 2]);
            bound[i] = 0u;
            depth[i] = 0x7fffffff;
            if (w[i] > 0.0f) {
                uint32_t cell;
                int d;
                if (sky_cell(sv, j, px, py, pz, cell, d)) {
                    bound[i] = __ldg(sv.bound + cell);
                    depth[i] = d;
                }
            }
        }
        uint32_t seen = 0u, open = 0u;  // reaches the sky; not decided
#pragma unroll
        for (int i = 0; i < kSkyGroup; i++) {
            const bool past = (bound[i] & kSkyPast) != 0u;
            const bool above = depth[i] > (int)((bound[i] & ~kSkyPast) >> 16) * 2;
            if (above && !past) seen |= 1u << i;
            else if (!((above || !past) && (int)(bound[i] & 0xffffu) > max(depth[i], 0))) open |= 1u << i;
        }
        while (open) {
            const int i = __ffs(open) - 1;
            open &= open - 1u;
            if (!sky_list_occluded(s, sv, j0 + i, px, py, pz)) seen |= 1u << i;
        }
#pragma unroll
        for (int i = 0; i < kSkyGroup; i++) {
            if (!(w[i] > 0.0f)) continue;
            sw = radd(sw, w[i]);
            rays++;
            if ((seen >> i) & 1u) sum = radd(sum, w[i]);
        }
    }
    return sw > 0.0f ? rdiv(sum, sw) : -1.0f;
}

}  // namespace vrg
