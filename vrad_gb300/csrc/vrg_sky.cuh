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
// nearest finds the cell): the margins of the bounds cover both roundings.  A
// value below -2^23 would wrap: such a cell is outside the map all the same, and
// no sample point lies at such a depth (faces_in_sky_range).
__device__ __forceinline__ int round_bits(float v) {
    return (int)(__float_as_uint(v + 12582912.0f) - 0x4b400000u);
}

__device__ __forceinline__ bool sky_cell(const SkyView &sv, int j, float px, float py, float pz, uint32_t &cell,
                                         int &depth) {
    const float4 gu = __ldg(sv.dirs + 4 * j), gv = __ldg(sv.dirs + 4 * j + 1), gd = __ldg(sv.dirs + 4 * j + 2);
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
    const float4 a = __ldg(sv.dirs + 4 * j + 3);
    const Line L = make_line(px, py, pz, radd(px, rmul(a.x, kMaxTraceLength)), radd(py, rmul(a.y, kMaxTraceLength)),
                             radd(pz, rmul(a.z, kMaxTraceLength)));
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

// The directions that a normal faces, for a warp to share.  Every direction's
// opposite is in the table with the same bits but the sign, so a normal faces
// 81 at most.
constexpr int kSkyGroup = 8;    // directions whose loads overlap
constexpr int kSkyWarps = 4;    // warps of a block, at most
constexpr int kSkyListed = 88;  // list entries: 81, rounded up to whole groups
constexpr int kSkyNormals = 2;  // normals a warp goes through at a time
struct alignas(16) SkyWarp {
    float w[kSkyNormals][kSkyListed];  // the listed directions' cosines, zero past the list
    uint8_t dir[kSkyNormals][kSkyListed];
};

// sky_fraction for lanes whose normal is that of the list they are given.
// cnt: their list's length, most: the longest list's.
__device__ __forceinline__ float sky_sweep(const DevScene &s, const SkyView &sv, const SkyWarp &sh, int list, int cnt,
                                           int most, float px, float py, float pz) {
    float sw = 0.0f, sum = 0.0f;
    for (int p0 = 0; p0 < most; p0 += kSkyGroup) {
        const uint2 dirs = *reinterpret_cast<const uint2 *>(sh.dir[list] + p0);
        int depth[kSkyGroup];
        uint32_t bound[kSkyGroup];
#pragma unroll
        for (int i = 0; i < kSkyGroup; i++) {
            const int j = (int)(((i < 4 ? dirs.x : dirs.y) >> (8 * (i & 3))) & 0xffu);
            uint32_t cell;
            bound[i] = 0u;
            depth[i] = 0x7fffffff;
            int d;
            if (sky_cell(sv, j, px, py, pz, cell, d)) {
                bound[i] = __ldg(sv.bound + cell);
                depth[i] = d;
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
        open &= (1u << min(max(cnt - p0, 0), kSkyGroup)) - 1u;
        while (open) {
            const int i = __ffs(open) - 1;
            open &= open - 1u;
            if (!sky_list_occluded(s, sv, sh.dir[list][p0 + i], px, py, pz)) seen |= 1u << i;
        }
#pragma unroll
        for (int i = 0; i < kSkyGroup; i++) {
            const float w = sh.w[list][p0 + i];
            sw = radd(sw, w);
            sum = radd(sum, (seen >> i) & 1u ? w : 0.0f);
        }
    }
    return sw > 0.0f ? rdiv(sum, sw) : -1.0f;
}

// Cosine-weighted share of the sky directions that reach the sky from p with
// normal n (sums in direction order, as the walk adds them); -1 when no
// direction faces the normal.  `lanes` call together, for points of one scene.
//
// A line is decided by its cell's two depths where they can (93 % of the lines
// of the 4,096-face room: 32 bits read instead of a walk); the rest test the
// cell's triangles, 2.5 on average.  Issue-bound, so the directions that a
// normal faces are listed once for all lanes with their cosines, for the two
// normals of a warp at the end of a face at a time.  The room's sky takes
// 1.66 ms (2.24 with every lane asking all 162 for their cosine, 15.4 by the
// walk), with 152 x 152 cells per direction.  Queueing the undecided lines for
// a full warp at a time cost more in locality than it saved: 1.79 ms, and a
// batch of 48-unit scenes 3.0 instead of 2.7.
__device__ __forceinline__ float sky_fraction(const DevScene &s, const SkyView &sv, unsigned lanes, float px, float py,
                                              float pz, float nx, float ny, float nz, uint32_t &rays) {
    __shared__ SkyWarp warps[kSkyWarps];
    SkyWarp &sh = warps[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const unsigned below = lanes & ((1u << lane) - 1u);
    const int rank = __popc(below), chunk = __popc(lanes);
    float m = -1.0f;
    unsigned left = lanes;
    while (left) {
        unsigned part = 0u;
        int list = 0, cnt = 0, most = 0;
#pragma unroll 1
        for (int l = 0; l < kSkyNormals && part != left; l++) {
            const int lead = __ffs(left & ~part) - 1;
            const float lx = __shfl_sync(lanes, nx, lead), ly = __shfl_sync(lanes, ny, lead),
                        lz = __shfl_sync(lanes, nz, lead);
            // (a lane whose normal is not a number is a list of its own)
            const bool mine = lane == lead || (nx == lx && ny == ly && nz == lz);
            int n = 0;
            for (int j0 = 0; j0 < kNumAnorms; j0 += chunk) {
                const int j = j0 + rank;
                float w = 0.0f;
                if (j < kNumAnorms) {
                    const float4 a = __ldg(sv.dirs + 4 * j + 3);
                    w = dot3r(lx, ly, lz, a.x, a.y, a.z);
                }
                const unsigned faced = __ballot_sync(lanes, w > 0.0f);
                if (w > 0.0f) {
                    const int at = n + __popc(faced & below);
                    sh.dir[l][at] = (uint8_t)j;
                    sh.w[l][at] = w;
                }
                n += __popc(faced);
            }
            for (int i = n + rank; i < kSkyListed; i += chunk) {
                sh.dir[l][i] = 0;
                sh.w[l][i] = 0.0f;
            }
            const unsigned same = __ballot_sync(lanes, mine) & left & ~part;
            if ((same >> lane) & 1u) {
                list = l;
                cnt = n;
            }
            most = max(most, n);
            part |= same;
        }
        __syncwarp(lanes);
        if ((part >> lane) & 1u) {
            m = sky_sweep(s, sv, sh, list, cnt, most, px, py, pz);
            rays += (uint32_t)cnt;
        }
        __syncwarp(lanes);  // before the lists change
        left &= ~part;
    }
    return m;
}

}  // namespace vrg
