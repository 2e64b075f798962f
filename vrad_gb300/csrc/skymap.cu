// skymap.cu -- building a scene's sky maps (layout and use in vrg_device.h and
// vrg_sky.cuh): per sky direction the triangles rasterised into a grid of
// cells, conservatively.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "anorms_table.h"
#include "vrg_device.h"
#include "vrg_internal.h"

namespace vrg {

namespace {

constexpr int kThreads = 128;
constexpr int kWarps = kThreads / 32;
constexpr float kDepthLevels = 65000.0f;  // depths lie in [1, 65001]

// What the kernels read of one triangle: its vertices and the leaf record
// that holds it (-1: none, the walk never tests it).
struct alignas(16) SkyTri {
    float v[9];
    int32_t rec;
    int32_t sky;
    int32_t pad;
};

// One direction: the map's three dot products (SkyView::dirs), the way back
// from a cell coordinate to the sheared world coordinate, and the margin in
// cells and in depth levels.
struct SkyDir {
    float4 gu, gv, gd;
    float a0, sa, b0, sb;  // sheared coordinate = a0 + sa * cu
    float ka, kb;          // the direction's other components over its main one
    float mu, mv, mq;      // margins
    float dq0, dqs;        // depth level = dq0 + dqs * (sign * main coordinate)
    float sign;
    int32_t axis;
    float d[3];
};

// One triangle seen along one direction, ready for its cells: the inner side
// of edge e is ea[e] * cu + eb[e] * cv + ec[e] >= 0 in cells, te[e] how far a
// cell's centre may lie outside (or must lie inside) for the widened cell to
// touch (be covered); depth over a cell is q0 + qu * cu + qv * cv +- qh, within
// [lo, hi].
struct alignas(16) Splat {
    float ea[3], eb[3], ec[3], te[3];
    float q0, qu, qv, qh, lo, hi;
    int32_t x0, x1, y0, y1;
    int32_t rec, flags;
};
static_assert(sizeof(Splat) % 16 == 0, "read as whole float4s");
constexpr int kCover = 1, kSky = 2;

__device__ bool make_splat(const SkyTri &t, const float4 plane, const SkyDir &d, int n, Splat &o) {
    if (t.rec < 0) return false;
    float cu[3], cv[3], q[3];
    for (int k = 0; k < 3; k++) {
        const float x = t.v[3 * k], y = t.v[3 * k + 1], z = t.v[3 * k + 2];
        if (!(fabsf(x) <= 1e30f && fabsf(y) <= 1e30f && fabsf(z) <= 1e30f)) return false;
        cu[k] = __fmaf_rn(d.gu.x, x, __fmaf_rn(d.gu.y, y, __fmaf_rn(d.gu.z, z, d.gu.w)));
        cv[k] = __fmaf_rn(d.gv.x, x, __fmaf_rn(d.gv.y, y, __fmaf_rn(d.gv.z, z, d.gv.w)));
        q[k] = __fmaf_rn(d.gd.x, x, __fmaf_rn(d.gd.y, y, __fmaf_rn(d.gd.z, z, d.gd.w)));
    }
    o.lo = fminf(q[0], fminf(q[1], q[2]));
    o.hi = fmaxf(q[0], fmaxf(q[1], q[2]));
    const float umin = fminf(cu[0], fminf(cu[1], cu[2])), umax = fmaxf(cu[0], fmaxf(cu[1], cu[2]));
    const float vmin = fminf(cv[0], fminf(cv[1], cv[2])), vmax = fmaxf(cv[0], fmaxf(cv[1], cv[2]));
    o.x0 = max(0, (int)floorf(umin - d.mu));
    o.x1 = min(n - 1, (int)floorf(umax + d.mu));
    o.y0 = max(0, (int)floorf(vmin - d.mv));
    o.y1 = min(n - 1, (int)floorf(vmax + d.mv));
    o.rec = t.rec;
    o.flags = t.sky ? kSky : 0;
    const float area2 = (cu[1] - cu[0]) * (cv[2] - cv[0]) - (cv[1] - cv[0]) * (cu[2] - cu[0]);
    const float span = fmaxf(umax - umin, vmax - vmin);
    // seen (nearly) edge-on its edge lines lose their side: the bounding box
    // stands for it
    const bool flat = !(fabsf(area2) > 1e-3f * span + 1e-6f);
    float l2min = kDepthLevels * kDepthLevels, l2max = 0.0f;
    for (int e = 0; e < 3; e++) {
        const int f = e == 2 ? 0 : e + 1;
        const float du = cu[f] - cu[e], dv = cv[f] - cv[e];
        const float len = sqrtf(du * du + dv * dv);
        const float s = flat || !(len > 0.0f) ? 0.0f : (area2 < 0.0f ? -1.0f : 1.0f) / len;
        o.ea[e] = -dv * s;
        o.eb[e] = du * s;
        o.ec[e] = -(o.ea[e] * cu[e] + o.eb[e] * cv[e]);
        o.te[e] = fabsf(o.ea[e]) * (0.5f + d.mu) + fabsf(o.eb[e]) * (0.5f + d.mv) + 1e-3f;
        // edge lengths in space, for the shape test below
        const float ex = t.v[3 * f] - t.v[3 * e], ey = t.v[3 * f + 1] - t.v[3 * e + 1], ez = t.v[3 * f + 2] - t.v[3 * e + 2];
        const float l2 = ex * ex + ey * ey + ez * ez;
        l2min = fminf(l2min, l2);
        l2max = fmaxf(l2max, l2);
    }
    // A cell inside the triangle stops lines for certain when the exact test
    // is well conditioned: the plane not seen edge-on (its t is then right to
    // a few roundings) and no extreme sliver (nor are its edge equations off
    // by more than the margin at the far corner).
    const float nd = plane.x * d.d[0] + plane.y * d.d[1] + plane.z * d.d[2];
    if (!flat && fabsf(nd) >= 0.0625f) {
        if (!t.sky && l2max <= 1024.0f * l2min) o.flags |= kCover;
        // depth over the sheared plane: main = (D - Na * a - Nb * b) * dm / (N . d)
        const int a = (d.axis + 1) % 3, b = (d.axis + 2) % 3;
        const float nv[3] = {plane.x, plane.y, plane.z};
        const float r = d.d[d.axis] / nd * d.sign * d.dqs;
        const float pa = -nv[a] * r * d.sa, pb = -nv[b] * r * d.sb;
        o.qu = pa;
        o.qv = pb;
        o.q0 = d.dq0 + (plane.w - nv[a] * d.a0 - nv[b] * d.b0) * r;
        o.qh = fabsf(pa) * (0.5f + d.mu) + fabsf(pb) * (0.5f + d.mv) + 1.0f;
    } else {
        o.qu = o.qv = 0.0f;
        o.q0 = 0.5f * (o.lo + o.hi);
        o.qh = 0.5f * (o.hi - o.lo) + 1.0f;
    }
    return o.x0 <= o.x1 && o.y0 <= o.y1;
}

// What a pass over the cells does with each (triangle, cell).
// Sky triangles enter a list only where an opaque triangle of the cell
// reaches past them (else what they stop is stopped by nothing: the line is
// clear either way, and the ceiling of a room would stand in every list).
enum Pass { kSkyBound, kCoverBound, kCount, kCountSky, kFill };

// The grids a pass reads and writes, one word per direction and cell: the
// covered depth of cells without sky or before it (bound; after k_sky_pack
// the packed bounds), the covered depth past the sky (past), the least and
// largest depth of sky triangles (sky_lo, sky_hi; null: the scene has none),
// the clear depth (clear; then the fill counter).
struct SkyGrids {
    uint32_t *bound, *past, *sky_lo, *sky_hi, *clear;
    uint2 *info, *pool;
};

__device__ __forceinline__ uint32_t even_up(uint32_t v) { return (v + 1u) & ~1u; }

// Pass PASS for one splat over cells first, first + 32, ... < end of its box.
template <int PASS>
__device__ __forceinline__ void splat_cells(const Splat &s, uint32_t base, float m, int n, const SkyGrids &g,
                                            int first, int end) {
    const int w = s.x1 - s.x0 + 1;
    for (int c = first; c < end; c += 32) {
        const int y = s.y0 + c / w, x = s.x0 + c % w;
        const float xc = (float)x + 0.5f, yc = (float)y + 0.5f;
        float in = kDepthLevels;
#pragma unroll
        for (int e = 0; e < 3; e++) {
            const float v = s.ea[e] * xc + s.eb[e] * yc + s.ec[e];
            in = fminf(in, PASS == kCoverBound ? v - s.te[e] : v + s.te[e]);
        }
        if (!(in >= 0.0f)) continue;
        const uint32_t cell = base + (uint32_t)(y * n + x);
        const float qc = s.q0 + s.qu * xc + s.qv * yc;
        const float low = fmaxf(s.lo, qc - s.qh), high = fminf(s.hi, qc + s.qh);
        const uint32_t top = (uint32_t)fminf(fmaxf(ceilf(high + m), 1.0f), 65534.0f);
        const uint32_t bot = (uint32_t)fminf(fmaxf(floorf(low - m), 0.0f), 65534.0f);
        if (PASS == kSkyBound) {
            atomicMin(g.sky_lo + cell, bot);
            atomicMax(g.sky_hi + cell, top);
        } else if (PASS == kCoverBound) {
            if (!g.sky_lo || top < g.sky_lo[cell]) {
                if (bot > 0u) atomicMax(g.bound + cell, bot);
            } else if (bot > even_up(g.sky_hi[cell])) {
                atomicMax(g.past + cell, bot);
            }
        } else if (PASS == kCount) {
            const uint32_t past = g.sky_lo ? g.past[cell] : 0u;
            if (past) {
                if (top < past && bot > even_up(g.sky_hi[cell])) continue;
                atomicAdd(&g.info[cell].y, 1u);
                g.info[cell].x = 1u;
            } else {
                if (top < g.bound[cell]) continue;
                atomicMax(g.clear + cell, top);
                atomicAdd(&g.info[cell].y, 1u);
                if (g.sky_lo && top >= g.sky_lo[cell]) g.info[cell].x = 1u;
            }
        } else if (PASS == kCountSky) {
            if (g.info[cell].x) atomicAdd(&g.info[cell].y, 1u);
        } else {
            const uint2 run = g.info[cell];
            if (s.flags & kSky) {
                if (!(run.y & kSkyCellFlag)) continue;
            } else {
                const uint32_t b = g.bound[cell], lim = b & 0xffffu;
                if (top < lim && (!(b & kSkyPast) || bot > ((b & ~kSkyPast) >> 16) * 2u)) continue;
            }
            const uint32_t slot = atomicAdd(g.clear + cell, 1u);
            if (slot < (run.y & ~kSkyCellFlag)) g.pool[run.x + slot] = make_uint2((uint32_t)s.rec, top);
        }
    }
}

__device__ __forceinline__ int splat_size(const Splat &s) { return (s.x1 - s.x0 + 1) * (s.y1 - s.y0 + 1); }

// Splats of more cells than this (a room's walls) are left to k_sky_large,
// where kLargeSlices warps share each: a warp that took 32 of them in a row
// was the whole pass's time (4 ms of it in a room of 128 x 128 cells).
constexpr int kLargeCells = 512, kLargeSlices = 32;

// Lane l < batch of a warp readies pair (first + l), then the warp goes through
// the (at most 32) pairs together, 32 cells at a time; pairs are triangle-major, so a
// warp's pairs are mostly one triangle seen along 32 directions.  Bound by
// the cells' instructions and atomics; the readying (a hundred instructions)
// would cost as much again if every lane repeated it.  The pairs' splats that
// are too large go to large[0 ..], counted in *nlarge.
template <int PASS>
__global__ void __launch_bounds__(kThreads) k_sky_cells(const SkyTri *__restrict__ tris, int64_t ntris, int batch,
                                                        const float4 *__restrict__ planes,
                                                        const SkyDir *__restrict__ dirs, int n, SkyGrids g,
                                                        uint32_t *__restrict__ large, unsigned int *__restrict__ nlarge) {
    __shared__ Splat sh[kWarps][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int64_t pairs = ntris * kNumAnorms;
    const int64_t stride = (int64_t)gridDim.x * kWarps * batch;
    for (int64_t p0 = ((int64_t)blockIdx.x * kWarps + wid) * batch; p0 < pairs; p0 += stride) {
        const int64_t p = p0 + lane;
        bool on = false;
        int dir = 0;
        float mq = 0.0f;
        if (lane < batch && p < pairs) {
            const int64_t t = p / kNumAnorms;
            dir = (int)(p - t * kNumAnorms);
            const SkyTri tri = tris[t];
            if (tri.rec >= 0) {
                mq = dirs[dir].mq;
                on = make_splat(tri, __ldg(planes + tri.rec), dirs[dir], n, sh[wid][lane]);
                if (PASS == kCoverBound) on = on && (sh[wid][lane].flags & kCover) != 0;
                if (on && splat_size(sh[wid][lane]) > kLargeCells) {
                    large[atomicAdd(nlarge, 1u)] = (uint32_t)p;
                    on = false;
                }
            }
        }
        unsigned todo = __ballot_sync(0xffffffffu, on);
        __syncwarp();
        while (todo) {
            const int l = __ffs(todo) - 1;
            todo &= todo - 1u;
            const Splat s = sh[wid][l];
            const uint32_t base = (uint32_t)(__shfl_sync(0xffffffffu, dir, l) * n) * (uint32_t)n;
            splat_cells<PASS>(s, base, __shfl_sync(0xffffffffu, mq, l), n, g, lane, splat_size(s));
        }
        __syncwarp();
    }
}

// The large splats of a pass, kLargeSlices warps to each.
template <int PASS>
__global__ void __launch_bounds__(kThreads) k_sky_large(const SkyTri *__restrict__ tris,
                                                        const float4 *__restrict__ planes,
                                                        const SkyDir *__restrict__ dirs, int n, SkyGrids g,
                                                        const uint32_t *__restrict__ large,
                                                        const unsigned int *__restrict__ nlarge) {
    const int lane = threadIdx.x & 31;
    const int64_t items = (int64_t)*nlarge * kLargeSlices;
    const int64_t stride = (int64_t)gridDim.x * kWarps;
    for (int64_t i = (int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5); i < items; i += stride) {
        const uint32_t p = large[i / kLargeSlices];
        const int slice = (int)(i % kLargeSlices);
        const SkyTri tri = tris[p / kNumAnorms];
        const SkyDir &d = dirs[p % kNumAnorms];
        Splat s;
        if (!make_splat(tri, __ldg(planes + tri.rec), d, n, s)) continue;
        const int size = splat_size(s), part = ((size + kLargeSlices - 1) / kLargeSlices + 31) & ~31;
        splat_cells<PASS>(s, (uint32_t)((p % kNumAnorms) * n) * (uint32_t)n, d.mq, n, g, slice * part + lane,
                          min(size, (slice + 1) * part));
    }
}

// Between counting and filling: each cell takes its run of the pool (block
// scan, one atomic per block), the two bounds are packed, and `clear` becomes
// the fill counter.  The cursor counts in 64 bits: coincident triangles put
// thousands of entries into every cell, and past 2^32 the runs' starts would
// wrap (build gives up on such maps before anything is filled).
__global__ void __launch_bounds__(256) k_sky_pack(SkyGrids g, int64_t cells, unsigned long long *__restrict__ cursor) {
    __shared__ uint32_t warp_sum[8];
    __shared__ uint32_t base_sh;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int64_t c0 = (int64_t)blockIdx.x * 256; c0 < cells; c0 += (int64_t)gridDim.x * 256) {
        const int64_t c = c0 + threadIdx.x;
        const uint2 run = c < cells ? g.info[c] : make_uint2(0u, 0u);
        const uint32_t cnt = run.y;
        uint32_t incl = cnt;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        if (lane == 31) warp_sum[wid] = incl;
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t sum = 0;
            for (int k = 0; k < 8; k++) {
                const uint32_t v = warp_sum[k];
                warp_sum[k] = sum;
                sum += v;
            }
            base_sh = sum ? (uint32_t)atomicAdd(cursor, (unsigned long long)sum) : 0u;
        }
        __syncthreads();
        if (c < cells) {
            g.info[c] = make_uint2(base_sh + warp_sum[wid] + incl - cnt, cnt | (run.x ? kSkyCellFlag : 0u));
            const uint32_t past = g.sky_lo ? g.past[c] : 0u;
            g.bound[c] = past ? past | (even_up(g.sky_hi[c]) >> 1) << 16 | kSkyPast
                              : g.bound[c] | (even_up(g.clear[c]) >> 1) << 16;
            g.clear[c] = 0u;
        }
        __syncthreads();
    }
}

// Puts each cell's run in descending order of depth, so that a line stops at
// the first entry behind it: eight lanes per cell, bitonic through shuffles
// for up to eight entries, for up to 32 by the whole warp.  A longer run
// (rare) keeps its order with the largest depth in every entry, so that a line
// never stops early in it.
__device__ __forceinline__ uint2 sort_lanes(uint2 e, int lane, int width) {
    for (int size = 2; size <= width; size <<= 1)
        for (int step = size >> 1; step > 0; step >>= 1) {
            const uint2 o = make_uint2(__shfl_xor_sync(0xffffffffu, e.x, step), __shfl_xor_sync(0xffffffffu, e.y, step));
            const bool keep_max = ((lane & size & (width - 1)) == 0) == ((lane & step) == 0);
            if (keep_max ? o.y > e.y : o.y < e.y) e = o;
        }
    return e;
}

__global__ void __launch_bounds__(kThreads) k_sky_sort(const uint2 *__restrict__ info, uint2 *__restrict__ pool,
                                                       int64_t cells) {
    const int lane = threadIdx.x & 31, sub = lane & 7;
    const int64_t stride = (int64_t)gridDim.x * kWarps * 32;
    for (int64_t c0 = ((int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5)) * 32; c0 < cells; c0 += stride) {
        uint2 run = c0 + lane < cells ? info[c0 + lane] : make_uint2(0u, 0u);
        run.y &= ~kSkyCellFlag;
        for (int i = 0; i < 8; i++) {  // four cells at a time
            const uint32_t at = __shfl_sync(0xffffffffu, run.x, 4 * i + (lane >> 3));
            const uint32_t cnt = __shfl_sync(0xffffffffu, run.y, 4 * i + (lane >> 3));
            const bool few = cnt >= 2 && cnt <= 8;
            if (!__any_sync(0xffffffffu, few)) continue;
            const bool mine = few && (uint32_t)sub < cnt;
            const uint2 e = sort_lanes(mine ? pool[at + sub] : make_uint2(0u, 0u), lane, 8);
            if (mine) pool[at + sub] = e;
        }
        unsigned many = __ballot_sync(0xffffffffu, run.y > 8u);
        while (many) {
            const int l = __ffs(many) - 1;
            many &= many - 1u;
            const uint32_t at = __shfl_sync(0xffffffffu, run.x, l), cnt = __shfl_sync(0xffffffffu, run.y, l);
            if (cnt > 32) {
                for (uint32_t i = lane; i < cnt; i += 32) pool[at + i].y = 65535u;
                continue;
            }
            const uint2 e = sort_lanes((uint32_t)lane < cnt ? pool[at + lane] : make_uint2(0u, 0u), lane, 32);
            if ((uint32_t)lane < cnt) pool[at + lane] = e;
        }
    }
}

// How far the maps reach past the scene's bounds: eight times the walk's slab
// half-thickness for a point as far out as three times the scene's largest
// coordinate.
double sky_margin(const SceneGeom &g) { return 8.0 * std::ldexp(1.0, -17) * (3.0 * (double)g.scale + 1.0); }

// The directions' maps over the scene's bounds, n cells per axis.
void make_dirs(const vrg_env *env, int n, std::vector<SkyDir> &out) {
    static const float anorms[kNumAnorms * 3] = VRG_ANORMS_INIT;
    const SceneGeom &g = env->geom;
    const double m = sky_margin(g);
    out.resize(kNumAnorms);
    for (int j = 0; j < kNumAnorms; j++) {
        SkyDir &o = out[j];
        double d[3];
        for (int c = 0; c < 3; c++) d[c] = anorms[3 * j + c];
        int ax = 0;
        for (int c = 1; c < 3; c++)
            if (std::fabs(d[c]) > std::fabs(d[ax])) ax = c;
        const int a = (ax + 1) % 3, b = (ax + 2) % 3;
        const double ka = d[a] / d[ax], kb = d[b] / d[ax], sign = d[ax] < 0 ? -1.0 : 1.0;
        auto range = [&](int c, double k, double &lo, double &hi) {
            const double e0 = -k * g.bmin[ax], e1 = -k * g.bmax[ax];
            lo = (double)g.bmin[c] + std::min(e0, e1) - m;
            hi = (double)g.bmax[c] + std::max(e0, e1) + m;
        };
        double alo, ahi, blo, bhi;
        range(a, ka, alo, ahi);
        range(b, kb, blo, bhi);
        const double ia = (n - 2) / (ahi - alo), ib = (n - 2) / (bhi - blo);  // one cell of border on each side
        double gu[3] = {0, 0, 0}, gv[3] = {0, 0, 0}, gd[3] = {0, 0, 0};
        gu[a] = ia;
        gu[ax] = -ka * ia;
        gv[b] = ib;
        gv[ax] = -kb * ib;
        o.gu = make_float4((float)gu[0], (float)gu[1], (float)gu[2], (float)(1.0 - alo * ia));
        o.gv = make_float4((float)gv[0], (float)gv[1], (float)gv[2], (float)(1.0 - blo * ib));
        const double q0 = std::min(sign * g.bmin[ax], sign * g.bmax[ax]) - m;
        const double q1 = std::max(sign * g.bmin[ax], sign * g.bmax[ax]) + m;
        const double qs = kDepthLevels / (q1 - q0);
        gd[ax] = sign * qs;
        o.gd = make_float4((float)gd[0], (float)gd[1], (float)gd[2], (float)(1.0 - q0 * qs));
        o.a0 = (float)(alo - 1.0 / ia);
        o.sa = (float)(1.0 / ia);
        o.b0 = (float)(blo - 1.0 / ib);
        o.sb = (float)(1.0 / ib);
        o.ka = (float)ka;
        o.kb = (float)kb;
        o.mu = (float)(m * ia + 2e-3);
        o.mv = (float)(m * ib + 2e-3);
        o.mq = (float)(m * qs + 1.0);
        o.dq0 = (float)(1.0 - q0 * qs);
        o.dqs = (float)qs;
        o.sign = (float)sign;
        o.axis = ax;
        for (int c = 0; c < 3; c++) o.d[c] = anorms[3 * j + c];
    }
}

static_assert(sizeof(SkyTri) == kSkyTriBytes && sizeof(SkyDir) == kSkyDirBytes, "SkyMapSizes counts them");

// Device memory outside the context's reserve.
size_t room_left(vrg_ctx *ctx) {
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    std::lock_guard<std::mutex> lk(ctx->mu);
    return free_b > ctx->hbm_reserve ? free_b - ctx->hbm_reserve : 0;
}

// Builds env's maps with the context's scratch, which one build at a time
// holds until its kernels are done.  The lists may take `room` bytes, or what is
// left when they are counted (asking takes 15 us, so that is asked only where
// `room` is too small).
int build(vrg_env *env, int n, size_t room) {
    vrg_ctx *ctx = env->ctx;
    std::lock_guard<std::mutex> scratch(ctx->scratch_mu);
    DevBuf &tmp = ctx->scratch;
    struct Trim {  // however the build ends
        DevBuf &buf;
        ~Trim() {
            if (buf.bytes > kScratchKept) buf.release();
        }
    } trim{tmp};
    cudaStream_t st = ctx->stream;
    const int64_t nt = env->geom.ntris;
    const SkyMapSizes sizes(nt, n, env->geom.has_sky != 0);
    const size_t cells = sizes.cells;
    // any leaf entry of a triangle holds its record; ids of -1 are the lines'
    // skip id, which no line hits
    const std::vector<int32_t> &refs = env->walk_tree.refs;
    std::vector<int32_t> rec(nt, -1);
    for (size_t r = 0; r < refs.size(); r++)
        if (env->ids[refs[r]] != -1) rec[refs[r]] = (int32_t)r;
    std::vector<SkyTri> tris(nt);  // the sky's first
    int64_t nsky = 0, at = 0;
    for (int sky = 1; sky >= 0; sky--) {
        for (int64_t t = 0; t < nt; t++) {
            if (((env->ids[t] & VRG_TRACE_ID_SKY) != 0) != (sky != 0)) continue;
            SkyTri &o = tris[at++];
            memcpy(o.v, &env->xyz[9 * t], sizeof o.v);
            o.rec = rec[t];
            o.sky = sky;
            o.pad = 0;
        }
        if (sky) nsky = at;
    }
    std::vector<SkyDir> dirs;
    make_dirs(env, n, dirs);
    std::vector<float4> view(4 * kNumAnorms);
    for (int j = 0; j < kNumAnorms; j++) {
        view[4 * j] = dirs[j].gu;
        view[4 * j].w -= 0.5f;  // the lookup rounds to the nearest cell
        view[4 * j + 1] = dirs[j].gv;
        view[4 * j + 1].w -= 0.5f;
        view[4 * j + 2] = dirs[j].gd;
        view[4 * j + 3] = make_float4(dirs[j].d[0], dirs[j].d[1], dirs[j].d[2], 0.0f);
    }
    const bool has_sky = env->geom.has_sky != 0;
    const size_t vbytes = sizes.view;
    VRG_CUDA(ctx, env->d_sky_cells.reserve(sizes.kept));
    VRG_CUDA(ctx, tmp.reserve(sizes.scratch));
    SkyTri *d_tris = reinterpret_cast<SkyTri *>(tmp.as<char>() + sizes.tri_at);
    SkyDir *d_dirs = reinterpret_cast<SkyDir *>(tmp.as<char>() + sizes.dir_at);
    char *base = env->d_sky_cells.as<char>();
    SkyGrids g{};
    g.info = reinterpret_cast<uint2 *>(base + vbytes);
    g.bound = reinterpret_cast<uint32_t *>(base + vbytes + 8 * cells);
    unsigned long long *cursor = tmp.as<unsigned long long>();
    g.clear = tmp.as<uint32_t>() + 64;
    uint32_t *large = g.clear + cells * (has_sky ? 4 : 1);
    if (has_sky) {
        g.past = g.clear + cells;
        g.sky_hi = g.past + cells;
        g.sky_lo = g.sky_hi + cells;
    }
    VRG_CUDA(ctx, cudaMemcpyAsync(base, view.data(), vbytes, cudaMemcpyHostToDevice, st));
    VRG_CUDA(ctx, cudaMemcpyAsync(d_tris, tris.data(), sizeof(SkyTri) * (size_t)nt, cudaMemcpyHostToDevice, st));
    VRG_CUDA(ctx, cudaMemcpyAsync(d_dirs, dirs.data(), sizeof(SkyDir) * kNumAnorms, cudaMemcpyHostToDevice, st));
    VRG_CUDA(ctx, cudaMemsetAsync(g.info, 0, 12 * cells, st));
    VRG_CUDA(ctx, cudaMemsetAsync(cursor, 0, 256 + 4 * cells * (has_sky ? 3 : 1), st));
    if (has_sky) VRG_CUDA(ctx, cudaMemsetAsync(g.sky_lo, 0xff, 4 * cells, st));
    const DevScene s = scene_view(env);
    cudaEvent_t ev = nullptr;
    unsigned int passes = 0;  // each pass counts its large splats in a word of its own after the cursor
    auto cells_pass = [&](auto kernel, auto kernel_large, int64_t first, int64_t count) {
        const SkyTri *t = d_tris + first;
        unsigned int *nlarge = reinterpret_cast<unsigned int *>(cursor + 1) + passes++;
        // a small scene's pairs go to more warps, fewer each
        const int64_t warps = (int64_t)ctx->num_sms * 48;
        const int batch = (int)std::min<int64_t>(32, std::max<int64_t>(1, count * kNumAnorms / warps));
        timing_begin(ctx, "sky_map", &ev);
        kernel<<<(int)std::min<int64_t>((count * kNumAnorms + kWarps * batch - 1) / (kWarps * batch),
                                        (int64_t)ctx->num_sms * 64), kThreads, 0, st>>>(t, count, batch, s.leaf_planes, d_dirs, n, g, large, nlarge);
        cudaError_t e = cudaGetLastError();
        timing_end(ctx, "sky_map", ev);
        if (e != cudaSuccess) return e;
        timing_begin(ctx, "sky_map", &ev);
        kernel_large<<<ctx->num_sms * 8, kThreads, 0, st>>>(t, s.leaf_planes, d_dirs, n, g, large, nlarge);
        e = cudaGetLastError();
        timing_end(ctx, "sky_map", ev);
        return e;
    };
    if (has_sky) VRG_CUDA(ctx, cells_pass(k_sky_cells<kSkyBound>, k_sky_large<kSkyBound>, 0, nsky));
    if (nt > nsky) {
        VRG_CUDA(ctx, cells_pass(k_sky_cells<kCoverBound>, k_sky_large<kCoverBound>, nsky, nt - nsky));
        VRG_CUDA(ctx, cells_pass(k_sky_cells<kCount>, k_sky_large<kCount>, nsky, nt - nsky));
    }
    if (has_sky) VRG_CUDA(ctx, cells_pass(k_sky_cells<kCountSky>, k_sky_large<kCountSky>, 0, nsky));
    timing_begin(ctx, "sky_map", &ev);
    k_sky_pack<<<(int)std::min<size_t>((cells + 255) / 256, (size_t)ctx->num_sms * 8), 256, 0, st>>>(
        g, (int64_t)cells, cursor);
    VRG_CUDA(ctx, cudaGetLastError());
    timing_end(ctx, "sky_map", ev);
    uint64_t entries = 0;
    VRG_CUDA(ctx, cudaMemcpyAsync(&entries, cursor, 8, cudaMemcpyDeviceToHost, st));
    VRG_CUDA(ctx, cudaStreamSynchronize(st));
    if (!sky_pool_indexable(entries)) return fail(ctx, VRG_ERR_UNSUPPORTED, "sky maps of more than 2^32 entries");
    if (8 * (size_t)entries > room && 8 * (size_t)entries > room_left(ctx)) return fail(ctx, VRG_ERR_NOMEM, "no room for the sky maps' lists");
    VRG_CUDA(ctx, env->d_sky_pool.reserve(8 * (size_t)entries));
    g.pool = env->d_sky_pool.as<uint2>();
    VRG_CUDA(ctx, cells_pass(k_sky_cells<kFill>, k_sky_large<kFill>, 0, nt));
    timing_begin(ctx, "sky_map", &ev);
    k_sky_sort<<<(int)std::min<size_t>((cells + kThreads - 1) / kThreads, (size_t)ctx->num_sms * 32), kThreads, 0,
                 st>>>(g.info, g.pool, (int64_t)cells);
    VRG_CUDA(ctx, cudaGetLastError());
    timing_end(ctx, "sky_map", ev);
    // later calls may launch on another stream, and the scratch is free again
    VRG_CUDA(ctx, cudaStreamSynchronize(st));
    env->sky_n = n;
    return VRG_OK;
}

}  // namespace

SkyView sky_view(const vrg_env *env) {
    SkyView v{};
    if (env->sky_n <= 0) return v;
    const size_t cells = (size_t)kNumAnorms * env->sky_n * env->sky_n;
    char *base = env->d_sky_cells.as<char>();
    const size_t vbytes = 4 * kNumAnorms * sizeof(float4);
    v.dirs = reinterpret_cast<const float4 *>(base);
    v.info = reinterpret_cast<const uint2 *>(base + vbytes);
    v.bound = reinterpret_cast<const uint32_t *>(base + vbytes + 8 * cells);
    v.pool = env->d_sky_pool.as<uint2>();
    v.n = env->sky_n;
    return v;
}

bool faces_in_sky_range(const vrg_env *env) {
    const SceneGeom &g = env->geom;
    const double m = sky_margin(g);
    for (int c = 0; c < 3; c++) {
        const double far = 128.0 * ((double)g.bmax[c] - g.bmin[c] + 2.0 * m) - 1.0;
        for (int32_t f = 0; f < env->nfaces; f++) {
            const double p = env->f_corner[3 * f + c], u = env->f_u[3 * f + c], v = env->f_v[3 * f + c];
            const double lo = p + std::min(0.0, u) + std::min(0.0, v), hi = p + std::max(0.0, u) + std::max(0.0, v);
            if (!(lo >= g.bmin[c] - far && hi <= g.bmax[c] + far)) return false;
        }
    }
    return true;
}

int64_t sky_map_points(const vrg_env *env) { return std::max<int64_t>(24 * env->geom.ntris, 40000); }

bool wants_sky_map(const vrg_env *env) {
    for (const vrg_light &l : env->lights)
        if (l.type == VRG_EMIT_SKYAMBIENT) return true;
    return false;
}

bool may_have_sky_map(const vrg_env *env) {
    const int64_t nt = env->geom.ntris;
    return env->sky_n >= 0 && env->faces_inside && env->faces_in_sky_range && nt >= 1 && nt <= (int64_t)1 << 23 &&
           env->geom.scale <= 16000.0f;
}

bool use_sky_map(vrg_env *env, int64_t points) {
    if (!wants_sky_map(env) || !may_have_sky_map(env)) return false;
    if (env->sky_n > 0) return true;
    // a build costs about what 24 sample points per triangle cost to walk, and
    // never less than 40,000 points: points walked so far count towards it, so
    // that a scene asked for a few at a time gets its maps when they repay
    env->sky_demand += points;
    return env->sky_demand >= sky_map_points(env) && have_sky_map(env);
}

bool use_sky_maps(const std::vector<vrg_env *> &envs, const std::vector<int64_t> &points) {
    // the maps serve a launch over several scenes when all that want them have
    // them, so none is built unless all can be, once the points that would else
    // be walked, with those walked so far, repay the builds that are left.  One
    // launch walks many scenes' points 5 ns apart from the maps' (twelve scenes
    // of 64 to 4,096 faces, 1.9 M points: 13.1 and 3.7 ms), and their builds, one
    // after the other, take 0.65 ms and 0.17 us a triangle each (together 11.3).
    std::vector<vrg_env *> unbuilt;
    int64_t asked = 0, repay = 0;
    bool any = false;
    for (size_t e = 0; e < envs.size(); e++) {
        if (!wants_sky_map(envs[e])) continue;
        if (!may_have_sky_map(envs[e])) return false;
        any = true;
        if (envs[e]->sky_n > 0) {
            asked += points[e];
            continue;
        }
        unbuilt.push_back(envs[e]);
        asked += envs[e]->sky_demand += points[e];
        repay += 130000 + 34 * envs[e]->geom.ntris;
    }
    if (!any || asked < repay) return false;
    for (vrg_env *env : unbuilt)
        if (!have_sky_map(env)) return false;
    return true;
}

bool have_sky_map(vrg_env *env) {
    if (env->sky_n != 0) return env->sky_n > 0;
    vrg_ctx *ctx = env->ctx;
    const int64_t nt = env->geom.ntris;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(ctx->stream, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) return false;
    // three cells per direction and triangle: on the 8,208-triangle room a gather
    // takes 2.64 / 2.50 / 2.38 ms with 2 / 3 / 6 of them, a first one with the
    // build 4.4 / 4.6 / 5.8 ms.  At least 96 cells an axis: where boxes are few
    // most lines pass them, and it is the wide cells around a sample's own box
    // that leave them undecided.  A gather of a 2,064-triangle brush map takes
    // 0.49 / 0.41 / 0.37 ms with 72 / 96 / 128 cells (first 1.43 / 1.40 / 1.65),
    // twelve scenes of 64 to 4,096 faces 4.0 / 3.8 / 3.55 ms at least 32 / 96 / 128
    // (first 14.0 / 14.5 / 16.1).
    const int n = std::min(512, std::max(96, (int)std::sqrt(3.0 * (double)nt) & ~7));
    // the maps and their scratch inside what the context may take; the lists,
    // whose size the build finds out, are asked for there
    const SkyMapSizes sizes(nt, n, env->geom.has_sky != 0);
    const size_t room = room_left(ctx);
    if (room < sizes.kept + sizes.scratch) return false;
    std::string said;
    {
        std::lock_guard<std::mutex> lk(ctx->mu);
        said = ctx->last_error;
    }
    if (build(env, n, room - sizes.kept - sizes.scratch) != VRG_OK) {
        fail(ctx, 0, said);  // the call goes on without: its caller's last error stays
        (void)cudaGetLastError();
        env->d_sky_cells.release();
        env->d_sky_pool.release();
        env->sky_n = -1;  // not tried again for this scene
        return false;
    }
    return true;
}

}  // namespace vrg
