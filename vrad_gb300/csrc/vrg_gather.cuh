// vrg_gather.cuh -- direct-light evaluation at one sample point, shared by the
// single-scene and batched gather kernels.
#pragma once

#include <cstdint>

#include "../../include/vradgpu.h"
#include "vrg_device.h"
#include "vrg_sky.cuh"
#include "vrg_trace.cuh"

namespace vrg {

// Device copy of a light: five 16-byte words.
struct alignas(16) DevLight {
    float4 origin;     // xyz, w = type (as int bits)
    float4 intensity;  // xyz, w = radius
    float4 normal;     // xyz, w = exponent
    float4 attn;       // constant, linear, quadratic, cap_distance
    float4 cone;       // stopdot, stopdot2, start_fade, end_fade
};

__device__ __forceinline__ uint64_t splitmix(uint64_t seed, uint64_t i) {
    uint64_t z = seed + (i + 1ull) * 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// The box around a warp's sample points, and whether they share their normal
// (and are numbers, so that the box holds them all).
struct PointBox {
    float lo[3], hi[3];
    bool one;
};

// Floats as integers of the same order, and back.
__device__ __forceinline__ int ordered_bits(float v) {
    const int b = __float_as_int(v);
    return b ^ ((b >> 31) & 0x7fffffff);
}

__device__ __forceinline__ float ordered_float(int b) { return __int_as_float(b ^ ((b >> 31) & 0x7fffffff)); }

__device__ __forceinline__ PointBox point_box(unsigned lanes, float px, float py, float pz, float nx, float ny,
                                              float nz) {
    PointBox b;
    const float p[3] = {px, py, pz};
#pragma unroll
    for (int c = 0; c < 3; c++) {
        b.lo[c] = ordered_float(__reduce_min_sync(lanes, ordered_bits(p[c])));
        b.hi[c] = ordered_float(__reduce_max_sync(lanes, ordered_bits(p[c])));
    }
    const int lead = __ffs(lanes) - 1;
    const float lx = __shfl_sync(lanes, nx, lead), ly = __shfl_sync(lanes, ny, lead), lz = __shfl_sync(lanes, nz, lead);
    // (a coordinate that is no number takes a bound's place and hides the others')
    b.one = __all_sync(lanes, nx == lx && ny == ly && nz == lz) && b.lo[0] <= b.hi[0] && b.lo[1] <= b.hi[1] &&
            b.lo[2] <= b.hi[2];
    return b;
}

// False for a light that adds to no point of the box: it is out of range, or
// behind the points' common normal.  The range test is the points' own on the
// gaps to the box, which rounding keeps at most as long as theirs; the other
// leaves out 25 times the rounding of the cosine.
__device__ __forceinline__ bool box_may_see(const PointBox &b, const DevLight &light, float nx, float ny, float nz) {
    const float4 o = __ldg(&light.origin);
    const int type = __float_as_int(o.w);
    if (type != VRG_EMIT_POINT && type != VRG_EMIT_SPOTLIGHT) return true;
    const float at[3] = {o.x, o.y, o.z}, n[3] = {nx, ny, nz};
    float gap[3], front = 0.0f, size = 0.0f;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const float u = rsub(at[c], b.lo[c]), v = rsub(at[c], b.hi[c]);
        gap[c] = fmaxf(fmaxf(-u, v), 0.0f);
        front += fmaxf(n[c] * u, n[c] * v);
        size += fabsf(n[c]) * fmaxf(fabsf(u), fabsf(v));
    }
    const float radius = __ldg(&light.intensity).w;
    if (radius > 0.0f && dot3r(gap[0], gap[1], gap[2], gap[0], gap[1], gap[2]) > rmul(radius, radius)) return false;
    return !(b.one && front < -1e-5f * size);
}

// Irradiance at p with normal n, summed over the lights in table order.
// Point / spot: distance cull by radius, cosine at the receiver, falloff
// 1 / ((c + b*d) + a*d*d) with d capped at cap_distance, smoothstep fade
// between start_fade and end_fade, spot cone ramp and exponent, and a
// shadow line to the light.  Sky light: direction -normal.  Sky ambient:
// cosine-weighted fraction of the 162 directions whose line reaches sky.
//
// SKY selects what happens to the sky-type lights (sky light, sky ambient),
// which do not depend on any light position: 0 traces them; 1 traces them
// and stores each one's multiplier (cosine or visible fraction, -1 when it
// adds nothing) in sky[0..]; 2 reads those multipliers instead of tracing.
// With a visibility cache vis (one bit per light, bit li of word li/32),
// mode 1 also stores whether each traced point/spot shadow line reached its
// light, and mode 2 traces only the lights flagged in `edited` (refreshing
// their bits) and takes every other light's visibility from the cache.
// The accumulation order and arithmetic are the same in all modes, so a
// relight that re-traces only edited lights is bit-identical to a full
// gather with the edited table.
// MAP answers the sky ambient's lines from the scene's sky maps (sv) instead
// of walking them; the results are the same.  The warp's `lanes` call
// together, for points of one scene.  They pick the lights within reach of the
// box around their points 32 at a time, one light to a lane, and go through
// those only: the 64 point lights of the 4,096-face room take 0.92 ms instead
// of 1.14.
enum SkyMode { kSkyTrace = 0, kSkyWrite = 1, kSkyRead = 2 };

template <int SKY, int OPT = 0, int WM = kWallAny, bool MAP = false>
static __device__ void gather_point(const DevScene &s, const SkyView &sv, unsigned lanes, const DevLight *__restrict__ lights, int nl,
                                    float px, float py, float pz, float nx, float ny, float nz,
                                    float &r, float &g, float &b, uint32_t &rays,
                                    float *__restrict__ sky = nullptr, uint32_t *__restrict__ vis = nullptr,
                                    const uint32_t *__restrict__ edited = nullptr) {
    float ar = 0.0f, ag = 0.0f, ab = 0.0f;
    const int lane = threadIdx.x & 31;
    float mapped = -1.0f;  // the sky ambient's multiplier, whichever light asks
    uint32_t mapped_rays = 0;
    if (MAP) {
        bool ambient = false;
        for (int li = __popc(lanes & ((1u << lane) - 1u)); li < nl; li += __popc(lanes))
            ambient = ambient || __float_as_int(__ldg(&lights[li].origin).w) == VRG_EMIT_SKYAMBIENT;
        if (__any_sync(lanes, ambient)) mapped = sky_fraction(s, sv, lanes, px, py, pz, nx, ny, nz, mapped_rays);
    }
    for (int l0 = 0; l0 < nl; l0 += 32) {
        // the lights that may add to one of the lanes (those of absent lanes
        // count as such), in table order
        unsigned todo;
        {
            const PointBox box = point_box(lanes, px, py, pz, nx, ny, nz);
            todo = __ballot_sync(lanes, l0 + lane < nl && box_may_see(box, lights[min(l0 + lane, nl - 1)], nx, ny, nz));
        }
        todo |= ~lanes & (nl - l0 >= 32 ? 0xffffffffu : (1u << (nl - l0)) - 1u);
        while (todo) {
            const int li = l0 + __ffs(todo) - 1;
            todo &= todo - 1u;
            const float4 lo = __ldg(&lights[li].origin);
            const int type = __float_as_int(lo.w);
            const float4 li_i = __ldg(&lights[li].intensity);
            if (type == VRG_EMIT_POINT || type == VRG_EMIT_SPOTLIGHT) {
                const float dlx = rsub(lo.x, px), dly = rsub(lo.y, py), dlz = rsub(lo.z, pz);
                const float dist2 = dot3r(dlx, dly, dlz, dlx, dly, dlz);
                const float radius = li_i.w;
                if (radius > 0.0f && dist2 > rmul(radius, radius)) continue;
                if (dist2 == 0.0f) continue;
                const float dist = rsqrt_rn(dist2);
                const float inv = rrcp(dist);
                const float Lx = rmul(dlx, inv), Ly = rmul(dly, inv), Lz = rmul(dlz, inv);
                const float cosr = dot3r(nx, ny, nz, Lx, Ly, Lz);
                if (!(cosr > 0.0f)) continue;
                const float4 at = __ldg(&lights[li].attn);
                float dc = dist, dc2 = dist2;
                if (dist > at.w) {
                    dc = at.w;
                    dc2 = rmul(at.w, at.w);
                }
                const float denom = radd(radd(at.x, rmul(at.y, dc)), rmul(at.z, dc2));
                if (!(denom > 0.0f)) continue;
                float f = rrcp(denom);
                const float4 cn = __ldg(&lights[li].cone);
                if (cn.w > cn.z && dist > cn.z) {
                    if (dist >= cn.w) continue;
                    const float sfr = rdiv(rsub(dist, cn.z), rsub(cn.w, cn.z));
                    const float om = rsub(1.0f, sfr);
                    f = rmul(f, rmul(rmul(om, om), radd(1.0f, rmul(2.0f, sfr))));
                }
                if (type == VRG_EMIT_SPOTLIGHT) {
                    const float4 ln = __ldg(&lights[li].normal);
                    const float dot2 = -dot3r(Lx, Ly, Lz, ln.x, ln.y, ln.z);
                    if (!(dot2 > cn.y)) continue;
                    if (dot2 < cn.x) f = rmul(f, rdiv(rsub(dot2, cn.y), rsub(cn.x, cn.y)));
                    if (ln.w == 1.0f) f = rmul(f, dot2);
                    else if (ln.w != 0.0f) f = rmul(f, powf(dot2, ln.w));
                }
                bool occ;
                const uint32_t bit = 1u << (li & 31);
                if (SKY == kSkyRead && vis && !(__ldg(edited + (li >> 5)) & bit)) {
                    occ = !(vis[li >> 5] & bit);
                } else {
                    rays++;
                    occ = line_occluded<OPT, WM>(s, make_line(px, py, pz, lo.x, lo.y, lo.z), -1);
                    if (SKY != kSkyTrace && vis) {
                        if (occ) vis[li >> 5] &= ~bit;
                        else vis[li >> 5] |= bit;
                    }
                }
                if (occ) continue;
                const float sc = rmul(f, cosr);
                ar = radd(ar, rmul(li_i.x, sc));
                ag = radd(ag, rmul(li_i.y, sc));
                ab = radd(ab, rmul(li_i.z, sc));
            } else if (type == VRG_EMIT_SKYLIGHT || type == VRG_EMIT_SKYAMBIENT) {
                float m = -1.0f;  // multiplier of the intensity; -1: adds nothing
                if (SKY == kSkyRead) {
                    m = *sky++;
                } else if (type == VRG_EMIT_SKYLIGHT) {
                    const float4 ln = __ldg(&lights[li].normal);
                    const float dx = -ln.x, dy = -ln.y, dz = -ln.z;
                    const float cosr = dot3r(nx, ny, nz, dx, dy, dz);
                    if (cosr > 0.0f) {
                        rays++;
                        const Line L = make_line(px, py, pz, radd(px, rmul(dx, kMaxTraceLength)),
                                                 radd(py, rmul(dy, kMaxTraceLength)),
                                                 radd(pz, rmul(dz, kMaxTraceLength)));
                        if (!line_occluded<OPT, WM>(s, L, -1)) m = cosr;
                    }
                } else if (MAP) {
                    m = mapped;
                    rays += mapped_rays;
                } else {
                    float sw = 0.0f, sum = 0.0f;
                    for (int j = 0; j < kNumAnorms; j++) {
                        const float ax = c_anorms[3 * j], ay = c_anorms[3 * j + 1], az = c_anorms[3 * j + 2];
                        const float w = dot3r(nx, ny, nz, ax, ay, az);
                        if (!(w > 0.0f)) continue;
                        sw = radd(sw, w);
                        rays++;
                        const Line L = make_line(px, py, pz, radd(px, rmul(ax, kMaxTraceLength)),
                                                 radd(py, rmul(ay, kMaxTraceLength)),
                                                 radd(pz, rmul(az, kMaxTraceLength)));
                        if (!line_occluded<OPT, WM>(s, L, -1)) sum = radd(sum, w);
                    }
                    if (sw > 0.0f) m = rdiv(sum, sw);
                }
                if (SKY == kSkyWrite) *sky++ = m;
                if (m >= 0.0f) {
                    ar = radd(ar, rmul(li_i.x, m));
                    ag = radd(ag, rmul(li_i.y, m));
                    ab = radd(ab, rmul(li_i.z, m));
                }
            }
        }
    }
    r = ar;
    g = ag;
    b = ab;
}

// Luxel supersample position: face f spans corner + U*su + V*sv; sample k of
// luxel (iu, iv) with global luxel index lux uses h = splitmix(seed, 4*lux+k),
// r1 = (h >> 40) * 2^-24, r2 = ((h >> 16) & 0xffffff) * 2^-24 and
// su = (iu + ((k & 1) + r1) * 0.5) * (1/nu), sv = (iv + ((k >> 1) + r2) * 0.5) * (1/nv)
// (S = 1: the luxel centre), then p = ((corner + U*su) + V*sv) + N*0.125.
__device__ __forceinline__ void luxel_sample(const FaceRec &f, int64_t lux, int iu, int iv, int k,
                                             int ss, uint64_t seed, float &px, float &py,
                                             float &pz) {
    const float inu = rrcp((float)f.nu), inv = rrcp((float)f.nv);
    float su, sv;
    if (ss == 4) {
        const uint64_t h = splitmix(seed, (uint64_t)(lux * 4 + k));
        const float r1 = rmul((float)(uint32_t)(h >> 40), 5.9604644775390625e-08f);
        const float r2 = rmul((float)(uint32_t)((h >> 16) & 0xffffffu), 5.9604644775390625e-08f);
        su = rmul(radd((float)iu, rmul(radd((float)(k & 1), r1), 0.5f)), inu);
        sv = rmul(radd((float)iv, rmul(radd((float)(k >> 1), r2), 0.5f)), inv);
    } else {
        su = rmul(radd((float)iu, 0.5f), inu);
        sv = rmul(radd((float)iv, 0.5f), inv);
    }
    px = radd(radd(radd(f.corner.x, rmul(f.u.x, su)), rmul(f.v.x, sv)), rmul(f.normal.x, kSampleOffset));
    py = radd(radd(radd(f.corner.y, rmul(f.u.y, su)), rmul(f.v.y, sv)), rmul(f.normal.y, kSampleOffset));
    pz = radd(radd(radd(f.corner.z, rmul(f.u.z, su)), rmul(f.v.z, sv)), rmul(f.normal.z, kSampleOffset));
}

// Walk order of a face's luxels in 4 x 2 tiles: ordinal o (0 .. nu*nv-1)
// -> (iu, iv), tiles left to right within bands of two rows (one row in the
// last band of a face with odd nv), the last tile of a band narrower when
// nu is not a multiple of 4.  A bijection, so every luxel is visited once;
// a warp's 8 consecutive luxels then cover a 64 x 32-unit patch of the face
// instead of a 128-unit strip, and its lanes' shadow lines stay together
// longer.
__device__ __forceinline__ void tile_luxel(int64_t o, int nu, int nv, int &iu, int &iv) {
    const int band = (int)(o / (2 * (int64_t)nu));
    const int h = (2 * band + 1 < nv) ? 2 : 1;
    const int r = (int)(o - (int64_t)band * 2 * nu);
    const int c = r / (4 * h);
    const int q = r - c * 4 * h;
    const int w = min(4, nu - 4 * c);
    iu = 4 * c + q % w;
    iv = 2 * band + q / w;
}

__device__ __forceinline__ int find_face(const int64_t *__restrict__ off, int nfaces, int64_t lux) {
    int lo = 0, hi = nfaces - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(off + mid) <= lux) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

}  // namespace vrg
