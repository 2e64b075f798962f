// trace.cu -- batched ray queries against a resident scene (Trace4Rays,
// raytracer/environment.go:140-145, and TestLineDoesHitSky,
// raytracer/trace/testline.go:18-94).
#include <algorithm>

#include "vrg_internal.h"
#include "vrg_bvh.cuh"
#include "vrg_trace.cuh"

namespace vrg {

namespace {

constexpr int kThreads = 128;

__device__ __forceinline__ void load3(const float *p, int64_t i, float &x, float &y, float &z) {
    x = __ldg(p + 3 * i);
    y = __ldg(p + 3 * i + 1);
    z = __ldg(p + 3 * i + 2);
}

// The refill loops read each line's end points when a lane takes the line,
// one lane at a time and out of step with its neighbours, so a line that is
// not yet in L2 costs the lane a full HBM round trip.  At launch every
// thread asks L2 for its share of the two end-point arrays (128-byte lines,
// addresses inside the arrays only), so they stream in at full bandwidth
// instead.
__device__ __forceinline__ void prefetch_lines(const float *start, const float *stop, int64_t n) {
    const int64_t bytes = 12 * n;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x * 128;
    const char *a = reinterpret_cast<const char *>(start), *b = reinterpret_cast<const char *>(stop);
    for (int64_t off = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 128; off < bytes; off += stride) {
        asm volatile("prefetch.global.L2 [%0];" ::"l"(a + off));
        asm volatile("prefetch.global.L2 [%0];" ::"l"(b + off));
    }
}

// Lines and rays through the hierarchy, one per lane with refill: a round
// either takes the lanes at inner nodes STEPS nodes further, or, when LEAVES
// lanes wait at leaves or none is at a node, tests those lanes' triangles;
// lanes that are done take new lines when at least FILL are.
enum Query { kQMask, kQMaskHit, kQClosest, kQLines };
struct QueryArgs {
    const float *a, *b;        // start and stop points, or origins and directions
    const float *tmin, *tmax;  // kQClosest
    int64_t n;
    int32_t skip;
    uint32_t *mask;
    int32_t *hit;
    float *t, *frac;
    unsigned long long *work;
};

template <Query Q, int STEPS, int LEAVES, int FILL, int MINB, bool ORDER>
__global__ void __launch_bounds__(kThreads, MINB) k_bvh(DevScene s, BvhView bv, QueryArgs q) {
    constexpr int MODE = Q == kQMask || Q == kQLines ? kSkyOcc : kClosest;
    constexpr int OPT = Q == kQClosest ? 0 : kOptSign;
    if (Q != kQClosest) prefetch_lines(q.a, q.b, q.n);
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    unsigned out_of_work = 0u;  // lanes that found no line left
    int64_t ri = -1;            // this lane's line (-1: none)
    bool active = false;
    Ray ray{};
    BoxRay rp{};
    float t0 = 0.0f, len = 0.0f, any_limit = 0.0f;
    uint32_t cur = 0u;
    int sp = 0;
    int32_t best = -1;
    float best_t = kInf;
    uint2 stk[kBvhStack];
    for (;;) {
        const unsigned busy = __ballot_sync(full, active);
        const unsigned idle = ~busy & ~out_of_work;
        if (idle == 0u && busy == 0u) break;
        if (idle != 0u && (__popc(idle) >= FILL || busy == 0u)) {
            const int leader = __ffs(idle) - 1;
            unsigned long long base = 0;
            if (lane == leader) base = atomicAdd(q.work, (unsigned long long)__popc(idle));
            base = __shfl_sync(full, base, leader);
            if ((idle >> lane) & 1u) {
                ri = (int64_t)base + __popc(idle & below);
                if (ri < q.n) {
                    best = -1;
                    best_t = kInf;
                    sp = 0;
                    cur = 0u;
                    if (Q == kQClosest) {
                        load3(q.a, ri, ray.ox, ray.oy, ray.oz);
                        load3(q.b, ri, ray.dx, ray.dy, ray.dz);
                        t0 = __ldg(q.tmin + ri);
                        len = __ldg(q.tmax + ri);
                        rp = box_ray(s.g, ray, ray_slack(s.g, ray.ox, ray.oy, ray.oz));
                        active = bv.nodes && t0 <= len && has_direction(ray);
                    } else {
                        float sx, sy, sz, ex, ey, ez;
                        load3(q.a, ri, sx, sy, sz);
                        load3(q.b, ri, ex, ey, ez);
                        const LinePlan p = plan_line(s, make_line(sx, sy, sz, ex, ey, ez));
                        ray = p.ray;
                        rp = box_ray(s.g, ray, p.slack);
                        len = p.len;
                        any_limit = p.any_limit;
                        active = bv.nodes && !p.trivial;
                    }
                    if (!active) {
                        if (Q == kQMaskHit || Q == kQClosest) {
                            q.hit[ri] = -1;
                            q.t[ri] = kInf;
                        }
                        if (Q == kQLines) q.frac[ri] = 1.0f;
                    }
                }
            }
            out_of_work = __ballot_sync(full, ri >= q.n);
        }
        const bool at_leaf = active && (cur & kBvhLeafBit) != 0u;
        const unsigned leaves = __ballot_sync(full, at_leaf);
        const unsigned inner = __ballot_sync(full, active && !at_leaf);
        bool done = false;
        if (inner == 0u || __popc(leaves) >= LEAVES) {
            if (at_leaf)
                done = bvh_leaf<MODE, OPT>(s, bv, ray, t0, len, q.skip, any_limit, cur, best, best_t) ||
                       !bvh_pop(stk, sp, best_t, cur);
        } else {
#pragma unroll
            for (int u = 0; u < STEPS; u++)
                if (active && !done && !(cur & kBvhLeafBit))
                    if (!bvh_step<ORDER>(bv, rp, t0, fminf(len, best_t), stk, sp, cur)) done = !bvh_pop(stk, sp, best_t, cur);
        }
        if (done) {
            active = false;
            bool occ;
            if (MODE == kClosest)
                occ = best >= 0 && (__ldg(&s.tri_ids[best]) & kTraceIdSky) == 0;
            else
                occ = best >= 0 && (best_t < any_limit || (__ldg(&s.tri_ids[best]) & kTraceIdSky) == 0);
            if (Q == kQMaskHit || Q == kQClosest) {
                q.hit[ri] = best;
                q.t[ri] = best_t;
            }
            if (Q == kQLines) q.frac[ri] = occ ? 0.0f : 1.0f;
            if ((Q == kQMask || Q == kQMaskHit) && occ) atomicOr(q.mask + (ri >> 5), 1u << (ri & 31));
        }
    }
}

// Few rays: every triangle is tested, 32 rays to a block and the triangles
// split over blockIdx.y and the block's warps.  A walk is a chain of dependent
// loads whatever the number of rays (23 us for four rays among 12,300
// triangles, 37 for 33); testing all of them keeps the whole GPU busy (10 and
// 12 us) until the tests cost more: about 4 us a million, a lane of the 32 or
// other taking the whole test nearly every time.  Each block takes the least
// (t, index) of its share per ray; blocks of one group of rays meet in `keys`,
// and the last one to finish writes the answers and leaves keys and counters
// as it found them.  The answer is the walk's: both are what testing every
// triangle gives.
constexpr int kFewWarps = 4, kFewUnroll = 4;
constexpr unsigned long long kFewNone = ~0ull;

template <Query Q>
__global__ void __launch_bounds__(32 * kFewWarps) k_few(DevScene s, QueryArgs q, int64_t base, int ntris, int slices,
                                                        unsigned long long *__restrict__ keys,
                                                        unsigned int *__restrict__ done) {
    __shared__ unsigned long long least[kFewWarps][32];
    __shared__ bool last_sh;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int64_t i = (int64_t)blockIdx.x * 32 + lane;
    Ray ray{0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    float t0 = 0.0f, t1 = -1.0f;
    if (i < q.n) {
        if (Q == kQClosest) {
            load3(q.a, i, ray.ox, ray.oy, ray.oz);
            load3(q.b, i, ray.dx, ray.dy, ray.dz);
            t0 = __ldg(q.tmin + i);
            t1 = __ldg(q.tmax + i);
        } else {
            float sx, sy, sz, ex, ey, ez;
            load3(q.a, i, sx, sy, sz);
            load3(q.b, i, ex, ey, ez);
            const Line L = make_line(sx, sy, sz, ex, ey, ez);
            ray = Ray{L.ox, L.oy, L.oz, L.dx, L.dy, L.dz};
            t1 = L.len;  // zero length: nothing in [0, 0)
        }
    }
    // this warp's triangles: first, first + kFewWarps, ... < end
    const int share = (ntris + slices - 1) / slices;
    const int first = blockIdx.y * share + wid, end = min(ntris, ((int)blockIdx.y + 1) * share);
    const float4 *planes = s.leaf_planes + base, *edges = s.leaf_edges + 2 * base;
    // whether a quotient's sign alone puts it out of range
    const bool ahead = t0 >= 0.0f && (Q != kQClosest || fabsf(ray.dx) + fabsf(ray.dy) + fabsf(ray.dz) <= 1e38f);
    int32_t best = -1;
    float best_t = t1;  // the first hit must be below
    for (int k0 = first; k0 < end; k0 += kFewWarps * kFewUnroll) {
        float4 w0[kFewUnroll];
#pragma unroll
        for (int u = 0; u < kFewUnroll; u++) {
            const int k = k0 + kFewWarps * u;
            w0[u] = k < end ? __ldg(planes + k) : make_float4(0.0f, 0.0f, 0.0f, __int_as_float(0x7fc00000));
        }
#pragma unroll
        for (int u = 0; u < kFewUnroll; u++) {
            const int k = k0 + kFewWarps * u;
            const float den = dot3r(w0[u].x, w0[u].y, w0[u].z, ray.dx, ray.dy, ray.dz);
            const float num = rsub(w0[u].w, dot3r(w0[u].x, w0[u].y, w0[u].z, ray.ox, ray.oy, ray.oz));
            // t < 0 where that is out of range, or past the best hit by more
            // than the quotient's rounding
            const bool neg = ((__float_as_uint(num) ^ __float_as_uint(den)) >> 31) != 0u;
            if (neg ? ahead && fabsf(num) > kSureNumerator : fabsf(num) > best_t * fabsf(den) * 1.000001f) continue;
            const float t = rdiv(num, den);
            if (!(t >= t0 && t < t1 && t <= best_t)) continue;
            const float4 w2 = __ldg(edges + 2 * (size_t)k + 1);
            if (__float_as_int(w2.z) == q.skip) continue;
            const float4 w1 = __ldg(edges + 2 * (size_t)k);
            const int drop = (int)(__float_as_uint(w2.w) & 3u);
            const float h0 = radd(pick3(drop, ray.oy, ray.oz, ray.ox), rmul(t, pick3(drop, ray.dy, ray.dz, ray.dx)));
            const float h1 = radd(pick3(drop, ray.oz, ray.ox, ray.oy), rmul(t, pick3(drop, ray.dz, ray.dx, ray.dy)));
            const float b0 = radd(radd(rmul(w1.x, h0), rmul(w1.z, h1)), w2.x);
            const float b1 = radd(radd(rmul(w1.y, h0), rmul(w1.w, h1)), w2.y);
            if (b0 >= 0.0f && b1 >= 0.0f && rsub(rsub(1.0f, b0), b1) >= 0.0f) {
                const int32_t ti = (int32_t)(__float_as_uint(w2.w) >> 2);
                if (t < best_t || best < 0 || ti < best) {
                    best = ti;
                    best_t = t;
                }
            }
        }
    }
    // (t, index) as one number that orders the same (-0 as +0, its sign in the
    // last bit)
    unsigned long long key = kFewNone;
    if (best >= 0) {
        const uint32_t u = __float_as_uint(best_t + 0.0f);
        key = ((unsigned long long)(u ^ ((u >> 31) ? 0xffffffffu : 0x80000000u)) << 32) | ((uint32_t)best << 1) |
              (best_t == 0.0f && signbit(best_t) ? 1u : 0u);
    }
    least[wid][lane] = key;
    __syncthreads();
    if (wid != 0) return;
#pragma unroll
    for (int w = 1; w < kFewWarps; w++) key = min(key, least[w][lane]);
    if (slices > 1) {
        if (i < q.n && key != kFewNone) atomicMin(keys + i, key);
        __threadfence();
        __syncwarp();
        if (lane == 0) last_sh = atomicAdd(done + blockIdx.x, 1u) == (unsigned)slices - 1u;
        __syncwarp();
        if (!last_sh) return;
        __threadfence();
        if (i < q.n) key = atomicExch(keys + i, kFewNone);
        if (lane == 0) done[blockIdx.x] = 0u;
    }
    best = -1;
    best_t = kInf;
    bool occ = false;
    if (key != kFewNone) {
        best = (int32_t)((uint32_t)key >> 1);
        const uint32_t u = (uint32_t)(key >> 32);
        best_t = (key & 1u) ? -0.0f : __uint_as_float(u ^ ((u >> 31) ? 0x80000000u : 0xffffffffu));
        occ = (__ldg(&s.tri_ids[best]) & kTraceIdSky) == 0;
    }
    if (Q == kQMask || Q == kQMaskHit) {
        const unsigned word = __ballot_sync(0xffffffffu, i < q.n && occ);
        if (lane == 0) q.mask[blockIdx.x] = word;
    }
    if (i < q.n) {
        if (Q == kQLines) q.frac[i] = occ ? 0.0f : 1.0f;
        if (Q == kQClosest || Q == kQMaskHit) {
            q.hit[i] = best;
            q.t[i] = best_t;
        }
    }
}

// Whether n rays are few enough against the scene for k_few, at 9 us and 4 us
// more a million tests.  The hierarchy takes 12 us for 33 to 1,000 rays among
// 204 triangles, 23 among 2,064, 37 to 40 among 12,300, 55 to 60 among 49,164.
bool few_rays(const vrg_env *env, int64_t n) {
    const int64_t rays = (n + 31) & ~(int64_t)31, tris = (int64_t)env->bvh_order.size();
    return n <= kFewRays && tris > 0 && rays * tris <= (tris >= 8192 ? 6000000 : 3000000) && env->d_few.ptr;
}

template <Query Q>
cudaError_t launch_few(vrg_env *env, const char *name, const QueryArgs &q) {
    vrg_ctx *ctx = env->ctx;
    const int groups = (int)((q.n + 31) / 32), tris = (int)env->bvh_order.size();
    // enough blocks for the GPU, at least four triangles to a warp
    const int64_t want = ((int64_t)ctx->num_sms * 8 + groups - 1) / groups;
    const int slices = (int)std::max<int64_t>(1, std::min<int64_t>(want, tris / (kFewWarps * kFewUnroll)));
    cudaEvent_t ev = nullptr;
    timing_begin(ctx, name, &ev);
    k_few<Q><<<dim3(groups, slices), 32 * kFewWarps, 0, ctx->stream>>>(
        scene_view(env), q, env->tri_base, tris, slices, env->d_few.as<unsigned long long>(),
        reinterpret_cast<unsigned int *>(env->d_few.as<char>() + kFewKeyBytes));
    const cudaError_t e = cudaGetLastError();
    timing_end(ctx, name, ev);
    return e;
}

// Persistent grid: resident blocks per SM times SMs, but no more blocks
// than the rays can keep busy.
template <class K>
int persistent_grid(const vrg_ctx *ctx, K kernel, int64_t n) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kThreads, 0) != cudaSuccess || per_sm < 1)
        per_sm = 4;
    int64_t blocks = (int64_t)ctx->num_sms * per_sm;
    const int64_t need = (n + kThreads - 1) / kThreads;
    if (blocks > need) blocks = need;
    return (int)(blocks < 1 ? 1 : blocks);
}

// One launch over the lines, the counter of taken lines and (for the mask
// queries) the mask zeroed before it.
template <Query Q, bool ORDER>
cudaError_t launch_query(vrg_env *env, const char *name, QueryArgs q) {
    vrg_ctx *ctx = env->ctx;
    if (few_rays(env, q.n)) return launch_few<Q>(env, name, q);
    const auto kernel = k_bvh<Q, 4, 4, 8, 8, ORDER>;
    cudaError_t e = env->d_work.reserve(256);
    if (e != cudaSuccess) return e;
    q.work = env->d_work.as<unsigned long long>();
    e = cudaMemsetAsync(q.work, 0, 8, ctx->stream);
    if (e == cudaSuccess && q.mask) e = cudaMemsetAsync(q.mask, 0, 4 * (size_t)((q.n + 31) / 32), ctx->stream);
    if (e != cudaSuccess) return e;
    cudaEvent_t ev = nullptr;
    timing_begin(ctx, name, &ev);
    kernel<<<persistent_grid(ctx, kernel, q.n), kThreads, 0, ctx->stream>>>(scene_view(env), bvh_view(env), q);
    e = cudaGetLastError();
    timing_end(ctx, name, ev);
    return e;
}

}  // namespace

DevScene scene_view(const vrg_env *env) {
    DevScene s;
    s.nodes = env->d_nodes.as<uint2>();
    s.leaf_planes = env->d_leaf_tris.as<float4>();
    s.leaf_edges = s.leaf_planes + env->walk_tree.refs.size() + env->n_extra_records;
    s.tri_ids = env->d_tri_ids.as<int32_t>();
    s.top = env->d_top.as<uint2>();
    s.ntop = env->ntop;
    s.g = env->geom;
    return s;
}

BvhView bvh_view(const vrg_env *env) {
    BvhView v{};
    if (env->bvh_nodes) v.nodes = env->d_bvh.as<float4>();
    v.base = env->tri_base;
    return v;
}

int launch_occlusion_mask(vrg_env *env, const float *start, const float *stop, int64_t n,
                          int32_t skip_id, uint32_t *mask, int32_t *hit, float *t) {
    if (n <= 0) return VRG_OK;
    QueryArgs q{};
    q.a = start;
    q.b = stop;
    q.n = n;
    q.skip = skip_id;
    q.mask = mask;
    if (hit && t) {
        q.hit = hit;
        q.t = t;
        VRG_CUDA(env->ctx, (launch_query<kQMaskHit, true>(env, "trace_mask", q)));
    } else {
        VRG_CUDA(env->ctx, (launch_query<kQMask, false>(env, "trace_mask", q)));
    }
    return VRG_OK;
}

int launch_trace_closest(vrg_env *env, const float *orig, const float *dir, const float *tmin,
                         const float *tmax, int64_t n, int32_t skip_id, int32_t *hit, float *t) {
    if (n <= 0) return VRG_OK;
    QueryArgs q{};
    q.a = orig;
    q.b = dir;
    q.tmin = tmin;
    q.tmax = tmax;
    q.n = n;
    q.skip = skip_id;
    q.hit = hit;
    q.t = t;
    VRG_CUDA(env->ctx, (launch_query<kQClosest, true>(env, "trace_closest", q)));
    return VRG_OK;
}

int launch_test_lines(vrg_env *env, const float *start, const float *stop, int64_t n,
                      int32_t skip_id, float *frac) {
    if (n <= 0) return VRG_OK;
    QueryArgs q{};
    q.a = start;
    q.b = stop;
    q.n = n;
    q.skip = skip_id;
    q.frac = frac;
    VRG_CUDA(env->ctx, (launch_query<kQLines, false>(env, "trace_lines", q)));
    return VRG_OK;
}

}  // namespace vrg
