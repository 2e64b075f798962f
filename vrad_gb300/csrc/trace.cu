// trace.cu -- batched ray queries against a resident scene (Trace4Rays,
// raytracer/environment.go:140-145, and TestLineDoesHitSky,
// raytracer/trace/testline.go:18-94).
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
                        rp = box_ray(ray, ray_slack(s.g, ray.ox, ray.oy, ray.oz));
                        active = bv.nodes && t0 <= len;
                    } else {
                        float sx, sy, sz, ex, ey, ez;
                        load3(q.a, ri, sx, sy, sz);
                        load3(q.b, ri, ex, ey, ez);
                        const LinePlan p = plan_line(s, make_line(sx, sy, sz, ex, ey, ez));
                        ray = p.ray;
                        rp = box_ray(ray, p.slack);
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
                       !bvh_pop<MODE>(stk, sp, best_t, cur);
        } else {
#pragma unroll
            for (int u = 0; u < STEPS; u++)
                if (active && !done && !(cur & kBvhLeafBit))
                    if (!bvh_step<ORDER>(bv, rp, t0, fminf(len, best_t), stk, sp, cur)) done = !bvh_pop<MODE>(stk, sp, best_t, cur);
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
