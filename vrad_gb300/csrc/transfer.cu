// transfer.cu -- form-factor transfer lists in CSR.  The reference only
// declares the storage (Transfer{Patch, Transfer}, common/types/transfer.go:3-6;
// Patch.NumTransfers/Transfers, common/types/patch.go:60-61); building them is
// the project's own stage:
//   row i = leaf patch with centre c on face f (normal N, edge U)
//   q = c + N*0.125 ; T1 = U * (1/sqrt(U.U)) ; T2 = N x T1
//   ray r: d = ((lx*T1 + ly*T2) + lz*N) per component, closest hit on
//   [0, MAX_TRACE_LENGTH); a hit on triangle h with tri_face[h] = g >= 0
//   descends g's patch tree at x = q + t*d (coordinate >= dist -> child1)
//   to leaf j.  Row i holds each j once, ascending, with weight hits/k.
#include <algorithm>
#include <cmath>

#include "vrg_internal.h"
#include "vrg_bvh.cuh"
#include "vrg_trace.cuh"

namespace vrg {

namespace {

constexpr int kStageMax = 8192;  // staged entries per row

// Row frame and ray directions shared by both row kernels.
struct RowFrame {
    float qx, qy, qz, t1x, t1y, t1z, t2x, t2y, t2z, nx, ny, nz;
};

__device__ __forceinline__ RowFrame row_frame(const LeafInfo &li, const FaceRec &F) {
    RowFrame fr;
    fr.qx = radd(li.center.x, rmul(F.normal.x, kSampleOffset));
    fr.qy = radd(li.center.y, rmul(F.normal.y, kSampleOffset));
    fr.qz = radd(li.center.z, rmul(F.normal.z, kSampleOffset));
    const float il = rrcp(rsqrt_rn(dot3r(F.u.x, F.u.y, F.u.z, F.u.x, F.u.y, F.u.z)));
    fr.t1x = rmul(F.u.x, il);
    fr.t1y = rmul(F.u.y, il);
    fr.t1z = rmul(F.u.z, il);
    fr.nx = F.normal.x;
    fr.ny = F.normal.y;
    fr.nz = F.normal.z;
    fr.t2x = rsub(rmul(fr.ny, fr.t1z), rmul(fr.nz, fr.t1y));
    fr.t2y = rsub(rmul(fr.nz, fr.t1x), rmul(fr.nx, fr.t1z));
    fr.t2z = rsub(rmul(fr.nx, fr.t1y), rmul(fr.ny, fr.t1x));
    return fr;
}

__device__ __forceinline__ void row_ray(const RowFrame &fr, const float *__restrict__ dirs, int r, float &dx,
                                        float &dy, float &dz) {
    const float lx = __ldg(dirs + 3 * r), ly = __ldg(dirs + 3 * r + 1), lz = __ldg(dirs + 3 * r + 2);
    dx = radd(radd(rmul(lx, fr.t1x), rmul(ly, fr.t2x)), rmul(lz, fr.nx));
    dy = radd(radd(rmul(lx, fr.t1y), rmul(ly, fr.t2y)), rmul(lz, fr.ny));
    dz = radd(radd(rmul(lx, fr.t1z), rmul(ly, fr.t2z)), rmul(lz, fr.nz));
}

// Leaf of the patch tree a hit on triangle h at t lands in (-1: no hit, or no
// lit face).
__device__ __forceinline__ int32_t hit_leaf(const RowFrame &fr, const PatchNode *__restrict__ pnodes,
                                            const int32_t *__restrict__ face_root,
                                            const int32_t *__restrict__ tri_face, int32_t h, float t, float dx,
                                            float dy, float dz) {
    if (h < 0) return -1;
    const int32_t g = __ldg(tri_face + h);
    const int32_t root = g >= 0 ? __ldg(face_root + g) : -1;
    if (root < 0) return -1;
    const float x0 = radd(fr.qx, rmul(t, dx)), x1 = radd(fr.qy, rmul(t, dy)), x2 = radd(fr.qz, rmul(t, dz));
    PatchNode pn = pnodes[root];
    while (pn.axis >= 0) {
        const float xa = pick3(pn.axis, x0, x1, x2);
        pn = pnodes[xa >= pn.dist ? pn.child1 : pn.child2];
    }
    return pn.leaf;
}

// Target leaf of ray r of a row (-1: no lit face hit), walked in the kd tree or
// the line queries' hierarchy.
template <bool BVH>
__device__ __forceinline__ int32_t row_ray_target(const DevScene &s, const BvhView &bv, const RowFrame &fr,
                                                  const PatchNode *__restrict__ pnodes,
                                                  const int32_t *__restrict__ face_root,
                                                  const int32_t *__restrict__ tri_face,
                                                  const float *__restrict__ dirs, int r) {
    float dx, dy, dz, t;
    row_ray(fr, dirs, r, dx, dy, dz);
    const Ray ray{fr.qx, fr.qy, fr.qz, dx, dy, dz};
    const int32_t h = BVH ? bvh_trace<kClosest, kOptSign>(s, bv, ray, ray_slack(s.g, fr.qx, fr.qy, fr.qz), 0.0f,
                                                          kMaxTraceLength, -1, 0.0f, &t)
                          : trace_ray<kClosest, kOptSkip>(s, ray, 0.0f, kMaxTraceLength, -1, &t);
    return hit_leaf(fr, pnodes, face_root, tri_face, h, t, dx, dy, dz);
}

// A row's hits, counted per target leaf: one 32-bit counter per leaf in global
// memory, a block's own and all zero between rows, and a bitmap of the leaves
// hit (in shared memory where it fits, else after the counters).  A row
// touches a few thousand counters in runs of neighbours, so they stay in L2;
// the bitmap in leaf order is the row's columns in ascending order, so nothing
// is sorted.  (A hash table sorted in place instead took 21,000 warp
// instructions a row at k = 1,024 and 116,000 from k = 4,096 on.)
struct RowCounts {
    uint32_t *count;
    uint32_t *bits;
    int words;  // of the bitmap
};
constexpr int kBitmapShared = 8192;  // largest bitmap kept in shared memory, in words (262,144 leaves)

__device__ __forceinline__ void row_add(const RowCounts &rc, int32_t target, uint32_t hits) {
    atomicAdd(rc.count + target, hits);
    const uint32_t bit = 1u << (target & 31);
    uint32_t *word = rc.bits + (target >> 5);
    if (!(*(volatile uint32_t *)word & bit)) atomicOr(word, bit);
}

__device__ __forceinline__ RowCounts row_counts(uint32_t *scratch, int64_t stride, int leaves, uint32_t *shared_bits) {
    RowCounts rc;
    rc.words = (leaves + 31) >> 5;
    rc.count = scratch + (int64_t)blockIdx.x * stride;
    rc.bits = rc.words <= kBitmapShared ? shared_bits : rc.count + 32 * (int64_t)rc.words;
    if (rc.words <= kBitmapShared)
        for (int i = threadIdx.x; i < rc.words; i += blockDim.x) rc.bits[i] = 0u;
    __syncthreads();
    return rc;
}

// The block writes the row's (target, hits) in ascending order of target into
// oc / on when there are at most `limit` of them, clears the counters and the
// bitmap, and returns their number.  Each warp has a run of the bitmap's
// words; `sums` holds a word per warp.
__device__ __forceinline__ int write_row(const RowCounts &rc, int limit, int *sums, int32_t *__restrict__ oc,
                                         int32_t *__restrict__ on) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int run = ((rc.words + nw - 1) / nw + 31) & ~31;
    const int w0 = min(rc.words, wid * run), w1 = min(rc.words, w0 + run);
    __syncthreads();
    int n = 0;
    for (int w = w0 + lane; w < w1; w += 32) n += __popc(((volatile uint32_t *)rc.bits)[w]);
    n = __reduce_add_sync(0xffffffffu, n);
    if (lane == 0) sums[wid] = n;
    __syncthreads();
    int at = 0, total = 0;
    for (int i = 0; i < nw; i++) {
        if (i < wid) at += sums[i];
        total += sums[i];
    }
    const bool keep = total <= limit;
    for (int w = w0; w < w1; w += 32) {
        const uint32_t mine = w + lane < w1 ? ((volatile uint32_t *)rc.bits)[w + lane] : 0u;
        unsigned todo = __ballot_sync(0xffffffffu, mine != 0u);
        if (w + lane < w1 && mine) rc.bits[w + lane] = 0u;
        while (todo) {  // one word at a time, a leaf per lane
            const int l = __ffs(todo) - 1;
            todo &= todo - 1u;
            const uint32_t bits = __shfl_sync(0xffffffffu, mine, l);
            const int32_t leaf = 32 * (w + l) + lane;
            if ((bits >> lane) & 1u) {
                const uint32_t hits = __ldcg(rc.count + leaf);
                rc.count[leaf] = 0u;
                if (keep) {
                    const int p = at + __popc(bits & ((1u << lane) - 1u));
                    oc[p] = leaf;
                    on[p] = (int32_t)hits;
                }
            }
            at += __popc(bits);
        }
    }
    __syncthreads();
    return total;
}

// One block per row: trace the k rays; the lanes of a warp that hit the same
// target add their hits with one update (warp match); the row's (col, count)
// go into the staging arrays at `stride`.  A row past `limit` distinct targets
// writes nnz = -1 and is rebuilt by k_transfer_rows_sorted.  NT threads per
// block at most; k is a multiple of the block size, so every lane of a warp
// runs the same rays.
template <int NT, bool BVH>
__global__ void __launch_bounds__(NT) k_transfer_rows(
    DevScene s, BvhView bv, const LeafInfo *__restrict__ leaves, const FaceRec *__restrict__ faces,
    const PatchNode *__restrict__ pnodes, const int32_t *__restrict__ face_root,
    const int32_t *__restrict__ tri_face, const float *__restrict__ dirs, int k, int64_t row0,
    int64_t rows, int nleaves, int stride, int limit, uint32_t *__restrict__ scratch, int64_t scratch_stride,
    int32_t *__restrict__ stage_col, int32_t *__restrict__ stage_cnt, int32_t *__restrict__ nnz) {
    extern __shared__ __align__(16) uint32_t shared_bits[];
    __shared__ int sums[NT / 32];
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31;
    const RowCounts rc = row_counts(scratch, scratch_stride, nleaves, shared_bits);
    for (int64_t rl = blockIdx.x; rl < rows; rl += gridDim.x) {
        const int64_t row = row0 + rl;
        const LeafInfo li = leaves[row];
        const RowFrame fr = row_frame(li, faces[__float_as_int(li.refl.w)]);
        for (int r = tid; r < k; r += nt) {
            const int32_t target = row_ray_target<BVH>(s, bv, fr, pnodes, face_root, tri_face, dirs, r);
            const unsigned peers = __match_any_sync(0xffffffffu, target);
            if (target >= 0 && lane == __ffs(peers) - 1) row_add(rc, target, (uint32_t)__popc(peers));
        }
        const int total = write_row(rc, limit, sums, stage_col + rl * (int64_t)stride, stage_cnt + rl * (int64_t)stride);
        if (tid == 0) nnz[rl] = total <= limit ? total : -1;
    }
}

// --- rows traced in tiles -------------------------------------------------
//
// A row's rays share their origin, so a tile of 64 or 128 neighbouring
// directions is a thin cone, and what the cone can hit is found once for the
// tile: clusters of neighbouring triangles, nearest first, by their bounding
// sphere, then the triangles by theirs, then by the three edge planes through
// the origin, for each of the tile's bundles of 32 rays.  A bundle's
// rays ask three plane signs (nine multiply-adds) per triangle left and run
// the exact test only inside.  Nearest first, and until the rest lies behind
// the hits: of the 8,208 triangles of the 4,096-face room a tile readies 47,
// 9 may touch it and 7 are taken up, and a bundle runs 2.4 exact tests.  All
// culls are conservative: a triangle the exact test could accept on a ray of
// the tile passes within `reach` of the ray (twice the walk's slab bound), and
// spheres, planes and distances are widened by it.

constexpr float kInfHost = __builtin_huge_valf();
constexpr int kTileBundles = 4;            // bundles of 32 rays to a tile (one ray of each per lane), at most
constexpr int kClusterMax = 1024;          // clusters
constexpr int kClusterMin = 16;            // triangles to a cluster: this times a power of two
constexpr int kDistBins = 64;

// A triangle as the tiles read it: vertices and leaf record.
struct alignas(16) TileTri {
    float v[9];
    int32_t rec;
    int32_t pad[2];
};

struct TileScene {
    const float4 *clusters;  // bounding spheres of `per` neighbouring triangles
    const float4 *spheres;   // per triangle: centre, radius; all spheres are widened by reach
    const TileTri *tris;
    const float4 *cones;     // per node of the heap over bundles of 32 (1: all): axis, cosine of the half angle
    const float2 *spread;    //   sine of the half angle, largest distance of a direction from the axis
    int ntris, nclusters, per, ntiles;  // tiles of a row (the kernel's number of bundles to each)
    int upper;  // no direction leaves below the face's plane
    float reach, plane_eps, bin_scale;
};

// The clusters as a row's origin sees them, in order of their distance's bin.
struct RowClusters {
    float4 *dir;    // unit direction to the centre, least distance
    float2 *angle;  // cosine and sine of the sphere's angular radius
    int32_t *id;
};

struct TileBound {
    float ux, uy, uz, lo, cb, sb;
};

__device__ __forceinline__ TileBound tile_bound(const float4 sp, const RowFrame &fr) {
    TileBound b;
    const float vx = sp.x - fr.qx, vy = sp.y - fr.qy, vz = sp.z - fr.qz;
    const float d2 = __fmaf_rn(vx, vx, __fmaf_rn(vy, vy, vz * vz));
    const float inv = rsqrtf(fmaxf(d2, 1e-20f));
    const float dist = d2 * inv;
    b.ux = vx * inv;
    b.uy = vy * inv;
    b.uz = vz * inv;
    b.lo = fmaxf(0.0f, (dist - sp.w) * 0.9999f);
    b.sb = sp.w * inv;
    // an origin inside (or nearly) sees the sphere everywhere
    if (b.sb < 0.9999f) {
        b.cb = sqrtf(fmaxf(0.0f, __fmaf_rn(-b.sb, b.sb, 1.0f)));
    } else {
        b.cb = -4.0f;
        b.sb = 0.0f;
    }
    return b;
}

__device__ __forceinline__ float rsqrt_fast(float v) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}

// The same for a sphere given by centre and radius, without its angle: the
// distance of the centre from the line along the cone's side is at most the
// radius (in front of the apex the distance from the cone, behind it less).
// d2: squared distance of the centre from the origin.
__device__ __forceinline__ bool cone_meets(const float4 sp, const RowFrame &fr, float3 axis, float ca, float sa,
                                           float &d2) {
    const float vx = sp.x - fr.qx, vy = sp.y - fr.qy, vz = sp.z - fr.qz;
    d2 = __fmaf_rn(vx, vx, __fmaf_rn(vy, vy, vz * vz));
    const float a = __fmaf_rn(vx, axis.x, __fmaf_rn(vy, axis.y, vz * axis.z));
    const float h = __fmaf_rn(a, sa, sp.w);  // (distance from the axis) * ca must not be more
    const float p2 = __fmaf_rn(-a, a, d2) * ca * ca;
    // 8e-6 d2: the rounding of both sides
    return ca < 0.5f || (h >= 0.0f && p2 <= __fmaf_rn(h, h, 8e-6f * d2));
}

// Whether a cone touches a sphere: the angle between them is at most the sum
// of the half angles (a cone wider than 60 degrees touches everything).
__device__ __forceinline__ bool cone_touches(float ux, float uy, float uz, float cb, float sb, float3 axis, float ca,
                                             float sa) {
    if (ca < 0.5f) return true;
    return __fmaf_rn(ux, axis.x, __fmaf_rn(uy, axis.y, uz * axis.z)) >= __fmaf_rn(ca, cb, -sa * sb) - 2e-5f;
}

__device__ __forceinline__ float3 to_world(const RowFrame &fr, const float4 c) {
    return make_float3(__fmaf_rn(c.x, fr.t1x, __fmaf_rn(c.y, fr.t2x, c.z * fr.nx)),
                       __fmaf_rn(c.x, fr.t1y, __fmaf_rn(c.y, fr.t2y, c.z * fr.ny)),
                       __fmaf_rn(c.x, fr.t1z, __fmaf_rn(c.y, fr.t2z, c.z * fr.nz)));
}

// The block puts the clusters in order for a row; returns their number.
__device__ __forceinline__ int row_clusters(const TileScene &ts, const RowFrame &fr, const RowClusters &rcl, int *bins) {
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, wid = tid >> 5;
    for (int i = tid; i < kDistBins; i += nt) bins[i] = 0;
    __syncthreads();
    auto bin_of = [&](int c, TileBound &b) {
        b = tile_bound(__ldg(ts.clusters + c), fr);
        // wholly below the face's plane, past what the frame's rounding tilts it
        const float up = __fmaf_rn(b.ux, fr.nx, __fmaf_rn(b.uy, fr.ny, b.uz * fr.nz));
        if (ts.upper && b.cb > 0.0f && up < -b.sb - 1e-3f) return -1;
        return min(kDistBins - 1, (int)(b.lo * ts.bin_scale));
    };
    TileBound b;
    for (int c = tid; c < ts.nclusters; c += nt) {
        const int bin = bin_of(c, b);
        if (bin >= 0) atomicAdd(bins + bin, 1);
    }
    __syncthreads();
    int n = 0;
    for (int i = 0; i < kDistBins; i++) n += bins[i];
    __syncthreads();
    if (wid == 0) {  // bin starts
        const int x = bins[2 * lane], y = bins[2 * lane + 1];
        int incl = x + y;
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        bins[2 * lane] = incl - x - y;
        bins[2 * lane + 1] = incl - y;
    }
    __syncthreads();
    for (int c = tid; c < ts.nclusters; c += nt) {
        const int bin = bin_of(c, b);
        if (bin < 0) continue;
        const int at = atomicAdd(bins + bin, 1);
        rcl.id[at] = c;
        rcl.dir[at] = make_float4(b.ux, b.uy, b.uz, b.lo);
        rcl.angle[at] = make_float2(b.cb, b.sb);
    }
    __syncthreads();
    return n;
}

// One warp, one tile: the closest hits of its rays, LR per lane.
// queue and queue_lo hold 64 entries of the warp's, bundle its LR axes.
template <int LR>
__device__ __forceinline__ void trace_tile(const DevScene &s, const TileScene &ts, const RowFrame &fr, int tile,
                                           const RowClusters &rcl, int n, int32_t *queue, float *queue_lo, float4 *bundle,
                                           const float (&dx)[LR], const float (&dy)[LR],
                                           const float (&dz)[LR], int32_t (&best)[LR],
                                           float (&best_t)[LR]) {
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    const float4 cone = __ldg(ts.cones + ts.ntiles + tile);
    const float2 sp = __ldg(ts.spread + ts.ntiles + tile);
    const float3 axis = to_world(fr, cone);
    const float chord = sp.y;
    if (lane < LR) {  // the bundles' axes and spreads
        const int node = LR * (ts.ntiles + tile) + lane;
        const float3 a = to_world(fr, __ldg(ts.cones + node));
        bundle[lane] = make_float4(a.x, a.y, a.z, __ldg(ts.spread + node).y);
    }
    float bfar[LR];  // largest best_t of each bundle's rays
#pragma unroll
    for (int r = 0; r < LR; r++) bfar[r] = kInf;
    float far = kInf;  // and of the tile's
    int queued = 0, c0 = 0, base = 0, pos = 0;
    unsigned open = 0u;  // clusters base + bit still to go through, the first from triangle pos on
    for (;;) {
        // triangles whose spheres touch the cone, until 32 are found
        while (queued < 32) {
            if (!open) {
                if (c0 >= n) break;
                bool in = false;
                float lo = kInf;
                if (c0 + lane < n) {
                    const float4 d = rcl.dir[c0 + lane];
                    const float2 a = rcl.angle[c0 + lane];
                    lo = d.w;
                    in = lo <= far && cone_touches(d.x, d.y, d.z, a.x, a.y, axis, cone.w, sp.x);
                }
                open = __ballot_sync(0xffffffffu, in);
                // the clusters are in order of distance bins: past the rays'
                // hits when the first one's bin is
                const int first = min(kDistBins - 1, (int)(__shfl_sync(0xffffffffu, lo, 0) * ts.bin_scale));
                if ((float)first * 0.999f > far * ts.bin_scale) {
                    open = 0u;
                    c0 = n;
                    break;
                }
                base = c0;
                c0 += 32;
                continue;
            }
            // the next 32 triangles: of one cluster, or of two of 16
            const int l0 = __ffs(open) - 1;
            int id = rcl.id[base + l0], t;
            if (ts.per == 16) {
                open &= open - 1u;
                const int l1 = __ffs(open) - 1;
                open &= open - 1u;
                if (lane >= 16) id = l1 >= 0 ? rcl.id[base + l1] : -1;
                t = id < 0 ? ts.ntris : id * 16 + (lane & 15);
            } else {
                t = id * ts.per + pos + lane;
                pos += 32;
                if (pos >= ts.per) {
                    pos = 0;
                    open &= open - 1u;
                }
            }
            bool in = false;
            float lo = 0.0f;
            if (t < ts.ntris) {
                const float4 ball = __ldg(ts.spheres + t);
                float d2;
                in = cone_meets(ball, fr, axis, cone.w, sp.x, d2);
                lo = fmaxf(0.0f, __fmaf_rn(d2, rsqrt_fast(fmaxf(d2, 1e-20f)), -ball.w) * 0.9999f);
                in = in && lo <= far;
            }
            const unsigned m = __ballot_sync(0xffffffffu, in);
            if (in) {
                queue[queued + __popc(m & below)] = t;
                queue_lo[queued + __popc(m & below)] = lo;
            }
            queued += __popc(m);
        }
        if (queued == 0) break;
        __syncwarp();
        const int take = min(queued, 32);
        // a lane readies one queued triangle: its edge planes seen from the
        // origin, inner side positive, and how far a ray may lie outside
        bool keep = lane < take;
        float mx[3], my[3], mz[3], eps[3], near = 0.0f;
        int32_t rec = 0;
        unsigned bundles = 0u;  // that the triangle may touch
        if (keep) {
            const TileTri t = ts.tris[queue[lane]];
            rec = t.rec;
            const float4 pl = __ldg(s.leaf_planes + rec);
            const float num = pl.w - __fmaf_rn(pl.x, fr.qx, __fmaf_rn(pl.y, fr.qy, pl.z * fr.qz));
            const float nc = __fmaf_rn(pl.x, axis.x, __fmaf_rn(pl.y, axis.y, pl.z * axis.z));
            const bool sided = fabsf(num) > ts.plane_eps;
            // the plane lies behind every ray of the cone
            if (sided && num * nc < 0.0f && fabsf(nc) > chord + 1e-5f) keep = false;
            near = fmaxf(queue_lo[lane], (fabsf(num) - ts.reach) / (fabsf(nc) + chord + 1e-5f)) * 0.999f;
            if (near > far) keep = false;
            const float wide = near > 2.0f * ts.reach ? ts.reach / (near - ts.reach) + 2e-6f : 4.0f;
            const float side = num < 0.0f ? -1.0f : 1.0f;
            float ax[3], ay[3], az[3], a2[3];
#pragma unroll
            for (int e = 0; e < 3; e++) {
                ax[e] = t.v[3 * e] - fr.qx;
                ay[e] = t.v[3 * e + 1] - fr.qy;
                az[e] = t.v[3 * e + 2] - fr.qz;
                a2[e] = __fmaf_rn(ax[e], ax[e], __fmaf_rn(ay[e], ay[e], az[e] * az[e]));
            }
#pragma unroll
            for (int e = 0; e < 3; e++) {
                const int f = e == 2 ? 0 : e + 1;
                const float cx = ay[e] * az[f] - az[e] * ay[f], cy = az[e] * ax[f] - ax[e] * az[f],
                            cz = ax[e] * ay[f] - ay[e] * ax[f];
                const float l2 = __fmaf_rn(cx, cx, __fmaf_rn(cy, cy, cz * cz));
                const float inv = rsqrt_fast(fmaxf(l2, 1e-30f));
                mx[e] = cx * inv * side;
                my[e] = cy * inv * side;
                mz[e] = cz * inv * side;
                // the cross product's rounding, as an angle
                eps[e] = sided ? __fmaf_rn(1e-6f * fmaxf(a2[e], a2[f]), inv, wide) : 4.0f;
            }
            float most = -1.0f;
#pragma unroll
            for (int r = 0; r < LR; r++) {
                const float4 ba = bundle[r];
                float in = 1.0f;
#pragma unroll
                for (int e = 0; e < 3; e++)
                    in = fminf(in, __fmaf_rn(mx[e], ba.x, __fmaf_rn(my[e], ba.y, __fmaf_rn(mz[e], ba.z, eps[e]))));
                in += ba.w;
                if (in >= 0.0f) bundles |= 1u << r;
                most = fmaxf(most, in);
            }
            // (not bundles != 0: of two bundles, ptxas 13.0 from -O1 on took that as
            // != 3.  In a 72-triangle room the tiles of 64 then took up 1,127 triangles
            // that touched neither bundle and none that touched both, of 13,238; at
            // -O0 the same source is right)
            keep = keep && most >= 0.0f;
        }
        __syncwarp();
        // the rest of the queue moves up
        if (queued > 32) {
            int32_t q = 0;
            float ql = 0.0f;
            if (lane < queued - 32) {
                q = queue[32 + lane];
                ql = queue_lo[32 + lane];
            }
            __syncwarp();
            if (lane < queued - 32) {
                queue[lane] = q;
                queue_lo[lane] = ql;
            }
        }
        queued -= take;
        // nearest first, until what is left lies behind every ray's hit
        for (;;) {
            const uint32_t key = keep ? __float_as_uint(near) : 0xffffffffu;
            const uint32_t least = __reduce_min_sync(0xffffffffu, key);
            if (least == 0xffffffffu || __uint_as_float(least) > far) break;
            const int l = __ffs(__ballot_sync(0xffffffffu, key == least)) - 1;
            if (lane == l) keep = false;
            unsigned todo = __shfl_sync(0xffffffffu, bundles, l);
#pragma unroll
            for (int r = 0; r < LR; r++)
                if (__uint_as_float(least) > bfar[r]) todo &= ~(1u << r);
            if (!todo) continue;
            float m0[3], m1[3], m2[3], e[3];
#pragma unroll
            for (int i = 0; i < 3; i++) {
                m0[i] = __shfl_sync(0xffffffffu, mx[i], l);
                m1[i] = __shfl_sync(0xffffffffu, my[i], l);
                m2[i] = __shfl_sync(0xffffffffu, mz[i], l);
                e[i] = __shfl_sync(0xffffffffu, eps[i], l);
            }
            const int32_t k = __shfl_sync(0xffffffffu, rec, l);
            // the exact test's part that the rays share: same origin, same plane
            const float4 w0 = __ldg(s.leaf_planes + k), w1 = __ldg(s.leaf_edges + 2 * (size_t)k),
                         w2 = __ldg(s.leaf_edges + 2 * (size_t)k + 1);
            const float num = rsub(w0.w, dot3r(w0.x, w0.y, w0.z, fr.qx, fr.qy, fr.qz));
            const uint32_t idx_drop = __float_as_uint(w2.w);
            const int drop = (int)(idx_drop & 3u);
            const float o0 = pick3(drop, fr.qy, fr.qz, fr.qx), o1 = pick3(drop, fr.qz, fr.qx, fr.qy);
#pragma unroll
            for (int r = 0; r < LR; r++) {
                if (!((todo >> r) & 1u)) continue;
                float in = 1.0f;
#pragma unroll
                for (int i = 0; i < 3; i++)
                    in = fminf(in, __fmaf_rn(m0[i], dx[r], __fmaf_rn(m1[i], dy[r], __fmaf_rn(m2[i], dz[r], e[i]))));
                if (!__any_sync(0xffffffffu, in >= 0.0f)) continue;
                if (in >= 0.0f) {  // tri_test<kClosest> (the tiles hold no triangle with the skip id)
                    const float t = rdiv(num, dot3r(w0.x, w0.y, w0.z, dx[r], dy[r], dz[r]));
                    if (t >= 0.0f && t < kMaxTraceLength && t <= best_t[r]) {
                        const float d0 = pick3(drop, dy[r], dz[r], dx[r]), d1 = pick3(drop, dz[r], dx[r], dy[r]);
                        const float h0 = radd(o0, rmul(t, d0)), h1 = radd(o1, rmul(t, d1));
                        const float b0 = radd(radd(rmul(w1.x, h0), rmul(w1.z, h1)), w2.x);
                        const float b1 = radd(radd(rmul(w1.y, h0), rmul(w1.w, h1)), w2.y);
                        const int32_t ti = (int32_t)(idx_drop >> 2);
                        if (b0 >= 0.0f && b1 >= 0.0f && rsub(rsub(1.0f, b0), b1) >= 0.0f && (t < best_t[r] || ti < best[r])) {
                            best[r] = ti;
                            best_t[r] = t;
                        }
                    }
                }
                __syncwarp();
                // (as numbers that order the same: a hit at -0 counts as +0)
                bfar[r] = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(radd(best_t[r], 0.0f))));
            }
            far = bfar[0];
#pragma unroll
            for (int r = 1; r < LR; r++) far = fmaxf(far, bfar[r]);
        }
        __syncwarp();
    }
}

// hit_leaf of a lane's rays, their descents side by side.
template <int LR>
__device__ __forceinline__ void hit_leaves(const RowFrame &fr, const PatchNode *__restrict__ pnodes,
                                           const int32_t *__restrict__ face_root,
                                           const int32_t *__restrict__ tri_face, const int32_t (&h)[LR],
                                           const float (&t)[LR], const float (&dx)[LR],
                                           const float (&dy)[LR], const float (&dz)[LR],
                                           int32_t (&leaf)[LR]) {
    int32_t node[LR];
#pragma unroll
    for (int r = 0; r < LR; r++) node[r] = h[r] >= 0 ? __ldg(tri_face + h[r]) : -1;
#pragma unroll
    for (int r = 0; r < LR; r++) {
        node[r] = node[r] >= 0 ? __ldg(face_root + node[r]) : -1;
        leaf[r] = -1;
    }
    bool more = true;
    while (more) {
        more = false;
        int4 pn[LR];
#pragma unroll
        for (int r = 0; r < LR; r++)
            pn[r] = node[r] >= 0 ? __ldg(reinterpret_cast<const int4 *>(pnodes + node[r])) : make_int4(0, 0, -1, -1);
#pragma unroll
        for (int r = 0; r < LR; r++) {
            if (node[r] < 0) continue;
            if (pn[r].z < 0) {
                leaf[r] = pn[r].w;
                node[r] = -1;
                continue;
            }
            const float o = pick3(pn[r].z, fr.qx, fr.qy, fr.qz), d = pick3(pn[r].z, dx[r], dy[r], dz[r]);
            node[r] = radd(o, rmul(t[r], d)) >= __int_as_float(pn[r].w) ? pn[r].x : pn[r].y;
            more = true;
        }
    }
}
static_assert(sizeof(PatchNode) == 16, "a patch node is read as four words");

// One block per row, its rays in tiles, which the warps take one at a time;
// hits are counted as in k_transfer_rows.
template <int LR, int NT>
__global__ void __launch_bounds__(NT, 1024 / NT) k_transfer_tiles(
    DevScene s, TileScene ts, const LeafInfo *__restrict__ leaves, const FaceRec *__restrict__ faces,
    const PatchNode *__restrict__ pnodes, const int32_t *__restrict__ face_root,
    const int32_t *__restrict__ tri_face, const float *__restrict__ dirs, int64_t row0, int64_t rows, int nleaves,
    int stride, int limit, uint32_t *__restrict__ scratch, int64_t scratch_stride, int32_t *__restrict__ stage_col,
    int32_t *__restrict__ stage_cnt, int32_t *__restrict__ nnz) {
    extern __shared__ __align__(16) uint32_t shared_bits[];
    __shared__ int32_t queues[NT / 32][64];
    __shared__ float queues_lo[NT / 32][64];
    __shared__ float4 bundles[NT / 32][LR];
    __shared__ int bins[kDistBins], sums[NT / 32];
    __shared__ int next_sh;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    RowClusters rcl;  // [clusters | bitmap]
    rcl.dir = reinterpret_cast<float4 *>(shared_bits);
    rcl.angle = reinterpret_cast<float2 *>(rcl.dir + ts.nclusters);
    rcl.id = reinterpret_cast<int32_t *>(rcl.angle + ts.nclusters);
    const RowCounts rc =
        row_counts(scratch, scratch_stride, nleaves, reinterpret_cast<uint32_t *>(rcl.id + ts.nclusters));
    for (int64_t rl = blockIdx.x; rl < rows; rl += gridDim.x) {
        const LeafInfo li = leaves[row0 + rl];
        const RowFrame fr = row_frame(li, faces[__float_as_int(li.refl.w)]);
        if (tid == 0) next_sh = 0;
        const int n = row_clusters(ts, fr, rcl, bins);
        for (;;) {
            int tile = 0;
            if (lane == 0) tile = atomicAdd(&next_sh, 1);
            tile = __shfl_sync(0xffffffffu, tile, 0);
            if (tile >= ts.ntiles) break;
            float dx[LR], dy[LR], dz[LR], best_t[LR];
            int32_t best[LR];
#pragma unroll
            for (int r = 0; r < LR; r++) {
                row_ray(fr, dirs, 32 * (LR * tile + r) + lane, dx[r], dy[r], dz[r]);
                best[r] = -1;
                best_t[r] = kInf;
            }
            trace_tile<LR>(s, ts, fr, tile, rcl, n, queues[wid], queues_lo[wid], bundles[wid], dx, dy, dz, best, best_t);
            int32_t target[LR];
            hit_leaves<LR>(fr, pnodes, face_root, tri_face, best, best_t, dx, dy, dz, target);
#pragma unroll
            for (int r = 0; r < LR; r++) {
                const unsigned peers = __match_any_sync(0xffffffffu, target[r]);
                if (target[r] >= 0 && lane == __ffs(peers) - 1) row_add(rc, target[r], (uint32_t)__popc(peers));
            }
        }
        const int total = write_row(rc, limit, sums, stage_col + rl * (int64_t)stride, stage_cnt + rl * (int64_t)stride);
        if (tid == 0) nnz[rl] = total <= limit ? total : -1;
    }
}

// Rows that overflowed: one block per listed row, its k targets
// sorted (bitonic) in a global scratch of 2k int32 per block, then a block
// scan finds the runs.  Without row_ptr it writes each listed row's nnz;
// with row_ptr it writes the row's (col, hits / k) straight into the CSR at
// row_ptr[row].  NT threads per block at most; k is a power of two and a
// multiple of the block size.
template <int NT>
__global__ void __launch_bounds__(NT) k_transfer_rows_sorted(
    DevScene s, BvhView bv, const LeafInfo *__restrict__ leaves, const FaceRec *__restrict__ faces,
    const PatchNode *__restrict__ pnodes, const int32_t *__restrict__ face_root,
    const int32_t *__restrict__ tri_face, const float *__restrict__ dirs, int k,
    const int64_t *__restrict__ row_list, int64_t nlist, int32_t *__restrict__ scratch,
    const int64_t *__restrict__ row_ptr, int32_t *__restrict__ col, float *__restrict__ w,
    int32_t *__restrict__ nnz) {
    __shared__ int32_t warp_sums[NT / 32];
    __shared__ int32_t total_sh;
    const int tid = threadIdx.x, nt = blockDim.x;
    int32_t *tg = scratch + (int64_t)blockIdx.x * 2 * k;
    int32_t *starts = tg + k;
    for (int64_t j = blockIdx.x; j < nlist; j += gridDim.x) {
        const int64_t row = row_list[j];
        const LeafInfo li = leaves[row];
        const RowFrame fr = row_frame(li, faces[__float_as_int(li.refl.w)]);
        for (int r = tid; r < k; r += nt) tg[r] = row_ray_target<true>(s, bv, fr, pnodes, face_root, tri_face, dirs, r);
        __syncthreads();
        for (int size = 2; size <= k; size <<= 1) {
            for (int stride = size >> 1; stride > 0; stride >>= 1) {
                for (int i = tid; i < (k >> 1); i += nt) {
                    const int lo = 2 * i - (i & (stride - 1));
                    const int hi = lo + stride;
                    const bool asc = (lo & size) == 0;
                    const int32_t a = tg[lo], b = tg[hi];
                    if ((a > b) == asc) {
                        tg[lo] = b;
                        tg[hi] = a;
                    }
                }
                __syncthreads();
            }
        }
        // run starts of valid targets; each thread owns a contiguous segment
        const int per = k / nt;
        const int seg = tid * per;
        int cnt = 0;
        for (int i = seg; i < seg + per; i++) cnt += (tg[i] >= 0 && (i == 0 || tg[i] != tg[i - 1])) ? 1 : 0;
        int incl = cnt;
        const int lane = tid & 31, wid = tid >> 5;
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        if (lane == 31) warp_sums[wid] = incl;
        __syncthreads();
        if (wid == 0) {
            const int w = lane < (nt >> 5) ? warp_sums[lane] : 0;
            int wi = w;
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, wi, o);
                if (lane >= o) wi += v;
            }
            if (lane < (nt >> 5)) warp_sums[lane] = wi - w;
            if (lane == (nt >> 5) - 1) total_sh = wi;
        }
        __syncthreads();
        int pos = warp_sums[wid] + incl - cnt;
        for (int i = seg; i < seg + per; i++)
            if (tg[i] >= 0 && (i == 0 || tg[i] != tg[i - 1])) starts[pos++] = i;
        __syncthreads();
        const int total = total_sh;
        if (row_ptr) {
            const int64_t b = row_ptr[row];
            const float fk = (float)k;
            for (int p = tid; p < total; p += nt) {
                const int st = starts[p];
                const int en = p + 1 < total ? starts[p + 1] : k;
                col[b + p] = tg[st];
                w[b + p] = __fdiv_rn((float)(en - st), fk);
            }
        } else if (tid == 0) {
            nnz[j] = total;
        }
        __syncthreads();
    }
}

// One warp per row: staged (col, count) at stride `tstride` -> final CSR
// (col, count / k).  Rows with nnz_chunk < 0 overflowed and are
// written by k_transfer_rows_sorted instead.
__global__ void k_transfer_gather(const int32_t *__restrict__ stage_col,
                                  const int32_t *__restrict__ stage_cnt, int tstride,
                                  const int32_t *__restrict__ nnz_chunk,
                                  const int64_t *__restrict__ row_ptr, int64_t row0, int64_t rows,
                                  int k, int32_t *__restrict__ col, float *__restrict__ w) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const float fk = (float)k;
    for (int64_t rl = warp; rl < rows; rl += nwarps) {
        if (nnz_chunk[rl] < 0) continue;
        const int64_t b = row_ptr[row0 + rl], e = row_ptr[row0 + rl + 1];
        const int32_t *sc = stage_col + rl * (int64_t)tstride;
        const int32_t *sn = stage_cnt + rl * (int64_t)tstride;
        for (int64_t i = lane; i < e - b; i += 32) {
            col[b + i] = sc[i];
            w[b + i] = __fdiv_rn((float)sn[i], fk);
        }
    }
}

int grow(vrg_ctx *ctx, DevBuf &buf, size_t need, size_t keep) {
    if (need <= buf.bytes && buf.ptr) return VRG_OK;
    size_t cap = std::max(need, buf.bytes + buf.bytes / 2);
    void *p = nullptr;
    VRG_CUDA(ctx, cudaMalloc(&p, cap));
    if (keep) VRG_CUDA(ctx, cudaMemcpyAsync(p, buf.ptr, keep, cudaMemcpyDeviceToDevice, ctx->stream));
    VRG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    buf.release();
    buf.ptr = p;
    buf.bytes = cap;
    return VRG_OK;
}

}  // namespace

namespace {

// The rays of a row go out in table order, 32 to a warp, 64 or
// 128 to a tile.  A row's CSR does not depend on that order (hits are counted per
// target), so the table is halved at the median of its widest axis down to
// runs of 32: every aligned power-of-two run is then a compact bundle of
// neighbouring directions, which walk much the same nodes and whose cone is
// thin (a tile of 128 of 65,536 cosine-weighted directions: 4.6 degrees of
// half angle on average; runs of a Morton order jump at arbitrary places, 9.9
// on average and up to 157).  A table with a non-finite entry keeps its order.
void order_directions(const float *d, int32_t k, std::vector<float> &out) {
    std::vector<int32_t> idx(k);
    bool finite = true;
    for (int32_t r = 0; r < k; r++) {
        idx[r] = r;
        for (int c = 0; c < 3; c++) finite = finite && std::isfinite(d[3 * r + c]);
    }
    std::vector<std::pair<int32_t, int32_t>> todo;  // runs still to halve
    if (finite && k > 32) todo.push_back({0, k});
    while (!todo.empty()) {
        const std::pair<int32_t, int32_t> run = todo.back();
        todo.pop_back();
        float lo[3] = {kInfHost, kInfHost, kInfHost}, hi[3] = {-kInfHost, -kInfHost, -kInfHost};
        for (int32_t i = run.first; i < run.second; i++)
            for (int c = 0; c < 3; c++) {
                lo[c] = std::min(lo[c], d[3 * idx[i] + c]);
                hi[c] = std::max(hi[c], d[3 * idx[i] + c]);
            }
        int ax = 0;
        for (int c = 1; c < 3; c++)
            if (hi[c] - lo[c] > hi[ax] - lo[ax]) ax = c;
        const int32_t mid = (run.first + run.second) / 2;
        std::nth_element(idx.begin() + run.first, idx.begin() + mid, idx.begin() + run.second,
                         [d, ax](int32_t a, int32_t b) {
                             const float x = d[3 * a + ax], y = d[3 * b + ax];
                             return x < y || (x == y && a < b);
                         });
        if (mid - run.first > 32) {
            todo.push_back({run.first, mid});
            todo.push_back({mid, run.second});
        }
    }
    out.resize(3 * (size_t)k);
    for (int32_t r = 0; r < k; r++)
        for (int c = 0; c < 3; c++) out[3 * r + c] = d[3 * idx[r] + c];
}

// What k_transfer_tiles reads: the scene's triangles in clusters with
// their spheres (kept with the scene: its geometry does not change) and the
// cones over the direction table (ray order as traced).  `tiles` says whether
// the tiles' margins hold: unit directions, orthonormal row frames, origins
// within the scene's coordinates.
int prepare_tiles(vrg_env *env, const std::vector<float> &dirs, int32_t k, TileScene &ts, std::vector<float4> &cones,
                  std::vector<float2> &spread, bool &tiles) {
    vrg_ctx *ctx = env->ctx;
    cudaStream_t st = ctx->stream;
    const int64_t nt = env->geom.ntris;
    tiles = false;
    if (k < 32 * kTileBundles || nt < 1 || nt > 262144 || !env->faces_inside || !(env->geom.scale <= 16000.0f)) return VRG_OK;
    for (int32_t r = 0; r < k; r++) {
        const double x = dirs[3 * r], y = dirs[3 * r + 1], z = dirs[3 * r + 2];
        if (!(std::fabs(x * x + y * y + z * z - 1.0) <= 1e-4)) return VRG_OK;
    }
    for (int32_t f = 0; f < env->nfaces; f++) {
        const float *u = &env->f_u[3 * f], *n = &env->f_normal[3 * f];
        const double uu = (double)u[0] * u[0] + (double)u[1] * u[1] + (double)u[2] * u[2];
        const double nn = (double)n[0] * n[0] + (double)n[1] * n[1] + (double)n[2] * n[2];
        const double un = (double)u[0] * n[0] + (double)u[1] * n[1] + (double)u[2] * n[2];
        if (!(std::fabs(nn - 1.0) <= 1e-4 && uu > 1e-12 && un * un <= 1e-8 * uu)) return VRG_OK;
    }
    const double reach = std::ldexp(2.0 * (2.01 * (double)env->geom.scale + 3.0), -17);
    if (env->tile_tris < 0) {
        const std::vector<int32_t> &refs = env->walk_tree.refs;
        std::vector<int32_t> rec(nt, -1);
        for (size_t r = 0; r < refs.size(); r++)
            if (env->ids[refs[r]] != -1) rec[refs[r]] = (int32_t)r;  // -1: the rays' skip id
        std::vector<int32_t> order;
        for (int64_t t = 0; t < nt; t++) {
            bool finite = rec[t] >= 0;  // a triangle with a non-finite corner is never hit
            for (int c = 0; c < 9; c++) finite = finite && std::isfinite(env->xyz[9 * t + c]);
            if (finite) order.push_back((int32_t)t);
        }
        const size_t n = order.size();
        size_t per = kClusterMin;
        while ((n + per - 1) / per > kClusterMax) per *= 2;
        const size_t nc = (n + per - 1) / per;
        // clusters: runs of the triangles halved near the median of their
        // centres' widest axis, at a whole number of clusters
        std::vector<std::pair<size_t, size_t>> todo;
        if (n > per) todo.push_back({0, n});
        while (!todo.empty()) {
            const std::pair<size_t, size_t> run = todo.back();
            todo.pop_back();
            auto centre = [&](int32_t t, int a) {
                const float *v = &env->xyz[9 * (size_t)t];
                return (v[a] + v[3 + a]) + v[6 + a];
            };
            float lo[3] = {kInfHost, kInfHost, kInfHost}, hi[3] = {-kInfHost, -kInfHost, -kInfHost};
            for (size_t i = run.first; i < run.second; i++)
                for (int a = 0; a < 3; a++) {
                    lo[a] = std::min(lo[a], centre(order[i], a));
                    hi[a] = std::max(hi[a], centre(order[i], a));
                }
            int ax = 0;
            for (int a = 1; a < 3; a++)
                if (hi[a] - lo[a] > hi[ax] - lo[ax]) ax = a;
            const size_t whole = (run.second - run.first + per - 1) / per;
            const size_t mid = run.first + (whole / 2) * per;
            std::nth_element(order.begin() + run.first, order.begin() + mid, order.begin() + run.second,
                             [&](int32_t x, int32_t y) {
                                 const float cx = centre(x, ax), cy = centre(y, ax);
                                 return cx < cy || (cx == cy && x < y);
                             });
            if (mid - run.first > per) todo.push_back({run.first, mid});
            if (run.second - mid > per) todo.push_back({mid, run.second});
        }
        // ball around the box of `count` vertices, widened by reach
        auto ball = [&](const std::vector<const float *> &vs) {
            double mn[3], mx[3], r2 = 0.0;
            for (int a = 0; a < 3; a++) mn[a] = mx[a] = vs[0][a];
            for (const float *v : vs)
                for (int a = 0; a < 3; a++) {
                    mn[a] = std::min(mn[a], (double)v[a]);
                    mx[a] = std::max(mx[a], (double)v[a]);
                }
            float c[3];
            for (int a = 0; a < 3; a++) c[a] = (float)(0.5 * (mn[a] + mx[a]));
            for (const float *v : vs) {
                double d2 = 0.0;
                for (int a = 0; a < 3; a++) d2 += ((double)v[a] - c[a]) * ((double)v[a] - c[a]);
                r2 = std::max(r2, d2);
            }
            return make_float4(c[0], c[1], c[2], (float)((std::sqrt(r2) + reach) * (1.0 + 1e-6)));
        };
        // [cluster spheres | triangle spheres | triangles]
        std::vector<float4> spheres(nc + n);
        std::vector<TileTri> tris(std::max<size_t>(n, 1));
        std::vector<const float *> vs;
        for (size_t c = 0; c < nc; c++) {
            vs.clear();
            for (size_t i = c * per; i < std::min(n, (c + 1) * per); i++) {
                const float *v = &env->xyz[9 * (size_t)order[i]];
                for (int p = 0; p < 3; p++) vs.push_back(v + 3 * p);
                spheres[nc + i] = ball({v, v + 3, v + 6});
                std::copy(v, v + 9, tris[i].v);
                tris[i].rec = rec[order[i]];
                tris[i].pad[0] = tris[i].pad[1] = 0;
            }
            spheres[c] = ball(vs);
        }
        const size_t sbytes = 16 * (nc + n);
        if (env->d_tile_scene.reserve(sbytes + sizeof(TileTri) * tris.size()) != cudaSuccess) {
            (void)cudaGetLastError();
            return VRG_OK;  // no room: the rows are walked
        }
        VRG_CUDA(ctx, cudaMemcpyAsync(env->d_tile_scene.ptr, spheres.data(), sbytes, cudaMemcpyHostToDevice, st));
        VRG_CUDA(ctx, cudaMemcpyAsync(env->d_tile_scene.as<char>() + sbytes, tris.data(), sizeof(TileTri) * tris.size(),
                                      cudaMemcpyHostToDevice, st));
        VRG_CUDA(ctx, cudaStreamSynchronize(st));
        env->tile_tris = (int32_t)n;
        env->tile_per = (int32_t)per;
    }
    const int32_t n = env->tile_tris, per = env->tile_per, nc = (n + per - 1) / per;
    ts.ntris = n;
    ts.nclusters = nc;
    ts.per = per;
    ts.upper = 1;
    for (int32_t r = 0; r < k; r++)
        if (!(dirs[3 * r + 2] >= 0.0f)) ts.upper = 0;
    ts.clusters = env->d_tile_scene.as<float4>();
    ts.spheres = ts.clusters + nc;
    ts.tris = reinterpret_cast<const TileTri *>(ts.spheres + n);
    ts.reach = (float)reach;
    ts.plane_eps = std::ldexp(16.0f * (env->geom.scale + 1.0f), -23);
    ts.bin_scale = (float)kDistBins / (2.0f * env->geom.scale + 1.0f);
    // cones of the bundles and the tiles
    const int nb = k / 32;
    cones.assign(2 * (size_t)nb, make_float4(0, 0, 1, -1));
    spread.assign(2 * (size_t)nb, make_float2(0, 2));
    for (int width = 1; width <= kTileBundles; width <<= 1)
        for (int t0 = 0; t0 < nb; t0 += width) {
            const float *d = &dirs[3 * (size_t)t0 * 32];
            const int m = width * 32;
            double c[3] = {0, 0, 0};
            for (int i = 0; i < m; i++)
                for (int a = 0; a < 3; a++) c[a] += d[3 * i + a];
            const double len = std::sqrt(c[0] * c[0] + c[1] * c[1] + c[2] * c[2]);
            if (!(len > 1e-3 * m)) continue;  // no axis: touches everything
            float cf[3];
            for (int a = 0; a < 3; a++) cf[a] = (float)(c[a] / len);
            float d2 = 0.0f;
            for (int i = 0; i < m; i++) {
                const float x = d[3 * i] - cf[0], y = d[3 * i + 1] - cf[1], z = d[3 * i + 2] - cf[2];
                d2 = std::max(d2, x * x + y * y + z * z);
            }
            // directions and rotated axes are off unit length by up to 1e-4
            const double chord = std::sqrt((double)d2) + 5e-4;
            const double half = 2.0 * std::asin(std::min(1.0, 0.5 * chord));
            cones[(nb + t0) / width] = make_float4(cf[0], cf[1], cf[2], (float)std::cos(half));
            spread[(nb + t0) / width] = make_float2((float)std::sin(half), (float)chord);
        }
    tiles = n > 0;
    return VRG_OK;
}

}  // namespace

int run_make_transfers(vrg_env *env, const float *dirs_local, int32_t k) {
    vrg_ctx *ctx = env->ctx;
    const int64_t rows = (int64_t)env->patches.leaf_patch.size();
    env->have_transfers = false;
    env->nnz = 0;
    env->transfer_k = k;
    std::vector<float> dirs;
    order_directions(dirs_local, k, dirs);
    TileScene ts{};
    std::vector<float4> cones;
    std::vector<float2> spread;
    bool tiles = false;
    {
        const int rc = prepare_tiles(env, dirs, k, ts, cones, spread, tiles);
        if (rc != VRG_OK) return rc;
    }
    // staged entries per row: a row has at most k, and one of more than the
    // limit (7,168 unless lowered) goes to the sorting kernel
    const int nleaves = (int)rows;
    const int tsize = std::min(k, kStageMax);
    const int limit = std::min(ctx->xfer_table_limit, tsize);
    const size_t words = (size_t)(nleaves + 31) / 32;
    const size_t smem = words <= kBitmapShared ? 4 * words : 0;
    const int64_t scratch_stride = 32 * (int64_t)std::max<size_t>(words, 1) + (words <= kBitmapShared ? 0 : (int64_t)words);
    // variants, picked per (triangles, rows) bucket: rows walked ray by ray in
    // the hierarchy by 256 threads or in the kd tree by 256 or 512, and where
    // they can be traced in tiles (prepare_tiles) tiles of 128 rays by 512
    // threads and of 64 by 256 or 128.  On lit rooms of 108, 420, 816, 2,016
    // and 8,208 triangles at k = 256, 1,024, 4,096, 8,192 and 65,536 the rows took
    // 0.05, 0.93, 6.4, 42 and 1,605 ms in the hierarchy, 0.07, 1.11, 6.7, 40 and
    // 845 ms in the kd tree (whose walk suits neighbouring rays) and 0.09, 1.09,
    // 5.2, 31 and 423 ms in the best tiles (the widest only at k = 65,536: wider
    // tiles see more triangles but share them among more rays).
    using RowKernel = void (*)(DevScene, BvhView, const LeafInfo *, const FaceRec *, const PatchNode *, const int32_t *,
                               const int32_t *, const float *, int, int64_t, int64_t, int, int, int, uint32_t *, int64_t,
                               int32_t *, int32_t *, int32_t *);
    using TileKernel = void (*)(DevScene, TileScene, const LeafInfo *, const FaceRec *, const PatchNode *,
                                const int32_t *, const int32_t *, const float *, int64_t, int64_t, int, int, int,
                                uint32_t *, int64_t, int32_t *, int32_t *, int32_t *);
    constexpr int kWalkVariants = 3, kTileVariants = 3;
    const RowKernel kvar[kWalkVariants] = {k_transfer_rows<256, true>, k_transfer_rows<256, false>,
                                            k_transfer_rows<512, false>};
    const TileKernel tvar[kTileVariants] = {k_transfer_tiles<4, 512>, k_transfer_tiles<2, 256>, k_transfer_tiles<2, 128>};
    const int vthreads[kWalkVariants + kTileVariants] = {256, 256, 512, 512, 256, 128};
    const int tbundles[kTileVariants] = {4, 2, 2};
    const size_t tile_smem = smem + 28 * (size_t)ts.nclusters;
    // (a kernel's limit is the process's, not the call's: always the largest that
    // a scene can need, so that no thread lowers another's)
    constexpr int kSmemMax = 4 * kBitmapShared, kTileSmemMax = kSmemMax + 28 * kClusterMax;
    for (const RowKernel kern : kvar)
        VRG_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax));
    for (const TileKernel kern : tvar)
        VRG_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileSmemMax));
    // rows go through in chunks whose staging stays near 1 GiB
    const int64_t chunk =
        std::max<int64_t>(1, std::min<int64_t>(rows, ((int64_t)1 << 30) / (8 * (int64_t)tsize)));
    // the context's scratch [staged columns | counts | row sizes | directions |
    // cones | spreads | counters]; this call waits for its kernels
    std::lock_guard<std::mutex> scratch(ctx->scratch_mu);
    struct Trim {  // however the call ends
        DevBuf &buf;
        ~Trim() {
            if (buf.bytes > kScratchKept) buf.release();
        }
    } trim{ctx->scratch};
    size_t at = 0;
    auto part = [&at](size_t bytes) {
        const size_t here = at;
        at = (at + bytes + 255) & ~(size_t)255;
        return here;
    };
    const size_t stage = 4 * (size_t)chunk * tsize;
    const size_t at_col = part(stage), at_cnt = part(stage), at_nnz = part(4 * (size_t)chunk),
                 at_dirs = part(12 * (size_t)k), at_cones = part(16 * cones.size()), at_spread = part(8 * spread.size()),
                 at_counters = at;
    const size_t row_counters = 4 * (size_t)scratch_stride;  // of one block
    int64_t grid_max = transfer_blocks(rows, ctx->num_sms, row_counters, (uint64_t)8 << 30, 0);
    if (at_counters + grid_max * row_counters > ctx->scratch.bytes) {
        // a larger scratch than the context holds: fewer blocks where memory is short
        size_t free_b = 0, total_b = 0;
        VRG_CUDA(ctx, cudaMemGetInfo(&free_b, &total_b));
        uint64_t reserve;
        {
            std::lock_guard<std::mutex> lk(ctx->mu);
            reserve = ctx->hbm_reserve;
        }
        free_b += ctx->scratch.bytes;
        grid_max = transfer_blocks(rows, ctx->num_sms, row_counters, free_b > at_counters ? free_b - at_counters : 0, reserve);
        for (;; grid_max = (grid_max + 1) / 2) {
            const cudaError_t e = ctx->scratch.reserve(at_counters + grid_max * row_counters);
            if (e == cudaSuccess) break;
            (void)cudaGetLastError();
            if (e != cudaErrorMemoryAllocation || grid_max == 1) return cuda_fail(ctx, e, "transfer scratch");
        }
    }
    const size_t count_bytes = grid_max * row_counters;
    char *base = ctx->scratch.as<char>();
    int32_t *stage_col = reinterpret_cast<int32_t *>(base + at_col), *stage_cnt = reinterpret_cast<int32_t *>(base + at_cnt);
    uint32_t *counters = reinterpret_cast<uint32_t *>(base + at_counters);
    int32_t *d_nnz = reinterpret_cast<int32_t *>(base + at_nnz);
    float *d_dirs = reinterpret_cast<float *>(base + at_dirs);
    ts.cones = reinterpret_cast<const float4 *>(base + at_cones);
    ts.spread = reinterpret_cast<const float2 *>(base + at_spread);
    VRG_CUDA(ctx, cudaMemsetAsync(counters, 0, count_bytes, ctx->stream));
    VRG_CUDA(ctx, cudaMemcpyAsync(d_dirs, dirs.data(), 12 * (size_t)k, cudaMemcpyHostToDevice, ctx->stream));
    if (!cones.empty()) {
        VRG_CUDA(ctx, cudaMemcpyAsync(base + at_cones, cones.data(), 16 * cones.size(), cudaMemcpyHostToDevice, ctx->stream));
        VRG_CUDA(ctx, cudaMemcpyAsync(base + at_spread, spread.data(), 8 * spread.size(), cudaMemcpyHostToDevice, ctx->stream));
    }
    // rows past the limit go to the sorting kernel twice: once for their
    // counts, once (after row_ptr is known) to write their entries; its
    // scratch is 2k int32 per block
    const int ovf_threads = std::min(512, k);
    const int ovf_grid_max = ctx->num_sms * 2;
    DevBuf ovf_scratch, ovf_rows, ovf_nnz;
    std::vector<int64_t> row_ptr(rows + 1, 0);
    std::vector<int32_t> h_nnz(chunk);
    std::vector<int64_t> ovf_list;
    VRG_CUDA(ctx, env->d_row_ptr.reserve(8 * (size_t)(rows + 1)));
    DevScene s = scene_view(env);
    env->transfer_overflow_rows = 0;
    for (int64_t r0 = 0; r0 < rows; r0 += chunk) {
        const int64_t nr = std::min(chunk, rows - r0);
        const int grid = (int)std::min<int64_t>(nr, grid_max);
        cudaEvent_t ev = nullptr;
        auto launch = [&](int v) -> cudaError_t {
            timing_begin(ctx, "transfer_rows", &ev);
            if (v >= kWalkVariants) {
                TileScene vts = ts;
                vts.ntiles = k / (32 * tbundles[v - kWalkVariants]);
                const int threads = std::min(vthreads[v], std::max(128, 32 * vts.ntiles));
                tvar[v - kWalkVariants]<<<grid, threads, tile_smem, ctx->stream>>>(
                    s, vts, env->d_leaf_info.as<LeafInfo>(), env->d_faces.as<FaceRec>(),
                    env->d_patch_nodes.as<PatchNode>(), env->d_face_root.as<int32_t>(),
                    env->d_tri_face.as<int32_t>(), d_dirs, r0, nr, nleaves, tsize, limit,
                    counters, scratch_stride, stage_col, stage_cnt,
                    d_nnz);
            } else {
                // a row block never has more threads than rays
                const int vv = vthreads[v] <= k ? v : v == 2 ? 1 : v;
                kvar[vv]<<<grid, std::min(vthreads[vv], k), smem, ctx->stream>>>(
                    s, bvh_view(env), env->d_leaf_info.as<LeafInfo>(), env->d_faces.as<FaceRec>(),
                    env->d_patch_nodes.as<PatchNode>(), env->d_face_root.as<int32_t>(),
                    env->d_tri_face.as<int32_t>(), d_dirs, k, r0, nr, nleaves, tsize, limit,
                    counters, scratch_stride, stage_col, stage_cnt,
                    d_nnz);
            }
            const cudaError_t e = cudaGetLastError();
            timing_end(ctx, "transfer_rows", ev);
            return e;
        };
        // scenes and directions that cannot be traced in tiles are tuned apart
        const std::string key = tune_key("transfer_rows", env->geom.ntris, rows * (int64_t)k);
        const int rc = tune_run(ctx, tiles ? key : tune_key("transfer_rows_walk", env->geom.ntris, rows * (int64_t)k),
                                kWalkVariants + (tiles ? kTileVariants : 0), launch, key);
        if (rc != VRG_OK) return rc;
        VRG_CUDA(ctx, cudaMemcpyAsync(h_nnz.data(), d_nnz, 4 * (size_t)nr, cudaMemcpyDeviceToHost, ctx->stream));
        VRG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        ovf_list.clear();
        for (int64_t i = 0; i < nr; i++)
            if (h_nnz[i] < 0) ovf_list.push_back(r0 + i);
        const int64_t novf = (int64_t)ovf_list.size();
        env->transfer_overflow_rows += novf;
        const int ovf_grid = (int)std::min<int64_t>(std::max<int64_t>(novf, 1), ovf_grid_max);
        auto sorted_rows = [&](const int64_t *rp) -> cudaError_t {
            timing_begin(ctx, "transfer_rows_sorted", &ev);
            k_transfer_rows_sorted<512><<<ovf_grid, ovf_threads, 0, ctx->stream>>>(
                s, bvh_view(env), env->d_leaf_info.as<LeafInfo>(), env->d_faces.as<FaceRec>(), env->d_patch_nodes.as<PatchNode>(),
                env->d_face_root.as<int32_t>(), env->d_tri_face.as<int32_t>(), d_dirs, k,
                ovf_rows.as<int64_t>(), novf, ovf_scratch.as<int32_t>(), rp, env->d_col.as<int32_t>(),
                env->d_weight.as<float>(), ovf_nnz.as<int32_t>());
            const cudaError_t e = cudaGetLastError();
            timing_end(ctx, "transfer_rows_sorted", ev);
            return e;
        };
        if (novf > 0) {
            VRG_CUDA(ctx, ovf_scratch.reserve(8 * (size_t)ovf_grid * k));
            VRG_CUDA(ctx, ovf_rows.reserve(8 * (size_t)novf));
            VRG_CUDA(ctx, ovf_nnz.reserve(4 * (size_t)novf));
            VRG_CUDA(ctx, cudaMemcpyAsync(ovf_rows.ptr, ovf_list.data(), 8 * (size_t)novf, cudaMemcpyHostToDevice,
                                          ctx->stream));
            VRG_CUDA(ctx, sorted_rows(nullptr));
            std::vector<int32_t> onnz(novf);
            VRG_CUDA(ctx, cudaMemcpyAsync(onnz.data(), ovf_nnz.ptr, 4 * (size_t)novf, cudaMemcpyDeviceToHost,
                                          ctx->stream));
            VRG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
            for (int64_t j = 0; j < novf; j++) h_nnz[ovf_list[j] - r0] = onnz[j];
        }
        for (int64_t i = 0; i < nr; i++) row_ptr[r0 + i + 1] = row_ptr[r0 + i] + h_nnz[i];
        const int64_t need = row_ptr[r0 + nr];
        if (grow(ctx, env->d_col, 4 * (size_t)std::max<int64_t>(need, 1), 4 * (size_t)row_ptr[r0]) != VRG_OK ||
            grow(ctx, env->d_weight, 4 * (size_t)std::max<int64_t>(need, 1), 4 * (size_t)row_ptr[r0]) != VRG_OK)
            return VRG_ERR_NOMEM;
        VRG_CUDA(ctx, cudaMemcpyAsync(env->d_row_ptr.as<int64_t>() + r0, row_ptr.data() + r0, 8 * (size_t)(nr + 1),
                                      cudaMemcpyHostToDevice, ctx->stream));
        if (novf > 0) VRG_CUDA(ctx, sorted_rows(env->d_row_ptr.as<int64_t>()));
        timing_begin(ctx, "transfer_gather", &ev);
        k_transfer_gather<<<(int)std::min<int64_t>((nr + 7) / 8, (int64_t)ctx->num_sms * 16), 256, 0, ctx->stream>>>(
            stage_col, stage_cnt, tsize, d_nnz,
            env->d_row_ptr.as<int64_t>(), r0, nr, k, env->d_col.as<int32_t>(), env->d_weight.as<float>());
        VRG_CUDA(ctx, cudaGetLastError());
        timing_end(ctx, "transfer_gather", ev);
        // the staging and the pageable row_ptr are reused by the next chunk
        VRG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    }
    VRG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    env->nnz = row_ptr[rows];
    env->have_transfers = true;
    return VRG_OK;
}

}  // namespace vrg
