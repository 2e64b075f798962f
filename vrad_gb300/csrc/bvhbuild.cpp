// bvhbuild.cpp -- the four-wide bounding-volume hierarchy the line queries
// walk (vrg_bvh.cuh), built on host threads while the device builds the walk
// tree.
//
// Top-down binned SAH (Wald, "On fast construction of SAH-based bounding
// volume hierarchies", 2007) over the triangles' boxes, 16 bins per axis of
// the box centres (every split of the widest axis for the last few triangles),
// down to leaves of at most kBvhLeaf triangles; the binary
// tree is then collapsed by opening the child of largest surface until a node
// has four.  Child boxes are kept as bytes on a grid of the node (as in Ylitie, Karras
// and Laine, "Efficient incoherent ray traversal on GPUs through compressed
// wide BVHs", 2017).  On the 12,300-triangle room an any-hit line visits 17 four-wide
// nodes and 0.3 triangles where the kd walk visits 51 nodes and 6.3.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <limits>
#include <thread>

#include "vrg_crew.h"
#include "vrg_internal.h"

namespace vrg {

namespace {

constexpr int kBins = 16;
constexpr int kSweepPrims = 24;       // so few are sorted, not binned
constexpr int kForkDepth = 4;         // both sides of a node above this depth are built at once
constexpr int32_t kForkPrims = 16384;  // a pass over fewer primitives is not shared among threads
constexpr float kInfH = std::numeric_limits<float>::infinity();

typedef float Float4 __attribute__((vector_size(16)));
typedef int32_t Int4 __attribute__((vector_size(16)));

inline Float4 least(Float4 a, Float4 b) { return a < b ? a : b; }

// A box as its lower corner and its negated upper corner, so that growing it
// is two vector minima; the fourth lane is not used.
struct Box {
    Float4 lo = {kInfH, kInfH, kInfH, 0.0f}, nhi = {kInfH, kInfH, kInfH, 0.0f};
    void add(const Box &b) {
        lo = least(lo, b.lo);
        nhi = least(nhi, b.nhi);
    }
    float hi(int a) const { return -nhi[a]; }
    float area() const {
        const float x = -nhi[0] - lo[0], y = -nhi[1] - lo[1], z = -nhi[2] - lo[2];
        return x >= 0.0f ? x * y + y * z + z * x : 0.0f;
    }
};

// A triangle: its box and its index.  Twice its centre is lo - nhi.
struct Prim {
    Box box;
    int32_t id;
    Float4 centre() const { return box.lo - box.nhi; }
};

struct Node2 {
    Box box;
    int32_t child[2];  // -1: leaf
    int32_t first, count;
};

struct Bins {
    Box box[3][kBins];
    int32_t count[3][kBins] = {};
};

// Runs f(part, first, last) over [first, last) in `parts` parts, on as many
// threads.
template <class F>
void parallel(int parts, int32_t first, int32_t last, F f) {
    const int64_t n = last - first;
    Crew crew;
    for (int p = 1; p < parts; p++)
        crew.run([=, &f] { f(p, first + (int32_t)(n * p / parts), first + (int32_t)(n * (p + 1) / parts)); });
    f(0, first, first + (int32_t)(n / parts));
    crew.join();
}

struct Builder {
    std::vector<Prim> prims, spare;
    std::vector<Node2> nodes;
    std::atomic<int32_t> used{0};
    int threads = 1;
    bool balanced = false;  // halve by count only (a tree of known depth)

    int parts(int depth, int32_t n) const {
        return (int)std::max<int64_t>(1, std::min<int64_t>(threads >> std::min(depth, 16), n / (kForkPrims / 4)));
    }

    // The box of [first, last) and of twice its centres.
    void bounds(int depth, int32_t first, int32_t last, Box &box, Box &cb) {
        const int np = last - first < kForkPrims ? 1 : parts(depth, last - first);
        std::vector<Box> b(np), c(np);
        parallel(np, first, last, [&](int p, int32_t i0, int32_t i1) {
            Box x, y;
            for (int32_t i = i0; i < i1; i++) {
                x.add(prims[i].box);
                const Float4 m = prims[i].centre();
                y.lo = least(y.lo, m);
                y.nhi = least(y.nhi, -m);
            }
            b[p] = x;
            c[p] = y;
        });
        for (int p = 0; p < np; p++) {
            box.add(b[p]);
            cb.add(c[p]);
        }
    }

    // The same for a few primitives: every split of their order along the
    // widest axis.
    int32_t sweep(int32_t first, int32_t n, const Box &box, const Box &cb, bool &leaf) {
        int ax = 0;
        for (int a = 1; a < 3; a++)
            if (cb.hi(a) - cb.lo[a] > cb.hi(ax) - cb.lo[ax]) ax = a;
        Prim *p = &prims[first];
        float key[kSweepPrims], right[kSweepPrims];
        for (int32_t i = 0; i < n; i++) {
            const Prim v = p[i];
            const float k = v.centre()[ax];
            int32_t j = i;
            for (; j > 0 && (key[j - 1] > k || (key[j - 1] == k && p[j - 1].id > v.id)); j--) {
                key[j] = key[j - 1];
                p[j] = p[j - 1];
            }
            key[j] = k;
            p[j] = v;
        }
        Box r;
        for (int32_t i = n - 1; i > 0; i--) {
            r.add(p[i].box);
            right[i] = r.area() * (float)(n - i);
        }
        Box l;
        float best = kInfH;
        int32_t at = n / 2;
        for (int32_t i = 1; i < n; i++) {
            l.add(p[i - 1].box);
            const float cost = l.area() * (float)i + right[i];
            if (cost < best) {
                best = cost;
                at = i;
            }
        }
        leaf = n <= kBvhLeaf && !(best + box.area() < box.area() * (float)n);
        return first + at;
    }

    // Splits [first, last); returns the first entry of the right side.
    int32_t split(int depth, int32_t first, int32_t last, const Box &box, const Box &cb, bool &leaf) {
        const int32_t n = last - first;
        leaf = false;
        int best_axis = -1, best_bin = 0;
        float best = kInfH;
        if (!balanced && n <= kSweepPrims) return sweep(first, n, box, cb, leaf);
        if (!balanced) {
            Float4 scale = {0.0f, 0.0f, 0.0f, 0.0f};
            for (int a = 0; a < 3; a++) {
                const float e = cb.hi(a) - cb.lo[a];
                scale[a] = e > 0.0f ? (float)kBins * 0.9999f / e : 0.0f;
            }
            const Float4 lo = {cb.lo[0], cb.lo[1], cb.lo[2], 0.0f};
            auto bins_of = [&](const Prim &p) { return __builtin_convertvector((p.centre() - lo) * scale, Int4); };
            auto clamp = [](int b) { return std::min(kBins - 1, std::max(0, b)); };
            const int np = n < kForkPrims ? 1 : parts(depth, n);
            std::vector<Bins> bins(np);
            parallel(np, first, last, [&](int p, int32_t i0, int32_t i1) {
                Bins &k = bins[p];
                for (int32_t i = i0; i < i1; i++) {
                    const Int4 b = bins_of(prims[i]);
                    for (int a = 0; a < 3; a++) {
                        const int c = clamp(b[a]);
                        k.box[a][c].add(prims[i].box);
                        k.count[a][c]++;
                    }
                }
            });
            Bins &k = bins[0];
            for (int p = 1; p < np; p++)
                for (int a = 0; a < 3; a++)
                    for (int b = 0; b < kBins; b++) {
                        k.box[a][b].add(bins[p].box[a][b]);
                        k.count[a][b] += bins[p].count[a][b];
                    }
            for (int a = 0; a < 3; a++) {
                if (!(scale[a] > 0.0f)) continue;
                float right[kBins];
                int32_t rn[kBins];
                Box r;
                int32_t c = 0;
                for (int b = kBins - 1; b > 0; b--) {
                    r.add(k.box[a][b]);
                    c += k.count[a][b];
                    right[b] = r.area();
                    rn[b] = c;
                }
                Box l;
                c = 0;
                for (int b = 1; b < kBins; b++) {
                    l.add(k.box[a][b - 1]);
                    c += k.count[a][b - 1];
                    if (c == 0 || rn[b] == 0) continue;
                    const float cost = l.area() * (float)c + right[b] * (float)rn[b];
                    if (cost < best) {
                        best = cost;
                        best_axis = a;
                        best_bin = b;
                    }
                }
            }
            if (best_axis >= 0) {
                auto goes_left = [&](const Prim &p) { return clamp(bins_of(p)[best_axis]) < best_bin; };
                int32_t m;
                if (np == 1) {
                    m = (int32_t)(std::partition(prims.begin() + first, prims.begin() + last, goes_left) - prims.begin());
                } else {  // counted per part, then moved through the spare array
                    std::vector<int32_t> left(np, 0), size(np, 0);
                    parallel(np, first, last, [&](int p, int32_t i0, int32_t i1) {
                        for (int32_t i = i0; i < i1; i++) left[p] += goes_left(prims[i]) ? 1 : 0;
                        size[p] = i1 - i0;
                    });
                    std::vector<int32_t> l(np), r(np);
                    m = first;
                    for (int p = 0; p < np; p++) {
                        l[p] = m;
                        m += left[p];
                    }
                    int32_t at = m;
                    for (int p = 0; p < np; p++) {
                        r[p] = at;
                        at += size[p] - left[p];
                    }
                    parallel(np, first, last, [&](int p, int32_t i0, int32_t i1) {
                        for (int32_t i = i0; i < i1; i++) spare[goes_left(prims[i]) ? l[p]++ : r[p]++] = prims[i];
                    });
                    parallel(np, first, last, [&](int, int32_t i0, int32_t i1) {
                        std::copy(spare.begin() + i0, spare.begin() + i1, prims.begin() + i0);
                    });
                }
                if (m > first && m < last) return m;
            }
        }
        if (n <= kBvhLeaf) {
            leaf = true;
            return first;
        }
        int ax = 0;
        for (int a = 1; a < 3; a++)
            if (cb.hi(a) - cb.lo[a] > cb.hi(ax) - cb.lo[ax]) ax = a;
        const int32_t m = (first + last) / 2;
        std::nth_element(prims.begin() + first, prims.begin() + m, prims.begin() + last, [ax](const Prim &x, const Prim &y) {
            const float cx = x.centre()[ax], cy = y.centre()[ax];
            return cx < cy || (cx == cy && x.id < y.id);
        });
        return m;
    }

    int32_t build(int depth, int32_t first, int32_t last) {
        const int32_t id = used.fetch_add(1);
        Node2 nd;
        Box cb;
        bounds(depth, first, last, nd.box, cb);
        nd.child[0] = nd.child[1] = -1;
        nd.first = first;
        nd.count = last - first;
        bool leaf = nd.count < 2;
        const int32_t mid = leaf ? first : split(depth, first, last, nd.box, cb, leaf);
        if (!leaf) {
            if (depth < kForkDepth && nd.count > 1024 && threads > 1) {
                Crew left;
                left.run([&] { nd.child[0] = build(depth + 1, first, mid); });
                nd.child[1] = build(depth + 1, mid, last);
                left.join();
            } else {
                nd.child[0] = build(depth + 1, first, mid);
                nd.child[1] = build(depth + 1, mid, last);
            }
        }
        nodes[id] = nd;
        return id;
    }

    // Which child a four-wide node opens: the one of larger surface; in a
    // balanced tree of more triangles, so that its levels pair up.
    bool wider(const Node2 &a, const Node2 &b) const {
        return balanced ? a.count > b.count : a.box.area() > b.box.area();
    }

    // A subtree left for later: its binary node, the walk's stack when it
    // enters it, and the child word that waits for its root.
    struct Task {
        int32_t id;
        int stack;
        uint32_t node;
        int child;
        std::vector<BvhNode> out;
        int deepest = 0;
    };

    // The four-wide node of binary node `id`, in preorder; `stack` is the
    // number of entries a walk may hold when it enters it.  With `tasks` the
    // children `levels` further down are put there instead.
    uint32_t collapse(int32_t id, int stack, std::vector<BvhNode> &out, int &deepest, std::vector<Task> *tasks = nullptr,
                      int levels = 0) {
        int32_t ch[4] = {id, -1, -1, -1};
        int n = 1;
        if (nodes[id].child[0] >= 0) {
            ch[0] = nodes[id].child[0];
            ch[1] = nodes[id].child[1];
            n = 2;
        }
        while (n < 4) {
            int open = -1;
            for (int c = 0; c < n; c++)
                if (nodes[ch[c]].child[0] >= 0 && (open < 0 || wider(nodes[ch[c]], nodes[ch[open]]))) open = c;
            if (open < 0) break;
            const int32_t o = ch[open];
            ch[open] = nodes[o].child[0];
            ch[n++] = nodes[o].child[1];
        }
        const uint32_t at = (uint32_t)out.size();
        out.emplace_back();
        // three siblings wait while a walk follows one child, whatever n is: a
        // ray whose reciprocal is no number passes the unused boxes too
        deepest = std::max(deepest, stack + 4);
        uint32_t word[4];
        for (int c = 0; c < 4; c++) {
            word[c] = bvh_leaf_word(0u, 1u);
            if (c >= n) continue;
            const Node2 &k = nodes[ch[c]];
            if (k.child[0] < 0)
                word[c] = bvh_leaf_word((uint32_t)k.first, (uint32_t)k.count);
            else if (tasks && levels == 0)
                tasks->push_back(Task{ch[c], stack + n - 1, at, c, {}});
            else
                word[c] = collapse(ch[c], stack + n - 1, out, deepest, tasks, levels - 1);
        }
        BvhNode o{};
        Box all;
        for (int c = 0; c < n; c++) all.add(nodes[ch[c]].box);
        float step[3];
        for (int a = 0; a < 3; a++) {
            // a step that takes 240 of them over the extent, none too small
            // to move a coordinate of this size
            const double lo = (double)all.lo[a], e = (double)all.hi(a) - lo;
            const double big = std::max(std::fabs(lo), std::fabs((double)all.hi(a)));
            int ex;
            std::frexp(std::max(std::max(e / 240.0, big * 0x1p-22), 1e-30), &ex);
            const double s = std::ldexp(1.0, ex);
            o.origin[a] = (float)(lo - 4.0 * s);
            step[a] = (float)s;
            for (int c = 0; c < 4; c++) {
                int64_t ql = 255, qh = 0;
                if (c < n) {
                    const Box &b = nodes[ch[c]].box;
                    ql = (int64_t)std::floor(((double)b.lo[a] - o.origin[a]) / s) - 2;
                    qh = (int64_t)std::ceil(((double)b.hi(a) - o.origin[a]) / s) + 2;
                }
                o.bound[2 * a] |= (uint32_t)std::max<int64_t>(0, std::min<int64_t>(255, ql)) << (8 * c);
                o.bound[2 * a + 1] |= (uint32_t)std::max<int64_t>(0, std::min<int64_t>(255, qh)) << (8 * c);
            }
        }
        o.step_x = step[0];
        o.step_y = step[1];
        o.step_z = step[2];
        for (int c = 0; c < 4; c++) o.child[c] = word[c];
        out[at] = o;
        return at;
    }
};

}  // namespace

// `order` gets the finite triangles as the leaves list them, `nodes` the
// four-wide tree over them, root first; an empty tree when there is none.  A
// tree a walk's stack could not hold is built again by halving (depth of the
// logarithm of the count); false when that does not fit either.
bool build_bvh(const std::vector<float> &xyz, std::vector<int32_t> &order, std::vector<BvhNode> &nodes) {
    Builder b;
    const int64_t n = (int64_t)xyz.size() / 9;
    b.threads = (int)std::min(16u, std::max(1u, std::thread::hardware_concurrency()));
    const bool many = n >= kForkPrims;
    std::vector<Prim> all(n);
    std::vector<char> finite(n);
    parallel(many ? b.threads : 1, 0, (int32_t)n, [&](int, int32_t t0, int32_t t1) {
        for (int32_t t = t0; t < t1; t++) {
            Prim &p = all[t];
            bool ok = true;
            for (int c = 0; c < 3; c++) {
                const float *v = &xyz[9 * (size_t)t + 3 * c];
                for (int a = 0; a < 3; a++) ok = ok && std::fabs(v[a]) <= 1e30f;
                const Float4 w = {v[0], v[1], v[2], 0.0f};
                p.box.lo = least(p.box.lo, w);
                p.box.nhi = least(p.box.nhi, -w);
            }
            p.id = t;
            finite[t] = ok;
        }
    });
    if (std::find(finite.begin(), finite.end(), 0) == finite.end()) {
        b.prims.swap(all);
    } else {
        for (int64_t t = 0; t < n; t++)
            if (finite[t]) b.prims.push_back(all[t]);
    }
    order.clear();
    nodes.clear();
    if (b.prims.empty()) return true;
    b.nodes.resize(2 * b.prims.size());
    if (many) b.spare.resize(b.prims.size());
    for (int pass = 0; pass < 2; pass++) {
        b.balanced = pass == 1;
        b.used = 0;
        const int32_t root = b.build(0, 0, (int32_t)b.prims.size());
        nodes.clear();
        int deepest = 0;
        if (!many) {
            b.collapse(root, 0, nodes, deepest);
        } else {  // the subtrees three levels down on all threads
            std::vector<Builder::Task> tasks;
            b.collapse(root, 0, nodes, deepest, &tasks, 2);
            std::atomic<size_t> next{0};
            parallel(b.threads, 0, b.threads, [&](int, int32_t, int32_t) {
                for (size_t i; (i = next.fetch_add(1)) < tasks.size();)
                    b.collapse(tasks[i].id, tasks[i].stack, tasks[i].out, tasks[i].deepest);
            });
            size_t at = nodes.size();
            for (Builder::Task &t : tasks) {
                nodes[t.node].child[t.child] = (uint32_t)at;
                at += t.out.size();
                deepest = std::max(deepest, t.deepest);
            }
            nodes.resize(at);
            next = 0;
            parallel(b.threads, 0, b.threads, [&](int, int32_t, int32_t) {
                for (size_t i; (i = next.fetch_add(1)) < tasks.size();) {
                    const Builder::Task &t = tasks[i];
                    const uint32_t base = nodes[t.node].child[t.child];
                    for (size_t k = 0; k < t.out.size(); k++) {
                        BvhNode o = t.out[k];
                        for (uint32_t &w : o.child)
                            if (!(w & kBvhLeafBit)) w += base;
                        nodes[base + k] = o;
                    }
                }
            });
        }
        if (deepest <= kBvhStack) break;
        nodes.clear();
    }
    if (nodes.empty()) return false;
    order.resize(b.prims.size());
    for (size_t i = 0; i < order.size(); i++) order[i] = b.prims[i].id;
    return true;
}

}  // namespace vrg
