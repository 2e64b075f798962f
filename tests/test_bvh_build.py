"""The line queries' hierarchy as the host builds it, without a device."""
import native

WALK = r"""
#include <cstdio>
#include <cstdlib>
#include <cmath>
#include "vrg_internal.h"
using namespace vrg;

// Most entries a walk can have stacked in a tree: every child but the one it follows.
static int deepest(const std::vector<BvhNode> &nodes, std::vector<char> &seen) {
    struct At { uint32_t node; int stacked; };
    std::vector<At> todo{{0u, 0}};
    int most = 0;
    while (!todo.empty()) {
        const At at = todo.back();
        todo.pop_back();
        most = std::max(most, at.stacked + 3);
        for (int c = 0; c < 4; c++) {
            const uint32_t w = nodes[at.node].child[c];
            if (!(w & kBvhLeafBit)) {
                todo.push_back({w, at.stacked + 3});
                continue;
            }
            const uint32_t lo = nodes[at.node].bound[0] >> (8 * c) & 255u, hi = nodes[at.node].bound[1] >> (8 * c) & 255u;
            if (lo > hi) continue;  // unused
            for (uint32_t i = 0; i < bvh_leaf_count(w); i++) seen[bvh_leaf_first(w) + i]++;
        }
    }
    return most;
}

static float u() { return (float)rand() / RAND_MAX; }

static std::vector<float> soup(int kind, int n) {
    std::vector<float> xyz;
    for (int t = 0; t < n; t++) {
        const float s = kind == 0 ? 1.0f : std::ldexp(1.0f, t % 60 - 30);  // 1: a chain of halves, a deep tree
        const float c[3] = {kind == 0 ? 900 * u() : 900 * s, kind == 0 ? 900 * u() : 0, 900 * u() * (kind == 0)};
        for (int k = 0; k < 3; k++)
            for (int a = 0; a < 3; a++) xyz.push_back(kind == 2 ? (float)(k * (a + 1)) : c[a] + 9 * s * u());
    }
    return xyz;
}
"""


def test_leaf_words_number_every_triangle(tmp_path):
    out = native.run(tmp_path, WALK + r"""
int main() {
    for (int64_t first : {(int64_t)0, (int64_t)1 << 27, ((int64_t)1 << 28) - 1, (int64_t)1 << 28, kBvhMax - 4})
        for (uint32_t count = 1; count <= (uint32_t)kBvhLeaf; count++) {
            const uint32_t w = bvh_leaf_word((uint32_t)first, count);
            printf("%d\n", (w & kBvhLeafBit) && w != kBvhNone && bvh_leaf_first(w) == (uint32_t)first &&
                               bvh_leaf_count(w) == count);
        }
}
""")
    assert set(out.split()) == {"1"}


def test_trees_hold_every_triangle_within_the_stack(tmp_path):
    out = native.run(tmp_path, WALK + r"""
int main() {
    for (int kind = 0; kind < 3; kind++)
        for (int n : {0, 1, 3, 700, 40000}) {
            const std::vector<float> xyz = soup(kind, n);
            std::vector<int32_t> order;
            std::vector<BvhNode> nodes;
            const bool ok = build_bvh(xyz, order, nodes);
            if (n == 0) {
                printf("%d\n", ok && nodes.empty() && order.empty());
                continue;
            }
            std::vector<char> seen(n, 0), once(n, 0);
            const int most = deepest(nodes, seen);
            bool all = (int)order.size() == n;
            for (int32_t t : order) once[t]++;
            for (int t = 0; t < n; t++) all = all && seen[t] == 1 && once[t] == 1;
            printf("%d\n", ok && all && most <= kBvhStack);
        }
}
""", ["bvhbuild.cpp"])
    assert out.split() == ["1"] * 15


def test_threads_that_cannot_start_or_run_out_of_memory(tmp_path):
    """No thread: the same tree on the caller's.  No memory, whichever allocation it is:
    an exception that the caller gets."""
    out = native.run(tmp_path, WALK + r"""
#include <atomic>
#include <cerrno>
#include <new>
#include <dlfcn.h>
static std::atomic<bool> no_threads{false};
static std::atomic<long> left{1l << 60};
extern "C" int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *p) {
    if (no_threads) return EAGAIN;
    static auto real = (int (*)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *))dlsym(RTLD_NEXT, "pthread_create");
    return real(t, a, f, p);
}
void *operator new(size_t n) {
    if (left.fetch_sub(1) <= 0) throw std::bad_alloc();
    if (void *p = malloc(n)) return p;
    throw std::bad_alloc();
}
void operator delete(void *p) noexcept { free(p); }
void operator delete(void *p, size_t) noexcept { free(p); }

int main() {
    const std::vector<float> xyz = soup(0, 40000);
    std::vector<int32_t> order, other;
    std::vector<BvhNode> nodes, same;
    build_bvh(xyz, order, nodes);
    no_threads = true;
    build_bvh(xyz, other, same);
    no_threads = false;
    std::vector<char> seen(40000, 0);
    bool all = other.size() == order.size() && deepest(same, seen) <= kBvhStack;
    for (char c : seen) all = all && c == 1;
    printf("%d\n", all);
    int failed = 0;
    for (long n = 0; n < 3000; n += n < 40 ? 1 : 97) {
        std::vector<int32_t> o;
        std::vector<BvhNode> k;
        left = n;
        try {
            build_bvh(xyz, o, k);
        } catch (const std::bad_alloc &) {
            failed++;
        }
        left = 1l << 60;
    }
    printf("%d\n", failed > 30);
}
""", ["bvhbuild.cpp"])
    assert out.split() == ["1", "1"]
