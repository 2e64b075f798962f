"""Sizes of the sky maps: what the host computes of them, and a scene whose maps would
not fit keeps the walk."""
import numpy as np
import pytest

from conftest import bits_equal

import native

OPAQUE = 0x02000000


def test_pool_entries_stay_in_32_bits(tmp_path):
    out = native.run(tmp_path, r"""
#include <cstdio>
#include "vrg_internal.h"
int main() {
    // 16,000 coincident triangles over a tenth of the cells of maps 216 cells wide
    const uint64_t cells = 162ull * 216 * 216, many = 16000ull * (cells / 10);
    printf("%d %d %d %d\n", (int)vrg::sky_pool_indexable(0), (int)vrg::sky_pool_indexable(0xffffffffull),
           (int)vrg::sky_pool_indexable(0x100000000ull), (int)vrg::sky_pool_indexable(many));
}
""")
    assert out.split() == ["1", "1", "0", "0"]


def test_sizes_hold_every_part(tmp_path):
    """What a build reserves: 12 bytes a cell to keep, 4 a cell and grid, 4 a
    triangle and direction and 48 a triangle of scratch."""
    out = native.run(tmp_path, r"""
#include <cstdio>
#include "vrg_internal.h"
int main() {
    for (int64_t nt : {1ll, 8208ll, 1200000ll, 1ll << 23})
        for (int n : {96, 512})
            for (int sky = 0; sky < 2; sky++) {
                const vrg::SkyMapSizes s(nt, n, sky);
                printf("%lld %d %d %zu %zu %zu %zu\n", (long long)nt, n, sky, s.kept, s.tri_at, s.dir_at, s.scratch);
            }
}
""")
    for line in out.splitlines():
        nt, n, sky, kept, tri_at, dir_at, scratch = map(int, line.split())
        cells = 162 * n * n
        assert kept >= 12 * cells + 162 * 64
        assert tri_at >= 256 + 4 * cells * (4 if sky else 1) + 4 * 162 * nt and tri_at % 16 == 0
        assert dir_at >= tri_at + 48 * nt and dir_at % 16 == 0
        assert scratch >= dir_at + 162 * 112


def _sheets(copies, n_faces=30):
    """Lit boxes under an opaque sheet across the room, there many times over."""
    from vrad_gb300 import scenes

    lit = scenes.lit_scene(5, n_faces=n_faces, spacing=16.0, n_point=1, n_spot=1)
    z = 4000.0
    sheet = np.array([[0, 0, z, 4096, 0, z, 4096, 4096, z], [0, 0, z, 4096, 4096, z, 0, 4096, z]], np.float32)
    lit.xyz = np.concatenate([lit.xyz, np.tile(sheet, (copies // 2, 1))])
    lit.ids = np.concatenate([lit.ids, np.full(copies, OPAQUE, np.int32)])
    lit.tri_face = np.concatenate([lit.tri_face, np.full(copies, -1, np.int32)])
    return lit


def _env(ctx, lit):
    from vrad_gb300.environment import Environment

    env = Environment(ctx)
    env.add_triangles(lit.xyz, lit.ids)
    env.SetupAccelerationStructure()
    env.set_faces(lit)
    env.set_lights(lit.lights)
    return env


def _gather_until_tried(ctx, env):
    """First and later gathers, and the launches that the maps took."""
    ctx.reset_stats()
    ctx.set_timing(True)
    try:
        first = env.gather_direct_light(1, 3)
        assert ctx.kernel_stats("sky_map")[1] == 0  # the first call walks
        for _ in range(max(24 * env.num_triangles(), 40000) // env.num_luxels() + 1):
            later = env.gather_direct_light(1, 3)
        tried = ctx.kernel_stats("sky_map")[1]
        again = env.gather_direct_light(1, 3)
        assert ctx.kernel_stats("sky_map")[1] == tried  # settled
    finally:
        ctx.set_timing(False)
    for got in (later, again):
        assert got[1] == first[1] > 0 and bits_equal(got[0], first[0])
    return tried


@pytest.mark.gpu
def test_too_many_entries_keep_the_walk(gpu_ctx):
    gpu_ctx.set_autotune(False)
    try:
        built = _gather_until_tried(gpu_ctx, _env(gpu_ctx, _sheets(2)))
        tried = _gather_until_tried(gpu_ctx, _env(gpu_ctx, _sheets(16000)))
    finally:
        gpu_ctx.set_autotune(True)
    assert 0 < tried < built  # counted, never filled


@pytest.mark.gpu
def test_lists_leave_the_reserve(gpu_ctx):
    """Lists larger than what the reserve leaves: counted, never allocated."""
    import torch

    gpu_ctx.set_autotune(False)
    try:
        built = _gather_until_tried(gpu_ctx, _env(gpu_ctx, _sheets(2)))
        env = _env(gpu_ctx, _sheets(8000))  # 8 GB of lists and more
        gpu_ctx.set_hbm_reserve(torch.cuda.mem_get_info()[0] - (5 << 30))
        tried = _gather_until_tried(gpu_ctx, env)
    finally:
        gpu_ctx.set_hbm_reserve(1 << 30)
        gpu_ctx.set_autotune(True)
    assert 0 < tried < built


@pytest.mark.gpu
def test_grids_and_triangles_leave_the_reserve(gpu_ctx):
    """1.2 million triangles: the maps and their scratch take 2.0 GB before any list."""
    import torch

    lit = _sheets(2)
    lit.nu[:] *= 12
    lit.nv[:] *= 12
    rng = np.random.default_rng(3)
    more = 1_200_000
    v = rng.uniform(1, 4000, (more, 1, 3)) + rng.uniform(-2, 2, (more, 3, 3))
    lit.xyz = np.concatenate([lit.xyz, v.reshape(-1, 9).astype(np.float32)])
    lit.ids = np.concatenate([lit.ids, np.full(more, OPAQUE, np.int32)])
    lit.tri_face = np.concatenate([lit.tri_face, np.full(more, -1, np.int32)])
    env = _env(gpu_ctx, lit)
    gpu_ctx.set_autotune(False)
    gpu_ctx.reset_stats()
    gpu_ctx.set_timing(True)
    try:
        gpu_ctx.set_hbm_reserve(torch.cuda.mem_get_info()[1])
        first = env.gather_direct_light(4, 3)
        for _ in range(24 * env.num_triangles() // (4 * env.num_luxels())):
            env.gather_direct_light(4, 3)
        gpu_ctx.set_hbm_reserve(torch.cuda.mem_get_info()[0] - 1_900_000_000)
        last = env.gather_direct_light(4, 3)
        assert gpu_ctx.kernel_stats("sky_map")[1] == 0
    finally:
        gpu_ctx.set_hbm_reserve(1 << 30)
        gpu_ctx.set_timing(False)
        gpu_ctx.set_autotune(True)
    assert last[1] == first[1] > 0 and bits_equal(last[0], first[0])
