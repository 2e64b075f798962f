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
