"""Memory of the transfer build: as many counting blocks as there is room for, one at least."""
import pytest

import native


def test_counting_blocks_fit_the_memory(tmp_path):
    out = native.run(tmp_path, r"""
#include <cstdio>
#include "vrg_internal.h"
int main() {
    for (int64_t rows : {1ll, 100ll, 55000ll, 1000000ll, 2000000000ll})
        for (uint64_t free_gb : {0ull, 1ull, 3ull, 12ull, 280ull})
            for (uint64_t reserve_gb : {0ull, 1ull, 300ull}) {
                const uint64_t counters = 4 * ((uint64_t)rows + 31) / 32 * 32;
                printf("%lld %llu %llu %llu %lld\n", (long long)rows, (unsigned long long)counters, (unsigned long long)free_gb,
                       (unsigned long long)reserve_gb,
                       (long long)vrg::transfer_blocks(rows, 152, counters, free_gb << 30, reserve_gb << 30));
            }
}
""")
    lines = [tuple(map(int, line.split())) for line in out.splitlines()]
    assert len(lines) == 75
    for rows, counters, free, reserve, blocks in lines:
        assert 1 <= blocks <= min(rows, 152 * 8)
        room = min(8 << 30, max(256 << 20, (max(free - reserve, 0)) << 30))
        assert blocks == 1 or blocks * counters <= room
        assert blocks == min(rows, 152 * 8) or (blocks + 1) * counters > room


@pytest.mark.gpu
def test_lists_with_nothing_outside_the_reserve(gpu_ctx):
    import torch
    import numpy as np
    from test_gpu_transfer_tiles import _env, _same
    from vrad_gb300 import scenes

    env, leaves = _env(gpu_ctx, scenes.lit_scene(3, n_faces=96, spacing=48.0, n_point=1, n_spot=1))
    dirs = scenes.transfer_directions(256)
    want = env.get_transfers(leaves, env.make_transfers(dirs))
    gpu_ctx.set_hbm_reserve(torch.cuda.mem_get_info()[1])
    try:
        got = env.get_transfers(leaves, env.make_transfers(dirs))
    finally:
        gpu_ctx.set_hbm_reserve(1 << 30)
    assert np.count_nonzero(np.diff(want[0])) > 0 and _same(got, want)
