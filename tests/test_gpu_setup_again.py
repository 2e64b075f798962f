"""SetupAccelerationStructure again: what was made of the first tree is made anew."""
import numpy as np
import pytest

from conftest import bits_equal

pytestmark = pytest.mark.gpu


def test_maps_and_tiles_follow_the_tree(gpu_ctx):
    from test_sky_map_sizes import _gather_until_tried
    from test_gpu_transfer_tiles import _env, _same
    from vrad_gb300 import scenes

    env, leaves = _env(gpu_ctx, scenes.lit_scene(3, n_faces=96, spacing=24.0, n_point=2, n_spot=1))
    dirs = scenes.transfer_directions(512)
    built = _gather_until_tried(gpu_ctx, env)
    light = env.gather_direct_light(1, 3)
    lists = env.get_transfers(leaves, env.make_transfers(dirs))
    rng = np.random.default_rng(1)
    a, b = (rng.uniform(1, 4095, (6000, 3)).astype(np.float32) for _ in range(2))
    lines = env.occlusion_mask(a, b, closest=True)
    for _ in range(2):
        env.SetupAccelerationStructure()
        assert _gather_until_tried(gpu_ctx, env) == built > 0
        again = env.gather_direct_light(1, 3)
        assert again[1] == light[1] and bits_equal(again[0], light[0])
        assert _same(env.get_transfers(leaves, env.make_transfers(dirs)), lists)
        assert all(bits_equal(x, y) for x, y in zip(env.occlusion_mask(a, b, closest=True), lines))
