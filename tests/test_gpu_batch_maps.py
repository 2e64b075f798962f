"""Sky maps in a batch: scenes that need none do not keep the others from theirs, and
none is built where one scene that wants them cannot have them."""
import numpy as np
import pytest

from conftest import bits_equal

pytestmark = pytest.mark.gpu


def _scene(ctx, seed, sky=True, outside=False):
    from vrad_gb300 import scenes
    from vrad_gb300.environment import Environment

    lit = scenes.lit_scene(seed, n_faces=40, spacing=12.0, n_point=2, n_spot=1, sky=sky)
    if outside:  # past what the maps' margins cover
        lit.corner[3] = (9000.0, 0.0, 0.0)
    env = Environment(ctx)
    env.add_triangles(lit.xyz, lit.ids)
    env.SetupAccelerationStructure()
    env.set_faces(lit)
    env.set_lights(lit.lights)
    leaves = env.make_patches()["n_leaves"]
    env.make_transfers(scenes.transfer_directions(64))
    return env, leaves


def _bake(ctx, made):
    from vrad_gb300.environment import Batch

    batch = Batch(ctx)
    for env, _ in made:
        batch.add(env)
    ctx.reset_stats()
    ctx.set_timing(True)
    try:
        batch.bake(supersamples=4, seed=9, max_bounces=2)
        maps = ctx.kernel_stats("sky_map")[1]
    finally:
        ctx.set_timing(False)
    return maps, [env.get_bake(leaves) for env, leaves in made]


def _alone(made):
    return [env.gather_direct_light(4, 9)[0] for env, _ in made]


def test_a_scene_without_sky_light_among_others(gpu_ctx):
    made = [_scene(gpu_ctx, 80 + i, sky=i != 1) for i in range(3)]
    alone = _alone([_scene(gpu_ctx, 80 + i, sky=i != 1) for i in range(3)])
    passes = [_bake(gpu_ctx, made) for _ in range(6)]  # enough points to repay the maps
    built = [maps > 0 for maps, _ in passes]
    assert sum(built) == 1 and not built[-1]
    got, same = passes[0][1], passes[-1][1]
    for want, a, b in zip(alone, got, same):
        assert np.abs(want).max() > 0
        assert bits_equal(a["luxels"], want) and bits_equal(b["luxels"], want)


def test_none_is_built_where_one_cannot_be(gpu_ctx):
    made = [_scene(gpu_ctx, 90 + i, outside=i == 2) for i in range(3)]
    for _ in range(6):
        maps, got = _bake(gpu_ctx, made)
        assert maps == 0
    for want, a in zip(_alone(made), got):
        assert bits_equal(a["luxels"], want)
