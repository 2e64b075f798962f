"""The buckets that launches are tuned under: by the work that was asked for, and by
the kind of kernel that does it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(ctx, seed, n_faces, spacing, sky=True):
    from vrad_gb300 import scenes
    from vrad_gb300.environment import Environment

    lit = scenes.lit_scene(seed, n_faces=n_faces, spacing=spacing, n_point=2, n_spot=1, sky=sky)
    env = Environment(ctx)
    env.add_triangles(lit.xyz, lit.ids)
    env.SetupAccelerationStructure()
    env.set_faces(lit)
    env.set_lights(lit.lights)
    leaves = env.make_patches()["n_leaves"]
    env.make_transfers(scenes.transfer_directions(64))
    return env, leaves


@pytest.fixture
def fresh_ctx(vlib):
    from vrad_gb300.environment import Context

    return Context(0)


def _tuned(ctx, tmp_path):
    """The keys tuned so far and their variants."""
    p = tmp_path / "tuned.txt"
    ctx.autotune_save(str(p))
    return {k: int(v) for k, v in (line.split() for line in p.read_text().splitlines())}


def test_batches_are_keyed_by_their_points(fresh_ctx, tmp_path):
    from vrad_gb300.environment import Batch

    for spacing in range(20, 90):
        made = [_scene(fresh_ctx, 70 + i, 1 + i % 3, float(spacing), sky=False) for i in range(12)]
        points = [n for env, leaves in made for n in (env.num_luxels(), leaves)]
        total, padded = sum(points), sum((n + 31) // 32 * 32 for n in points)
        if total.bit_length() != padded.bit_length():
            break
    else:
        pytest.fail("no batch near a power of two")
    batch = Batch(fresh_ctx)
    for env, _ in made:
        batch.add(env)
    batch.bake(supersamples=1, max_bounces=2)
    tris = sum(env.num_triangles() for env, _ in made)
    keys = [k for k in _tuned(fresh_ctx, tmp_path) if k.startswith("batch_gather")]
    assert [k[k.index("/"):] for k in keys] == [f"/t{tris.bit_length() - 1}/n{total.bit_length() - 1}"]
