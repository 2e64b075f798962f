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


def _bucket(env, work):
    return f"/t{env.num_triangles().bit_length() - 1}/n{work.bit_length() - 1}"


def test_maps_and_walk_are_tuned_apart(fresh_ctx, tmp_path):
    env, leaves = _scene(fresh_ctx, 60, 30, 24.0)
    points = env.num_luxels() * 4
    env.gather_direct_light(4, 1)  # walks
    assert set(_tuned(fresh_ctx, tmp_path)) >= {"direct_luxels_walk" + _bucket(env, points)}
    assert "direct_luxels" + _bucket(env, points) not in _tuned(fresh_ctx, tmp_path)
    for _ in range(40000 // points + 1):
        env.gather_direct_light(4, 1)
    assert "direct_luxels" + _bucket(env, points) in _tuned(fresh_ctx, tmp_path)


def test_batches_with_maps_are_tuned_apart(fresh_ctx, tmp_path):
    """One scene without a sky light does not send the others back to the walk."""
    from vrad_gb300.environment import Batch

    made = [_scene(fresh_ctx, 61 + i, 30, 8.0, sky=i != 1) for i in range(3)]
    batch = Batch(fresh_ctx)
    for env, _ in made:
        batch.add(env)
    batch.bake(supersamples=4, max_bounces=2)
    assert [k.split("/")[0] for k in _tuned(fresh_ctx, tmp_path) if "batch" in k] == ["batch_gather"]


def test_rows_that_cannot_be_tiled_are_tuned_apart(fresh_ctx, tmp_path):
    from vrad_gb300 import scenes

    env, leaves = _scene(fresh_ctx, 62, 30, 48.0)
    dirs = scenes.transfer_directions(512)
    lists = env.get_transfers(leaves, env.make_transfers(dirs * np.float32(3.0)))  # not unit vectors
    key = "transfer_rows" + _bucket(env, leaves * 512)
    assert key.replace("rows", "rows_walk") in _tuned(fresh_ctx, tmp_path) and key not in _tuned(fresh_ctx, tmp_path)
    env.make_transfers(dirs)
    v, ms = fresh_ctx.autotune_choice(key)
    assert v in range(6) and len(ms) == 6
    # a tiled choice is nothing to rows that are walked
    again = env.get_transfers(leaves, env.make_transfers(dirs * np.float32(3.0)))
    assert all(np.array_equal(x, y) for x, y in zip(lists, again))


def test_choices_of_a_file_count_for_both(fresh_ctx, tmp_path):
    env, leaves = _scene(fresh_ctx, 63, 30, 24.0)
    points = env.num_luxels() * 4
    p = tmp_path / "one.txt"
    p.write_text(f"direct_luxels{_bucket(env, points)} 5\n")
    fresh_ctx.autotune_load(str(p))
    for _ in range(40000 // points + 2):
        env.gather_direct_light(4, 1)
    assert _tuned(fresh_ctx, tmp_path)["direct_luxels" + _bucket(env, points)] == 5
    assert not any(k.startswith("direct_luxels_walk") for k in _tuned(fresh_ctx, tmp_path))
