"""Transfer rows traced in tiles give the lists of rows walked ray by ray.

Variants 0 to 2 of the launch site walk, 3 to 5 trace in tiles (where the
directions and faces allow it); every one must give the same CSR."""
import numpy as np
import pytest

from conftest import bits_equal

from test_gpu_sky_map import _lit

pytestmark = pytest.mark.gpu
VARIANTS = 6


def _lists(ctx, tmp_path, env, leaves, dirs, variant):
    from vrad_gb300.environment import Context

    key = Context.tune_key("transfer_rows", env.num_triangles(), leaves * len(dirs))
    p = tmp_path / "tune.txt"
    p.write_text(f"{key} {variant}\n")
    ctx.autotune_load(str(p))
    nnz = env.make_transfers(dirs)
    return env.get_transfers(leaves, nnz), env.transfer_info()[2]


def _env(ctx, lit):
    from vrad_gb300.environment import Environment

    env = Environment(ctx)
    env.add_triangles(lit.xyz, lit.ids)
    env.SetupAccelerationStructure()
    env.set_faces(lit)
    env.set_lights(lit.lights)
    return env, env.make_patches()["n_leaves"]


def _same(a, b):
    return np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]) and bits_equal(a[2], b[2])


def _directions(k, kind):
    from vrad_gb300 import scenes

    d = scenes.transfer_directions(k)
    if kind == "sphere":  # half of them below the face
        d = d.copy()
        d[1::2, 2] *= -1.0
    elif kind == "narrow":  # a tight bundle, and many equal directions
        d = np.tile(d[: max(1, k // 64)], (64, 1))[:k]
    elif kind == "long":  # not unit vectors: the rows are walked
        d = d * np.float32(3.0)
    return np.ascontiguousarray(d, np.float32)


@pytest.mark.parametrize("kind,n_faces,k,directions", [
    ("plain", 30, 128, "hemisphere"), ("plain", 30, 64, "hemisphere"), ("plain", 7, 4096, "hemisphere"),
    ("open", 24, 512, "hemisphere"), ("tilted", 30, 1024, "hemisphere"), ("slivers", 30, 1024, "hemisphere"),
    ("sky_inside", 30, 512, "sphere"), ("skip_ids", 30, 512, "sphere"), ("plain", 30, 1024, "narrow"),
    ("tilted", 30, 256, "long")])
def test_tiles_give_the_walks_lists(gpu_ctx, tmp_path, kind, n_faces, k, directions):
    env, leaves = _env(gpu_ctx, _lit(kind, n_faces, 48.0))
    dirs = _directions(k, directions)
    ref, _ = _lists(gpu_ctx, tmp_path, env, leaves, dirs, 0)
    assert ref[0][-1] > 0
    for v in range(1, VARIANTS):
        got, _ = _lists(gpu_ctx, tmp_path, env, leaves, dirs, v)
        assert _same(got, ref), v


def test_tiles_rows_past_the_limit(gpu_ctx, tmp_path):
    env, leaves = _env(gpu_ctx, _lit("plain", 60, 48.0))
    dirs = _directions(1024, "hemisphere")
    ref, none = _lists(gpu_ctx, tmp_path, env, leaves, dirs, 0)
    assert none == 0
    gpu_ctx.set_transfer_table_limit(20)
    try:
        for v in range(VARIANTS):
            got, past = _lists(gpu_ctx, tmp_path, env, leaves, dirs, v)
            assert past == np.count_nonzero(np.diff(ref[0]) > 20) > 0
            assert _same(got, ref), v
    finally:
        gpu_ctx.set_transfer_table_limit(7168)


def test_tiles_with_many_small_triangles(gpu_ctx, tmp_path):
    # more triangles than 1,024 clusters of 16 hold: wider clusters
    from vrad_gb300 import scenes

    lit = _lit("plain", 30, 48.0)
    rng = np.random.default_rng(9)
    c = rng.uniform(200, 3900, (20000, 1, 3))
    extra = (c + rng.uniform(-12, 12, (20000, 3, 3))).astype(np.float32).reshape(-1, 9)
    lit.xyz = np.concatenate([lit.xyz, extra])
    lit.ids = np.concatenate([lit.ids, np.full(len(extra), scenes.TRACE_ID_OPAQUE, np.int32)])
    lit.tri_face = np.concatenate([lit.tri_face, np.full(len(extra), -1, np.int32)])
    env, leaves = _env(gpu_ctx, lit)
    dirs = _directions(512, "hemisphere")
    ref, _ = _lists(gpu_ctx, tmp_path, env, leaves, dirs, 0)
    for v in range(1, VARIANTS):
        assert _same(_lists(gpu_ctx, tmp_path, env, leaves, dirs, v)[0], ref), v
