"""Transfer rows whose origin lies on a triangle: every ray that crosses its plane hits it at
t = +0 or -0, a ray that stays in the plane goes on.  A tile's rays must not end with the others."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _on_triangles(lit, P, rng):
    """`lit` with a small triangle through the origin of every third leaf's rays, across the face's
    second axis: the first direction of the table stays in its plane."""
    leaf = np.nonzero(P["leaf_index"] >= 0)[0][::3]
    extra = []
    for p in leaf:
        f = P["face"][p]
        q = P["center"][p] + lit.normal[f] * np.float32(0.125)
        across = int(np.argmax(np.abs(np.cross(lit.normal[f], lit.u[f]))))
        a, b = (across + 1) % 3, (across + 2) % 3
        size = rng.uniform(2.0, 9.0)
        v = np.tile(q, (3, 1))
        v[:, a] += np.float32(size) * np.array([-1, 1, 0], np.float32)
        v[:, b] += np.float32(size) * np.array([-1, -1, 1], np.float32)
        extra.append(v.ravel())
    lit.xyz = np.concatenate([lit.xyz, np.array(extra, np.float32)])
    lit.ids = np.concatenate([lit.ids, np.full(len(extra), 0x02000000, np.int32)])
    lit.tri_face = np.concatenate([lit.tri_face, np.full(len(extra), -1, np.int32)])
    return lit


@pytest.mark.parametrize("seed,n_faces,k", [(5, 300, 512), (6, 700, 128), (7, 300, 4096)])
def test_rays_in_the_plane_go_on(gpu_ctx, oracle, tmp_path, seed, n_faces, k):
    from test_gpu_transfer_tiles import VARIANTS, _env, _lists, _same
    from vrad_gb300 import scenes

    lit = scenes.lit_scene(seed, n_faces=n_faces, spacing=96.0, n_point=1, n_spot=1)
    P = oracle.make_patches(lit)
    lit = _on_triangles(lit, P, np.random.default_rng(seed))
    dirs = scenes.transfer_directions(k)
    assert dirs[0, 1] == 0.0
    ptr, col, cnt = oracle.make_transfers(oracle.Scene(lit.xyz, lit.ids), lit, P, dirs, threads=16)
    want = ptr, col, (cnt / np.float32(k)).astype(np.float32)
    assert (np.diff(ptr) == 1).sum() > 10  # rows of which only that direction gets anywhere
    env, leaves = _env(gpu_ctx, lit)
    for v in range(VARIANTS):
        for _ in range(3):  # a row's clusters come in any order within a distance
            assert _same(_lists(gpu_ctx, tmp_path, env, leaves, dirs, v)[0], want), v
