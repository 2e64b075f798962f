"""Sky maps: the sky-ambient lines answered from the maps give the walk's bits.

A scene's first gathers walk; once the points asked for repay a build the maps
answer.  The same call before and after must give the same luxels, shadow-ray
count and patch light."""
import numpy as np
import pytest

from conftest import bits_equal

SKY, OPAQUE = 0x01000000, 0x02000000
pytestmark = pytest.mark.gpu


def _rotated(soup, rng, n, sliver):
    """n triangles at random angles (edges to 700 units, or slivers half a unit wide), some degenerate."""
    c = rng.uniform(300, 3800, (n, 1, 3))
    v = c + rng.uniform(-350, 350, (n, 3, 3))
    if sliver:
        v[:, 2] = v[:, 1] + rng.uniform(-0.5, 0.5, (n, 3))
    v[::17, 2] = v[::17, 1]
    for t in v.astype(np.float32):
        soup.append((tuple(map(float, t.ravel())), OPAQUE))


def _lit(kind, n_faces, spacing):
    """A lit room with the change `kind` makes to its triangles."""
    from vrad_gb300 import scenes

    lit = scenes.lit_scene(5, n_faces=n_faces, spacing=spacing, n_point=2, n_spot=1)
    rng = np.random.default_rng(3)
    xyz, ids, face = lit.xyz.copy(), lit.ids.copy(), list(lit.tri_face)
    extra = []
    if kind == "no_sky":
        ids[ids == SKY] = OPAQUE
    elif kind == "open":  # no room at all: most lines hit nothing
        xyz, ids, face = xyz[12:], ids[12:], face[12:]
    elif kind == "sky_walls":  # sky on the floor and two walls, opaque ceiling
        ids[:12] = OPAQUE
        ids[[2, 3, 4, 5, 8, 9]] = SKY
    elif kind == "sky_inside":  # sky sheets with opaque things on both sides
        for z in (1500.0, 2500.5):
            extra.append(((500, 500, z, 3500, 700, z, 900, 3300, z + 40.0), SKY))
            extra.append(((600, 3000, z, 3300, 3200, z + 9.0, 3100, 800, z), SKY))
    elif kind == "tilted":
        _rotated(extra, rng, 120, False)
    elif kind == "slivers":
        _rotated(extra, rng, 300, True)
    elif kind == "skip_ids":  # lines skip triangles whose id is their skip id, -1
        ids[12::5] = -1
    if extra:
        xyz = np.concatenate([xyz, np.array([e[0] for e in extra], np.float32)])
        ids = np.concatenate([ids, np.array([e[1] for e in extra], np.int32)])
        face += [-1] * len(extra)
    lit.xyz, lit.ids, lit.tri_face = xyz, ids, np.asarray(face, np.int32)
    return lit


@pytest.mark.parametrize("kind,n_faces,spacing,ss", [
    ("plain", 30, 40.0, 4), ("plain", 7, 16.0, 1), ("no_sky", 24, 48.0, 4), ("open", 24, 48.0, 4),
    ("sky_walls", 30, 40.0, 4), ("sky_inside", 30, 40.0, 4), ("tilted", 30, 40.0, 4), ("slivers", 30, 40.0, 1),
    ("skip_ids", 30, 48.0, 4)])
def test_maps_give_the_walks_bits(gpu_ctx, kind, n_faces, spacing, ss):
    from vrad_gb300.environment import Environment

    lit = _lit(kind, n_faces, spacing)
    env = Environment(gpu_ctx)
    env.add_triangles(lit.xyz, lit.ids)
    env.SetupAccelerationStructure()
    env.set_faces(lit)
    env.set_lights(lit.lights)
    leaves = env.make_patches()["n_leaves"]
    gpu_ctx.reset_stats()
    gpu_ctx.set_timing(True)
    try:
        points = env.num_luxels() * ss
        assert 0 < points < 40000  # the first call walks
        walked = env.gather_direct_light(ss, 3), env.gather_patch_direct(leaves)
        assert gpu_ctx.kernel_stats("sky_map")[1] == 0
        repaid = max(40000, 24 * env.num_triangles())
        for _ in range(repaid // points + 1):
            mapped = env.gather_direct_light(ss, 3), env.gather_patch_direct(leaves)
        assert gpu_ctx.kernel_stats("sky_map")[1] > 0
    finally:
        gpu_ctx.set_timing(False)
    assert walked[0][1] == mapped[0][1] > 0
    assert np.abs(walked[0][0]).max() > 0
    assert bits_equal(walked[0][0], mapped[0][0])
    assert bits_equal(walked[1], mapped[1])


def test_faces_outside_the_scene_keep_the_walk(gpu_ctx):
    from vrad_gb300.environment import Environment

    lit = _lit("plain", 30, 40.0)
    lit.corner[0] = (9000.0, 0.0, 0.0)  # beyond what the maps' margins cover
    env = Environment(gpu_ctx)
    env.add_triangles(lit.xyz, lit.ids)
    env.SetupAccelerationStructure()
    env.set_faces(lit)
    env.set_lights(lit.lights)
    gpu_ctx.reset_stats()
    gpu_ctx.set_timing(True)
    try:
        first = env.gather_direct_light(4, 3)
        for _ in range(40000 // (env.num_luxels() * 4) + 1):
            last = env.gather_direct_light(4, 3)
        assert gpu_ctx.kernel_stats("sky_map")[1] == 0
    finally:
        gpu_ctx.set_timing(False)
    assert first[1] == last[1] and bits_equal(first[0], last[0])
