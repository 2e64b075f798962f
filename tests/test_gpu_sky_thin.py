"""Sky maps of a scene much thinner than the faces' distance from it: a point far
below a roof is many times the map's depth away, on every direction's axis."""
import numpy as np
import pytest

from conftest import bits_equal

pytestmark = pytest.mark.gpu
OPAQUE, SKY = 0x02000000, 0x01000000


def _roof(axis, side, thick, sky):
    """A roof across one axis, and faces in a row of distances from it that no triangle covers."""
    from vrad_gb300 import scenes

    lit = scenes.lit_scene(5, n_faces=40, spacing=64.0, n_point=1, n_spot=1)
    a, b = (axis + 1) % 3, (axis + 2) % 3
    at = side * 4000.0
    quads = []
    rng = np.random.default_rng(2)
    for tid, level in ((OPAQUE, at), (SKY if sky else OPAQUE, at + side * thick)):
        for c in rng.uniform(-3000, 3000, (12, 2)):
            p = np.zeros((3, 3))
            p[:, axis] = level
            p[:, a] = c[0] + np.array([-900.0, 900.0, 0.0])
            p[:, b] = c[1] + np.array([-900.0, -900.0, 900.0])
            quads.append((p.ravel(), tid))
    lit.xyz = np.array([q[0] for q in quads], np.float32)
    lit.ids = np.array([q[1] for q in quads], np.int32)
    lit.tri_face = np.full(len(quads), -1, np.int32)
    n = lit.n_faces
    lit.corner[:] = rng.uniform(-2500, 2000, (n, 3))
    lit.corner[:, axis] = np.linspace(-3900, 3900, n)
    lit.u[:], lit.v[:], lit.normal[:] = 0.0, 0.0, 0.0
    lit.u[:, a], lit.v[:, b] = 400.0, 400.0
    lit.normal[:, axis] = side
    lit.nu[:], lit.nv[:] = 9, 9
    return lit


@pytest.mark.parametrize("axis,side", [(0, 1), (0, -1), (1, 1), (1, -1), (2, 1), (2, -1)])
@pytest.mark.parametrize("thick,sky", [(10.0, False), (0.5, True), (300.0, True)])
def test_maps_far_from_a_thin_scene(gpu_ctx, axis, side, thick, sky):
    from vrad_gb300.environment import Environment

    lit = _roof(axis, side, thick, sky)
    env = Environment(gpu_ctx)
    env.add_triangles(lit.xyz, lit.ids)
    env.SetupAccelerationStructure()
    env.set_faces(lit)
    env.set_lights(lit.lights)
    leaves = env.make_patches()["n_leaves"]
    points = env.num_luxels() * 4
    assert 0 < points < 40000  # the first call walks
    walked = env.gather_direct_light(4, 3), env.gather_patch_direct(leaves)
    for _ in range(40000 // points + 2):
        later = env.gather_direct_light(4, 3), env.gather_patch_direct(leaves)
    assert walked[0][1] == later[0][1] > 0
    assert bits_equal(walked[0][0], later[0][0]) and bits_equal(walked[1], later[1])
