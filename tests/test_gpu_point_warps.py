"""Sample points that are not numbers share a warp with points that are: the box
the warp picks its lights by must not lose a light for the others."""
import numpy as np
import pytest

from conftest import bits_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [np.nan, -np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("normal", [(-0.6, 0.0, 0.8), (0.6, -0.8, 0.0), (0.0, 0.0, -1.0)])
def test_neighbours_of_a_bad_point(gpu_ctx, oracle, bad, normal):
    from vrad_gb300 import scenes
    from vrad_gb300.environment import Environment

    lit = scenes.lit_scene(11, n_faces=12, n_point=40, n_spot=6)
    for light in lit.lights:  # in reach of every point
        if "distance" in light.keys:
            light.keys["distance"] = 0.0
    env = Environment(gpu_ctx)
    env.add_triangles(lit.xyz, lit.ids)
    env.SetupAccelerationStructure()
    env.set_lights(lit.lights)
    rng = np.random.default_rng(4)
    pts = rng.uniform(1.0, 4095.0, (96, 3)).astype(np.float32)
    for i, axis in enumerate((0, 1, 2)):
        pts[32 * i + 7, axis] = np.float32(bad)
        pts[32 * i + 19, (axis + 1) % 3] = np.float32(bad)
    nrm = np.tile(np.asarray(normal, np.float32), (len(pts), 1))
    got, rays = env.gather_points(pts, nrm)
    fine = np.isfinite(pts).all(axis=1)
    want, _ = oracle.gather_points(oracle.Scene(lit.xyz, lit.ids), oracle.make_lights(lit.lights), len(lit.lights),
                                   pts[fine], nrm[fine])
    den = np.maximum(np.abs(want), 1e-3 * np.abs(want).max())
    assert np.abs(want).max() > 0
    assert (np.abs(got[fine].astype(np.float64) - want) / den).max() <= 1e-4
    alone = np.concatenate([env.gather_points(p[None], n[None])[0] for p, n in zip(pts[fine], nrm[fine])])
    assert bits_equal(got[fine], alone)
