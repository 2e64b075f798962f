"""Line queries against testing every triangle: trees and rays at which a bound
of the hierarchy could be a rounding too tight (more than 4,096 rays walk it),
and the same through the kernel that tests every triangle for few rays."""
import numpy as np
import pytest

from conftest import bits_equal

pytestmark = pytest.mark.gpu
OPAQUE, SKY = 0x02000000, 0x01000000


def _soup(kind, rng):
    n = 700
    c = rng.uniform(-900, 900, (n, 1, 3))
    v = c + rng.uniform(-120, 120, (n, 3, 3))
    if kind == "one":
        v = v[:1]
    elif kind == "five":
        v = v[:5]
    elif kind == "tiny":  # a scene a millimetre wide
        v = v * 1e-6
    elif kind == "far":  # coordinates of 2e6 with detail of a few units
        v = v + 2.0e6
    elif kind == "flat":  # every triangle in one plane
        v[:, :, 1] = 37.25
    elif kind == "same":  # one triangle many times: no plane parts them
        v = np.repeat(v[:1], 600, axis=0)
    elif kind == "line":  # a chain growing by powers of two: a deep tree
        s = 2.0 ** np.arange(-30, 12, 0.5)
        v = np.stack([np.stack([s, 0 * s, 0 * s], 1), np.stack([s * 1.2, s * 0.1, 0 * s], 1),
                      np.stack([s * 1.1, 0 * s, s * 0.3], 1)], 1)
    elif kind == "degenerate":  # points, segments, and corners that are not numbers
        v[::5, 2] = v[::5, 1]
        v[1::5, 1:] = v[1::5, :1]
        v[2, 0, 0] = np.nan
        v[7, 1, 2] = np.inf
    xyz = v.reshape(-1, 9).astype(np.float32)
    ids = np.full(len(xyz), OPAQUE, np.int32)
    ids[::3] = SKY
    ids[1::7] = 0x04000000 | 5
    return np.ascontiguousarray(xyz), ids


@pytest.mark.parametrize("kind", ["plain", "one", "five", "tiny", "far", "flat", "same", "line", "degenerate"])
@pytest.mark.parametrize("m", [1, 33, 2500, 6000])
def test_queries_equal_brute_force(gpu_ctx, oracle, kind, m):
    from vrad_gb300.environment import Environment

    rng = np.random.default_rng(17)
    xyz, ids = _soup(kind, rng)
    env = Environment(gpu_ctx)
    env.add_triangles(xyz, ids)
    env.SetupAccelerationStructure()
    ref = oracle.Scene(xyz, ids)
    tri = xyz.reshape(-1, 3, 3)
    tri = tri[np.isfinite(tri).all(axis=(1, 2))]
    lo, hi = tri.min(axis=(0, 1)), tri.max(axis=(0, 1))
    size = (hi - lo).max()
    a = (lo + rng.uniform(-0.3, 1.3, (m, 3)) * (hi - lo)).astype(np.float32)
    b = (lo + rng.uniform(-0.3, 1.3, (m, 3)) * (hi - lo)).astype(np.float32)
    b[::4] = tri[rng.integers(0, len(tri), len(b[::4]))].mean(axis=1)  # ends on triangles
    a[1::4] = tri[rng.integers(0, len(tri), len(a[1::4]))].mean(axis=1)  # starts on triangles
    b[2::8] = a[2::8]  # no length
    for ax in range(3):  # along the axes
        b[3 + 8 * ax::24] = a[3 + 8 * ax::24]
        b[3 + 8 * ax::24, ax] += np.float32(0.7 * size)
    for skip in (-1, 0x04000000 | 5):
        mask, hit, t = env.occlusion_mask(a, b, skip_id=skip, closest=True)
        rmask, rhit, rt = ref.occlusion_mask(a, b, skip=skip, closest=True)
        assert np.array_equal(hit, rhit) and bits_equal(t, rt)
        assert np.array_equal(mask, rmask)
        assert np.array_equal(env.occlusion_mask(a, b, skip_id=skip), rmask)
    want = ref.test_lines(a, b, skip=0x04000000 | 5, brute=True)
    assert np.array_equal(env.test_line_does_hit_sky(a, b, 5), want)
    d = b - a
    t0 = rng.uniform(-0.5, 0.3, m).astype(np.float32)  # negative starts too
    t1 = np.where(np.arange(m) % 3 == 0, np.inf, rng.uniform(-0.2, 1.5, m)).astype(np.float32)
    hit, t = env.trace_closest(a, d, t0, t1)
    rhit, rt = ref.trace_closest(a, d, t0, t1, brute=True)
    assert np.array_equal(hit, rhit) and bits_equal(t, rt)
