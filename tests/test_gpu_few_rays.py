"""The kernel that tests every triangle for few rays, where a quotient underflows: a plane
behind the origin by less than a rounding is met at t = -0, which a start of 0 accepts."""
import numpy as np
import pytest

from conftest import bits_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 40])
def test_hits_at_minus_zero(gpu_ctx, oracle, m):
    from vrad_gb300.environment import Environment

    xyz = np.array([[-1, -1, 0, 1, -1, 0, 0, 1, 0], [-1, -1, 2, 1, -1, 2, 0, 1, 2]], np.float32)
    ids = np.full(2, 0x02000000, np.int32)
    env = Environment(gpu_ctx)
    env.add_triangles(xyz, ids)
    env.SetupAccelerationStructure()
    o = np.zeros((m, 3), np.float32)
    o[:, 2] = np.float32(1e-28) * (1 + np.arange(m, dtype=np.float32))  # just past the first plane
    d = np.zeros((m, 3), np.float32)
    d[:, 2] = np.where(np.arange(m) % 2 == 0, np.float32(1e25), np.float32(1.0))
    t0, t1 = np.zeros(m, np.float32), np.full(m, np.inf, np.float32)
    hit, t = env.trace_closest(o, d, t0, t1)
    rhit, rt = oracle.Scene(xyz, ids).trace_closest(o, d, t0, t1, brute=True)
    assert rhit[0] == 0 and rt[0] == 0.0 and np.signbit(rt[0])
    assert np.array_equal(hit, rhit) and bits_equal(t, rt)
