"""Scenes as wide as a map may be (32,768 units) and lines along their axes: a
direction component of zero must not push the hierarchy's box test out of range.
Every answer against testing every triangle."""
import numpy as np
import pytest

from conftest import bits_equal

pytestmark = pytest.mark.gpu
OPAQUE, SKY = 0x02000000, 0x01000000


def _soup(width, rng, n=700):
    c = rng.uniform(-0.5 * width, 0.5 * width, (n, 1, 3))
    v = c + rng.uniform(-0.06 * width, 0.06 * width, (n, 3, 3))
    v[::9, :, 2] = v[::9, :1, 2]  # some lie flat, some stand along an axis
    v[1::9, :, 0] = v[1::9, :1, 0]
    ids = np.full(n, OPAQUE, np.int32)
    ids[::3] = SKY
    return np.ascontiguousarray(v.reshape(-1, 9), np.float32), ids


def _directions(m, rng):
    """Along each axis, in each axis plane and anywhere, with both zeros."""
    d = rng.standard_normal((m, 3))
    d /= np.linalg.norm(d, axis=1)[:, None]
    zero = np.where(rng.integers(0, 2, (m, 3)) > 0, 0.0, -0.0)
    kind = np.arange(m) % 7
    for ax in range(3):
        d[kind == ax, ax] = zero[kind == ax, ax]  # in a plane
        for other in range(3):
            if other != ax:
                d[kind == 3 + ax, other] = zero[kind == 3 + ax, other]  # along the axis
    return d.astype(np.float32)


@pytest.mark.parametrize("width", [7000.0, 8192.0, 16384.0, 32768.0, 4.0e6, 3.0e9])
def test_axis_lines_equal_brute_force(gpu_ctx, oracle, width):
    from vrad_gb300.environment import Environment

    rng = np.random.default_rng(23)
    xyz, ids = _soup(width, rng)
    env = Environment(gpu_ctx)
    env.add_triangles(xyz, ids)
    env.SetupAccelerationStructure()
    ref = oracle.Scene(xyz, ids)
    m = 7000  # more than the kernel for few rays takes
    a = rng.uniform(-0.5 * width, 0.5 * width, (m, 3)).astype(np.float32)
    a[::2] = xyz.reshape(-1, 3, 3)[rng.integers(0, len(xyz), m)].mean(axis=1)[::2]
    d = _directions(m, rng)
    b = np.where(d == 0.0, a, a + d * np.float32(0.8 * width)).astype(np.float32)
    mask, hit, t = env.occlusion_mask(a, b, closest=True)
    rmask, rhit, rt = ref.occlusion_mask(a, b, closest=True)
    assert (rhit >= 0).mean() > 0.2
    assert np.array_equal(hit, rhit) and bits_equal(t, rt) and np.array_equal(mask, rmask)
    assert np.array_equal(env.occlusion_mask(a, b), rmask)
    assert np.array_equal(env.test_line_does_hit_sky(a, b, 5), ref.test_lines(a, b, skip=0x04000000 | 5, brute=True))
    hit, t = env.trace_closest(a, d, np.zeros(m, np.float32), np.full(m, np.inf, np.float32))
    rhit, rt = ref.trace_closest(a, d, 0.0, np.inf, brute=True)
    assert np.array_equal(hit, rhit) and bits_equal(t, rt)


@pytest.mark.parametrize("length", [1e-30, 1e-24, 1e-18, 1e-9, 1e9, 1e18, 1e25])
def test_directions_of_any_length(gpu_ctx, oracle, length):
    """Ray directions are taken as they come; a direction of no length hits nothing."""
    from vrad_gb300.environment import Environment

    rng = np.random.default_rng(29)
    xyz, ids = _soup(16384.0, rng, 300)
    env = Environment(gpu_ctx)
    env.add_triangles(xyz, ids)
    env.SetupAccelerationStructure()
    m = 5000
    a = rng.uniform(-8192.0, 8192.0, (m, 3)).astype(np.float32)
    d = (_directions(m, rng) * np.float32(length)).astype(np.float32)
    d[5::50] = 0.0
    t0 = np.zeros(m, np.float32)
    t1 = np.full(m, np.inf, np.float32)
    hit, t = env.trace_closest(a, d, t0, t1)
    rhit, rt = oracle.Scene(xyz, ids).trace_closest(a, d, t0, t1, brute=True)
    assert np.array_equal(hit, rhit) and bits_equal(t, rt)
    assert (hit[5::50] == -1).all()


def test_leaves_of_a_full_size_map(gpu_ctx, oracle):
    from vrad_gb300 import scenes
    from vrad_gb300.environment import Environment, leaf_sky_lines

    rng = np.random.default_rng(31)
    w, h, t = scenes.BrushMap(), 16384.0, 64.0
    w.box((-h, -h, -h), (h, h, -h + t))
    for ax in range(2):
        for side in (-1, 1):
            lo, hi = np.array([-h, -h, -h]), np.array([h, h, h])
            lo[ax], hi[ax] = sorted((side * h, side * (h - t)))
            w.box(lo, hi)
    w.face([(-h, -h, h), (h, -h, h), (h, h, h), (-h, h, h)], texinfo=1)
    centres, sizes = rng.uniform(-14000, 14000, (120, 3)), rng.uniform(200, 1500, (120, 3))
    for c, e in zip(centres, sizes):
        w.box(c - e, c + e)
    env = Environment(gpu_ctx)
    env.add_bsp_world(w.lumps())
    env.SetupAccelerationStructure()
    xyz, ids = env.get_triangle_vertices()
    mins = rng.integers(-16000, 15000, (300, 3)).astype(np.int32)
    maxs = (mins + rng.integers(1, 900, (300, 3))).astype(np.int32)
    solid = np.arange(120)
    mins[solid] = np.rint(centres - 20).astype(np.int32)  # inside the boxes
    maxs[solid] = mins[solid] + 40
    got = env.CanLeafTraceToSky(mins, maxs)
    a, b = leaf_sky_lines(mins, maxs)
    frac = oracle.Scene(xyz, ids).test_lines(a, b, skip=-1, threads=16)
    want = (frac.reshape(-1, 162) > 0).any(axis=1)
    assert 0.1 < want.mean() < 0.9
    assert np.array_equal(got, want)


@pytest.mark.parametrize("factor", [2.0, 8.0])
def test_transfer_rows_of_wide_scenes(gpu_ctx, oracle, tmp_path, factor):
    """Rows of every variant and of the sorted path, with directions along the normal and the edges."""
    from test_gpu_transfer_tiles import VARIANTS, _env, _lists, _same
    from vrad_gb300 import scenes

    f = np.float32(factor)
    lit = scenes.lit_scene(5, n_faces=240, spacing=96.0, n_point=1, n_spot=1)
    lit.xyz, lit.corner, lit.u, lit.v = (x * f for x in (lit.xyz, lit.corner, lit.u, lit.v))
    lit.luxscale = lit.luxscale / f
    dirs = scenes.transfer_directions(256)
    dirs[::16, 0] = -0.0  # in the planes of the faces' edges
    dirs[5::16, 1] = 0.0
    dirs[8::64] = (0.0, -0.0, 1.0)
    dirs = (dirs / np.linalg.norm(dirs, axis=1)[:, None]).astype(np.float32)
    env, leaves = _env(gpu_ctx, lit)
    P = oracle.make_patches(lit)
    ptr, col, cnt = oracle.make_transfers(oracle.Scene(lit.xyz, lit.ids), lit, P, dirs)
    want = ptr, col, (cnt / np.float32(256)).astype(np.float32)
    axial = (dirs == 0.0).any(axis=1)
    assert len(col) > len(oracle.make_transfers(oracle.Scene(lit.xyz, lit.ids), lit, P, dirs[~axial])[1])
    for v in range(VARIANTS):
        assert _same(_lists(gpu_ctx, tmp_path, env, leaves, dirs, v)[0], want), v
    gpu_ctx.set_transfer_table_limit(2)
    try:
        got, past = _lists(gpu_ctx, tmp_path, env, leaves, dirs, 1)
    finally:
        gpu_ctx.set_transfer_table_limit(7168)
    assert past > 0 and _same(got, want)
