"""Gather steps that the lanes of a warp share: the sky directions their normals face and the lights
within reach of their points.  Every sum keeps the order of one point alone, so the luxels are the
oracle's (within the bound of the one library call, powf) and the shadow-ray counts are equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lit(normals, n_faces, spacing, n_lights):
    from vrad_gb300 import scenes

    lit = scenes.lit_scene(9, n_faces=n_faces, spacing=spacing, n_point=max(n_lights - 2, 1), n_spot=1)
    rng = np.random.default_rng(8)
    if normals == "each":  # every face another: a warp holds many
        v = rng.standard_normal((n_faces, 3))
        lit.normal[:] = (v / np.linalg.norm(v, axis=1)[:, None]).astype(np.float32)
    elif normals == "odd":  # no direction at all, and normals of other lengths
        lit.normal[::3] = 0.0
        lit.normal[1::3] *= np.float32(1e-3)
    if n_lights == 65:  # one without range, and a sky ambient between the 32-light steps
        lit.lights[5].keys["distance"] = 0.0
        lit.lights.insert(31, lit.lights[-1])
    return lit


@pytest.mark.parametrize("normals", ["box", "each", "odd"])
@pytest.mark.parametrize("n_faces,spacing,ss,n_lights", [
    (1, 60.0, 1, 3), (33, 600.0, 1, 33), (70, 600.0, 4, 65), (31, 120.0, 4, 34)])
def test_warps_of_many_normals_and_lights(gpu_ctx, oracle, normals, n_faces, spacing, ss, n_lights):
    from vrad_gb300.environment import Environment

    lit = _lit(normals, n_faces, spacing, n_lights)
    env = Environment(gpu_ctx)
    env.add_triangles(lit.xyz, lit.ids)
    env.SetupAccelerationStructure()
    env.set_faces(lit)
    env.set_lights(lit.lights)
    scene = oracle.Scene(lit.xyz, lit.ids)
    ref, ref_rays = oracle.gather_luxels(scene, oracle.make_lights(lit.lights), len(lit.lights), lit, 0, n_faces, ss=ss,
                                         seed=2, threads=8)
    points = env.num_luxels() * ss
    gpu_ctx.reset_stats()
    gpu_ctx.set_timing(True)
    try:
        walked = env.gather_direct_light(ss, 2)
        for _ in range(max(40000, 24 * env.num_triangles()) // points + 1):
            mapped = env.gather_direct_light(ss, 2)
        assert gpu_ctx.kernel_stats("sky_map")[1] > 0
    finally:
        gpu_ctx.set_timing(False)
    assert walked[1] == mapped[1] == ref_rays
    den = np.maximum(np.abs(ref), 1e-3 * max(np.abs(ref).max(), 1e-30))
    for got in (walked[0], mapped[0]):
        assert (np.abs(got.astype(np.float64) - ref) / den).max() <= 1e-4
    assert np.array_equal(walked[0].view(np.uint32), mapped[0].view(np.uint32))


@pytest.mark.parametrize("counts", [(1, 2, 40), (33, 5, 64, 7)])
def test_batch_segments_of_part_warps(gpu_ctx, counts):
    """A batch's scenes with ragged point counts give what each gives alone."""
    from vrad_gb300 import scenes
    from vrad_gb300.environment import Batch, Environment

    envs, leaves = [], []
    for i, n in enumerate(counts):
        lit = scenes.lit_scene(20 + i, n_faces=n, spacing=90.0, n_point=3 + i, n_spot=1)
        env = Environment(gpu_ctx)
        env.add_triangles(lit.xyz, lit.ids)
        env.SetupAccelerationStructure()
        env.set_faces(lit)
        env.set_lights(lit.lights)
        leaves.append(env.make_patches()["n_leaves"])
        env.make_transfers(scenes.transfer_directions(256))
        envs.append(env)
    for ss in (1, 4):
        batch = Batch(gpu_ctx)
        for env in envs:
            batch.add(env)
        batch.bake(supersamples=ss)
        together = [env.get_bake(n) for env, n in zip(envs, leaves)]
        for env, n, got in zip(envs, leaves, together):
            alone, _ = env.gather_direct_light(ss, 0)
            assert np.array_equal(got["luxels"].view(np.uint32), alone.view(np.uint32))
            assert np.array_equal(got["patch_direct"].view(np.uint32), env.gather_patch_direct(n).view(np.uint32))
