"""The bench's sizes: every line of the any-hit scene against the oracle, and the
direct-light walk's variants against the sky maps."""
import numpy as np
import pytest

from conftest import bits_equal

pytestmark = pytest.mark.gpu


def test_every_line_like_the_oracle(gpu_ctx, oracle, anyhit_scene):
    from vrad_gb300.environment import Environment

    sc = anyhit_scene
    env = Environment(gpu_ctx)
    env.add_triangles(sc.xyz, sc.ids)
    env.SetupAccelerationStructure()
    rmask, rhit, rt = oracle.Scene(sc.xyz, sc.ids).occlusion_mask(sc.starts, sc.stops, threads=16, closest=True)
    mask, hit, t = env.occlusion_mask(sc.starts, sc.stops, closest=True)
    assert np.array_equal(hit, rhit) and bits_equal(t, rt) and np.array_equal(mask, rmask)
    assert np.array_equal(env.occlusion_mask(sc.starts, sc.stops), rmask)


def test_walk_variants_give_the_maps_light(gpu_ctx, lit_scene, tmp_path):
    import torch

    from vrad_gb300.environment import Context, Environment

    env = Environment(gpu_ctx)
    env.add_triangles(lit_scene.xyz, lit_scene.ids)
    env.SetupAccelerationStructure()
    env.set_faces(lit_scene)
    env.set_lights(lit_scene.lights)
    key = Context.tune_key("direct_luxels_walk", env.num_triangles(), env.num_luxels() * 4)
    walked = []
    gpu_ctx.reset_stats()
    gpu_ctx.set_timing(True)
    gpu_ctx.set_hbm_reserve(torch.cuda.mem_get_info()[1])  # no room for maps
    try:
        for v in range(12):
            p = tmp_path / f"walk_{v}.txt"
            p.write_text(f"{key} {v}\n")
            gpu_ctx.autotune_load(str(p))
            walked.append(env.gather_direct_light(4, 2))
        assert gpu_ctx.kernel_stats("sky_map")[1] == 0
        gpu_ctx.set_hbm_reserve(1 << 30)
        mapped = env.gather_direct_light(4, 2)
        assert gpu_ctx.kernel_stats("sky_map")[1] > 0
    finally:
        gpu_ctx.set_hbm_reserve(1 << 30)
        gpu_ctx.set_timing(False)
    for rgb, rays in walked:
        assert rays == mapped[1] > 0 and bits_equal(rgb, mapped[0])
