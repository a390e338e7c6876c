"""Frames of one pixel, the smallest input of the kernels that move a warp's
slot records together: forty cameras around a scene and seeds, each pixel against
the FP32 oracle with the same random streams.  At least 97% of them agree within
1e-3, as of the pixels of the larger frames of test_gpu_render.py.
"""
import numpy as np
import pytest

import optixrender_b200 as rt
from optixrender_b200 import scenes, serve_bench
from test_gpu_render import pixel_agreement, pyoracle


@pytest.mark.gpu
@pytest.mark.parametrize("rng_mode", [rt.RNG_PCG32, rt.RNG_LCG])
@pytest.mark.parametrize("scene", ["cornell", "textured", "media"])
def test_single_pixels(scene, rng_mode):
    if scene == "media":
        spec = scenes.media(1, 1, 16, grid_res=16, env_size=(64, 32))
        spec.settings["max_depth"] = 8
    else:
        spec = getattr(scenes, scene)(1, 1, 16)
    spec.settings["rng"] = rng_mode
    s, r = scenes.build_renderer(spec)
    oracle = pyoracle.OracleScene(spec)
    g = np.random.default_rng(8)
    gpu, cpu = [], []
    for seed in range(1, 41):
        cam = rt.camera(**serve_bench.orbit_camera(spec.camera, g))
        opts = rt.options(**dict(spec.settings, seed=seed))
        r.set_options(opts)
        r.set_camera(cam)
        r.render()
        gpu.append(r.download_linear().reshape(4))
        cpu.append(oracle.render(opts, cam)[0].reshape(4))
    gpu, cpu = np.array(gpu), np.array(cpu)
    assert (cpu[:, :3].max(1) > 0).sum() >= 20  # most of them see light
    assert pixel_agreement(gpu, cpu) >= 0.97
    assert np.allclose(gpu[:, 3], 1.0)
