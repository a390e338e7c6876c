"""Frames smaller than a warp's batch, ragged ones and ones just past it: the
shade kernel moves the slot records of 32 queue items at a time through shared
memory, and the queues of a frame end anywhere in such a batch.  Same random
streams as the FP32 oracle: at least 97% of the pixels within 1e-3, as for the
larger frames of test_gpu_render.py (a frame of fewer than 34 pixels: all but one).
"""
import numpy as np
import pytest

import optixrender_b200 as rt
from optixrender_b200 import scenes
from test_gpu_render import pixel_agreement, render_both


@pytest.mark.gpu
@pytest.mark.parametrize("rng_mode", [rt.RNG_PCG32, rt.RNG_LCG])
@pytest.mark.parametrize("size", [(1, 1), (5, 3), (31, 1), (33, 1), (37, 19)])
@pytest.mark.parametrize("scene", ["cornell", "textured", "media"])
def test_frames_around_a_warps_batch(scene, size, rng_mode):
    w, h = size
    if scene == "media":
        spec = scenes.media(w, h, 2, grid_res=16, env_size=(64, 32))
        spec.settings["max_depth"] = 8
    else:
        spec = getattr(scenes, scene)(w, h, 2)
    r, gpu, cpu, alb, nrm = render_both(spec, rng=rng_mode)
    agree = pixel_agreement(gpu, cpu)
    assert agree >= min(0.97, 1 - 1 / (w * h))
    assert np.allclose(gpu[..., 3], 1.0)
