"""Ray queries need no unit directions.  A batch of more rays than the chip
holds threads (half-precision node boxes) gives the records of one thread per
ray (single-precision boxes), bit for bit, at direction lengths from 2^-20 to
2^95; rays along an axis and with a zero component are among them.  (From 2^97
on products of the triangle test fall below the smallest float and distances
come out wrong in both loops.)
"""
import numpy as np
import pytest

import optixrender_b200 as rt
from optixrender_b200 import scenes
from test_gpu_trace_queue import _rays


@pytest.mark.gpu
@pytest.mark.parametrize("any_hit", [False, True])
def test_direction_lengths(any_hit):
    torch = pytest.importorskip("torch")
    r = rt.Renderer(scenes.build_scene(scenes.spheres(ico_level=5, env_size=(64, 32))), rt.options(width=4, height=4))
    n = 160001
    part = 128 * torch.cuda.get_device_properties(0).multi_processor_count
    assert n > 8 * part  # more than the persistent loop's threads
    unit = _rays(n, 6)
    unit = unit[np.isfinite(unit).all(1)]
    for power in (-20, 0, 20, 60, 66, 73, 80, 90, 95):
        rays = unit.copy()
        rays[:, 4:7] = np.ldexp(unit[:, 4:7], power)
        rays[:, 3] = np.ldexp(unit[:, 3], -power)
        finite = unit[:, 7] < 1e30
        rays[finite, 7] = np.ldexp(unit[finite, 7], -power)
        whole = r.trace(rays, any_hit=any_hit)
        parts = np.concatenate([r.trace(rays[i:i + part], any_hit=any_hit) for i in range(0, len(rays), part)])
        assert (parts[:, 3].view(np.int32) >= 0).mean() > 0.1, power
        assert np.array_equal(whole.view(np.int32), parts.view(np.int32)), power
