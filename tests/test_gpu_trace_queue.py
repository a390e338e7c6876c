"""Ray queries of more rays than the chip holds threads go through the
persistent loop with lane refill; smaller batches take one thread per ray.

A ray meets the same boxes and triangles in the same order in both loops, so
its whole record is equal bit for bit, also where several triangles lie at
exactly the same distance (the Cornell boxes stand on the floor).  Rays that
are not numbers, have no direction or an empty extent, and ragged batch sizes,
are in the batch.
"""
import numpy as np
import pytest

import optixrender_b200 as rt
from optixrender_b200 import scenes

FMAX = np.float32(3.4028235e38)


def _rays(n, seed):
    g = np.random.default_rng(seed)
    o = g.uniform(-2.5, 2.5, (n, 3))
    d = g.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    r = np.zeros((n, 8), np.float32)
    r[:, :3], r[:, 3], r[:, 4:7], r[:, 7] = o, 1e-4, d, FMAX
    k = g.integers(0, n, n // 8)
    r[k, 7] = g.uniform(0.0, 3.0, len(k))       # finite extents
    k = g.integers(0, n, n // 16)
    r[k, 4 + g.integers(0, 3, len(k))] = 0.0    # parallel to an axis plane
    k = g.integers(0, n, n // 16)
    r[k, 4:7] = np.eye(3, dtype=np.float32)[g.integers(0, 3, len(k))] * np.where(g.random((len(k), 1)) < 0.5, 1, -1)
    odd = g.integers(0, n, 60)
    r[odd[:10], 4:7] = 0.0                      # no direction
    r[odd[10:20], 4] = np.nan
    r[odd[20:30], 0] = np.nan
    r[odd[30:40], 7] = 0.0                      # empty extent
    r[odd[40:50], 0] = 1e30
    r[odd[50:], 7] = np.inf
    return r


@pytest.mark.gpu
@pytest.mark.parametrize("any_hit", [False, True])
@pytest.mark.parametrize("scene", ["spheres", "cornell"])
def test_refilled_lanes_answer_like_one_thread_per_ray(scene, any_hit):
    torch = pytest.importorskip("torch")
    spec = scenes.spheres(ico_level=5, env_size=(64, 32)) if scene == "spheres" else scenes.cornell()
    r = rt.Renderer(scenes.build_scene(spec), rt.options(width=4, height=4))
    # no GPU this runs on holds 2^19 threads; one thread per ray up to a block per multiprocessor
    n = (1 << 19) + 77
    part = 128 * torch.cuda.get_device_properties(0).multi_processor_count
    rays = _rays(n, 3)
    whole = r.trace(rays, any_hit=any_hit)
    parts = np.concatenate([r.trace(rays[i:i + part], any_hit=any_hit) for i in range(0, n, part)])
    assert (whole[:, 3].view(np.int32) >= 0).any()  # the batch meets the scene
    assert np.array_equal(whole.view(np.int32), parts.view(np.int32))


@pytest.mark.gpu
def test_batches_around_the_line_between_the_two_loops():
    torch = pytest.importorskip("torch")
    r = rt.Renderer(scenes.build_scene(scenes.cornell()), rt.options(width=4, height=4))
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rays = _rays(sms * 16 * 128 + 1, 9)
    full = r.trace(rays, any_hit=True)
    for blocks in range(1, 17):  # the line is at a whole number of blocks per multiprocessor
        for n in (sms * blocks * 128 - 1, sms * blocks * 128, sms * blocks * 128 + 1):
            assert np.array_equal(r.trace(rays[:n], any_hit=True).view(np.int32), full[:n].view(np.int32))


@pytest.mark.gpu
@pytest.mark.parametrize("any_hit", [False, True])
def test_more_triangles_at_a_step_than_the_warps_list_holds(any_hit):
    """Thousands of large triangles through each other: every node a ray visits has most of its leaves hit, so a
    step brings several hundred triangles where the list holds 128, and rays keep the rest for later steps."""
    torch = pytest.importorskip("torch")
    g = np.random.default_rng(5)
    tri = (g.uniform(-1, 1, (6000, 1, 3)) + g.uniform(-1.5, 1.5, (6000, 3, 3))).astype(np.float32)
    s = rt.Scene()
    s.add_mesh(tri.reshape(-1, 3), rt.material(rt.MAT_DIFFUSE))
    r = rt.Renderer(s, rt.options(width=4, height=4))
    n = (1 << 19) + 5
    part = 128 * torch.cuda.get_device_properties(0).multi_processor_count
    rays = _rays(n, 21)
    whole = r.trace(rays, any_hit=any_hit)
    parts = np.concatenate([r.trace(rays[i:i + part], any_hit=any_hit) for i in range(0, n, part)])
    assert (whole[:, 3].view(np.int32) >= 0).mean() > 0.1
    assert np.array_equal(whole.view(np.int32), parts.view(np.int32))
