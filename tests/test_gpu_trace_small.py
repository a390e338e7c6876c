"""Host ray queries of up to 16384 rays go through blocks that the renderer
keeps; larger ones, and calls that find the blocks taken by another thread,
allocate theirs.  Every size around the line, calls in any order of sizes, and
calls from several threads at once give the records of the static-scratch
entry point, bit for bit.
"""
import ctypes as C
import threading

import numpy as np
import pytest

import optixrender_b200 as rt
from optixrender_b200 import scenes
from test_gpu_trace_queue import _rays


def _expected(r, rays, any_hit):
    f = rt.load_library().rt_renderer_trace_noalloc
    f.restype, f.argtypes = C.c_int32, [C.c_void_p, C.c_int32, C.c_void_p, C.c_int64, C.c_void_p]
    out = np.empty((len(rays), 4), np.float32)
    assert f(r.handle, int(any_hit), rays.ctypes.data, len(rays), out.ctypes.data) == rt.RT_OK
    return out.view(np.int32)


@pytest.mark.gpu
@pytest.mark.parametrize("any_hit", [False, True])
def test_sizes_around_the_line(any_hit):
    r = rt.Renderer(scenes.build_scene(scenes.cornell()), rt.options(width=4, height=4))
    rays = _rays(20000, 4)
    want = _expected(r, rays, any_hit)
    for n in (1, 2, 31, 33, 16383, 16384, 16385, 20000, 7, 16384):
        assert np.array_equal(r.trace(rays[:n], any_hit=any_hit).view(np.int32), want[:n])


@pytest.mark.gpu
def test_calls_from_several_threads():
    r = rt.Renderer(scenes.build_scene(scenes.cornell()), rt.options(width=4, height=4))
    sets = [_rays(500 + 997 * k, 50 + k) for k in range(6)]
    want = [_expected(r, s, False) for s in sets]
    bad = []

    def work(k):
        for _ in range(40):
            if not np.array_equal(r.trace(sets[k]).view(np.int32), want[k]):
                bad.append(k)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(sets))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
