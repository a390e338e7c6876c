"""Ray queries of several host threads on one renderer, each of more rays than
the chip holds threads, so that the persistent loop hands them out: every call
gets the records that it gets alone, bit for bit.  Calls with host and with
device buffers, of different sizes, closest and any hit, on a scene of few
nodes and a large one; and more calls at once than there are counters.
"""
import threading

import numpy as np
import pytest

import optixrender_b200 as rt
from optixrender_b200 import scenes
from test_gpu_trace_queue import _rays

COUNTS = [(1 << 19) + 77, 200003, (1 << 18) + 1, 640000]


def _run(calls):
    """Each call in a thread of its own, all started together; returns what they raised."""
    raised, start = [], threading.Barrier(len(calls))

    def work(call):
        try:
            start.wait()
            call()
        except BaseException as e:  # noqa: BLE001 - reported by the test
            raised.append(e)

    threads = [threading.Thread(target=work, args=(c,)) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return raised


@pytest.mark.gpu
@pytest.mark.parametrize("device", [False, True])
@pytest.mark.parametrize("scene", ["spheres", "cornell"])
def test_large_queries_from_several_threads(scene, device):
    torch = pytest.importorskip("torch")
    spec = scenes.spheres(ico_level=5, env_size=(64, 32)) if scene == "spheres" else scenes.cornell()
    r = rt.Renderer(scenes.build_scene(spec), rt.options(width=4, height=4))
    sets = [(_rays(n, 70 + k), bool(k & 1)) for k, n in enumerate(COUNTS)]
    want = [r.trace(rays, any_hit=a).view(np.int32) for rays, a in sets]
    bad = []

    def host(k):
        rays, a = sets[k]
        for _ in range(8):
            if not np.array_equal(r.trace(rays, any_hit=a).view(np.int32), want[k]):
                bad.append(k)

    def on_device(k):
        rays, a = sets[k]
        d, out = torch.from_numpy(rays).cuda(), torch.empty((8, len(rays), 4), device="cuda")
        torch.cuda.synchronize()
        for i in range(8):
            r.trace_device(d.data_ptr(), len(rays), out[i].data_ptr(), any_hit=a)
        got = out.cpu().numpy().view(np.int32)
        bad.extend(k for i in range(8) if not np.array_equal(got[i], want[k]))

    work = on_device if device else host
    assert not _run([lambda k=k: work(k) for k in range(len(sets))])
    assert not bad


@pytest.mark.gpu
def test_more_calls_at_once_than_counters():
    r = rt.Renderer(scenes.build_scene(scenes.cornell()), rt.options(width=4, height=4))
    rays = _rays(200003, 90)
    want = r.trace(rays).view(np.int32)
    bad = []

    def call(k):
        n = len(rays) - 17 * k
        if not np.array_equal(r.trace(rays[:n]).view(np.int32), want[:n]):
            bad.append(k)

    assert not _run([lambda k=k: call(k) for k in range(80)])
    assert not bad
