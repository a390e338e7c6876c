"""A guided job is admitted when the budget holds its buffers, the scene and
the guiding buffers of the wave slots (mixtures of 160 bytes, training records
of 192, samples of 96, one batch of 2^18): what the inference lays out for
itself takes no more.
"""
import pytest

import optixrender_b200 as rt
from optixrender_b200 import scenes
from test_gpu_server import _job_for

PATHS = 1 << 18
GUIDING = PATHS * (160 + 192 + 96) + 3 * (1 << 18) * 12


@pytest.mark.gpu
def test_a_guided_job_that_fits_exactly():
    spec = scenes.portal(32, 32, 4)
    scene = scenes.build_scene(spec)
    probe = rt.Server(rt.server_options(background=0, wave_paths=PATHS, max_depth=8))
    probe.add_scene(scene)
    resident = probe.stats()["bytes_in_use"]
    probe.close()
    job = 32 * 32 * 104
    for budget, fits in ((resident + GUIDING + job, True), (resident + GUIDING + job - 1, False)):
        srv = rt.Server(rt.server_options(background=0, wave_paths=PATHS, max_depth=8, hbm_budget_bytes=budget,
                                          guide_train_waves=1))
        sid = srv.add_scene(scene)
        desc = _job_for(spec, sid, guided=1, max_depth=8)
        if fits:
            assert srv.wait(srv.submit(desc))["state"] == rt.JOB_DONE
        else:
            with pytest.raises(rt.RTError):
                srv.submit(desc)
        srv.close()
