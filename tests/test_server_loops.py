"""The traversal loop of a server's wave follows the scenes of that wave's own
jobs, not every resident scene: the rule, compiled for the host, and jobs of
small and large scenes before and after a large scene becomes resident, whose
images equal renders alone bit for bit (the captured waves of both loops are in
use side by side).
"""
import subprocess

import numpy as np
import pytest

import optixrender_b200 as rt
from optixrender_b200 import scenes
from conftest import ROOT
from test_gpu_server import _alone, _job_for


def test_loop_of_a_wave(tmp_path):
    (tmp_path / "drv.cpp").write_text(r"""
#include <cstdio>
#include "rt_schedule.h"
int main() {
    long long few, large;
    while (std::scanf("%lld %lld", &few, &large) == 2) std::printf("%d\n", rti::few_loop(few, large) ? 1 : 0);
}
""")
    subprocess.run(["g++", "-std=c++17", "-I", str(ROOT / "optixrender_b200" / "csrc"), str(tmp_path / "drv.cpp"), "-o",
                    str(tmp_path / "drv")], check=True)
    cases = [(1, 0), (1 << 26, 0), (3, 1), (3 << 24, 1 << 24), (0, 1), (0, 1 << 26), (2, 1), ((3 << 20) - 1, 1 << 20)]
    out = subprocess.run([str(tmp_path / "drv")], input="".join(f"{a} {b}\n" for a, b in cases), text=True,
                         capture_output=True, check=True).stdout
    assert [int(x) for x in out.split()] == [1, 1, 1, 1, 0, 0, 0, 0]


@pytest.mark.gpu
def test_a_large_scene_added_between_jobs():
    small, large = scenes.cornell(64, 48, 6, seed=7), scenes.spheres(80, 45, 3, seed=3, ico_level=5, env_size=(64, 32))
    srv = rt.Server(rt.server_options(wave_paths=1 << 14, max_jobs=16, max_depth=32))
    keep = [scenes.build_scene(small), scenes.build_scene(large)]

    def check(jobs):
        for spec, seed, job in jobs:
            srv.wait(job, 120000.0)
            assert np.array_equal(srv.download(job).view(np.uint32), _alone(spec, seed=seed)[0].view(np.uint32))
            srv.release(job)

    sid = srv.add_scene(keep[0])
    before = [(small, 70 + k, srv.submit(_job_for(small, sid, seed=70 + k))) for k in range(3)]
    lid = srv.add_scene(keep[1])  # while the first jobs' waves may still run
    check(before)
    check([(small, 80, srv.submit(_job_for(small, sid, seed=80)))])
    check([(large, 81, srv.submit(_job_for(large, lid, seed=81)))])
    mixed = [(small, 90 + k, srv.submit(_job_for(small, sid, seed=90 + k))) for k in range(4)]
    mixed.append((large, 95, srv.submit(_job_for(large, lid, seed=95))))
    check(mixed)
    srv.close()
