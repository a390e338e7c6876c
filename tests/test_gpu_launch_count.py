"""rt_render_stats.launches counts every kernel of the last Render(): begin and
finalize; per wave raygen, resolve and the advance of the wave table, and per
bounce extend, shade, sample and shadow; guided, per wave the quads of the
dense grid levels and per bounce an inference; training, per wave the collected
samples and per step a batch, the backward and weight-gradient passes and the
two Adam kernels.
"""
import pytest

import optixrender_b200 as rt
from optixrender_b200 import scenes


@pytest.mark.gpu
@pytest.mark.parametrize("guided,train,steps", [(0, 0, 4), (1, 0, 4), (1, 2, 3), (1, 5, 1)])
def test_kernels_of_a_render(guided, train, steps):
    spec = scenes.portal(48, 32, 5)
    depth, spp = 6, 5
    s, r = scenes.build_renderer(spec, guided=guided, guide_train_spp=train, guide_steps=steps, max_depth=depth, spp=spp)
    trained = 0
    for _ in range(2):  # the second frame replays captured waves and trains what is left
        r.render()
        r.synchronize()
        st = r.stats()
        t = min(spp, train - trained) if guided else 0
        trained += t
        want = 2 + st["waves"] * (3 + 4 * depth)
        if guided:
            want += st["waves"] * (1 + depth) + t * (1 + 5 * steps)
        assert st["launches"] == want
