"""The half-precision node test (rt_traverse.cuh, intersect_children) over the
range of ray queries, which need no unit directions: lengths from 1e-6 to 1e36,
in scenes of 1e-6 to 1e6 times the size.  As tests/test_traversal_half.py does
for unit directions, it restates the test in numpy with the same roundings and
compares with the boxes met in double precision; here denormal results of single
precision are flushed to zero and reciprocals are off by up to two units, as
the kernels are built.
"""
import re
from pathlib import Path

import numpy as np
import pytest

from test_traversal_half import cases, exact_boxes, f16, f32

SOURCE = Path(__file__).resolve().parents[1] / "optixrender_b200" / "csrc" / "rt_traverse.cuh"


def _flush(x):
    return np.where(np.abs(x) < f32(2.0 ** -126), f32(0), x).astype(f32)


def half_boxes(g, p, e, lo, hi, o, d, tmin, tmax):
    """(n, 8) hits; p, o, d (n, 3) float32, e (n, 3) exponents, lo / hi (n, 8, 3) plane bytes."""
    least = re.search(r"mx = fmaxf\(mx, 0x1p-(\d+)f\);", SOURCE.read_text())
    z = _flush
    with np.errstate(all="ignore"):
        tiny = f32(1e-20)
        dd = np.where(np.abs(d) > tiny, d, np.where(d < 0, -tiny, tiny)).astype(f32)
        idir = z(f32(1) / dd)
        idir = z((idir.view(np.int32) + np.where(idir != 0, g.integers(-2, 3, idir.shape), 0).astype(np.int32)).view(f32))
        s = z(np.ldexp(f32(1), e).astype(f32) * idir)
        c = z(z(p - o) * idir)
        t0 = np.maximum(np.minimum(c, z(f32(255) * s + c)).max(1), tmin)[:, None]
        c = z(c - t0)
        mx = np.abs(s).max(1, keepdims=True)
        far_out = ~(np.maximum(mx, np.abs(t0)) < f32(1e30))
        lim = f32(1024) * np.maximum(np.maximum(np.abs(s).min(1, keepdims=True), z(np.abs(t0) * f32(2.0 ** -28))), f32(2.0 ** -112))
        clamped = np.abs(s) > lim
        wide = np.where(mx > lim, f32(0.65 * 2.0 ** -24), f32(0.4 * 2.0 ** -24))
        c = np.where(clamped, z(z(c / np.abs(s)) * lim), c)
        s = np.where(clamped, np.copysign(lim, s), s)
        mx = np.minimum(mx, lim)
        if least:
            mx = np.maximum(mx, f32(2.0 ** -int(least.group(1))))
        # the kernel's exponent arithmetic, out of the exponent's field included
        kb = (np.uint32(244 << 23) - (mx.view(np.uint32) & np.uint32(0x7F800000))).astype(np.uint32)
        k, k24 = kb.view(f32), (kb + np.uint32(24 << 23)).astype(np.uint32).view(f32)
        s, c = z(s * k24), z(c * k)
        b = z(z(np.abs(t0) * k) * f32(2.0 ** -21) + f32(2.0 ** -23))
        margin = z(np.abs(s) * wide + b)
        sh = s.astype(f16).astype(np.float64)
        cn, cf = ((c - margin).astype(f16).astype(np.float64), (c + margin).astype(f16).astype(np.float64))
        end = ((tmax[:, None] - t0) * (k * f32(1 + 2.0 ** -10)) + b).astype(f16).astype(np.float64)
        neg = (d < 0)[:, None, :]
        qn, qf = np.where(neg, hi, lo) * 2.0 ** -24, np.where(neg, lo, hi) * 2.0 ** -24
        tn = (qn * sh[:, None] + cn[:, None]).astype(f16).astype(np.float64)
        tf = (qf * sh[:, None] + cf[:, None]).astype(f16).astype(np.float64)
        return (np.maximum(tn.max(2), 0) <= np.minimum(tf.min(2), end)) | far_out


def _case(g, n, mode, length, scale):
    p, e, lo, hi, o, d, tmin, tmax = cases(g, n, mode)
    step = int(np.round(np.log2(scale)))
    p, o, e = np.ldexp(p, step), np.ldexp(o, step), np.where(e > -126, e + step, e)
    d = (d * f32(length)).astype(f32)
    tmin = np.where(g.random(n) < 0.5, 0, 1e-4 * scale / length).astype(f32)
    tmax = np.where(tmax < 3e38, tmax.astype(float) * (scale / length), tmax).astype(f32)
    return p.astype(f32), e, lo, hi, o.astype(f32), d, _flush(tmin), tmax


@pytest.mark.parametrize("mode", ["any", "inside", "axis", "flat"])
@pytest.mark.parametrize("length", [1e-6, 1e-3, 1.0, 1e3, 1e6, 1e12, 1e20, 1e22, 1e25, 1e28, 1e30, 1e33, 1e36])
def test_every_box_met_is_reported_at_any_direction_length(mode, length):
    g = np.random.default_rng(29)
    met = 0
    for scale in (1.0, 1e-6, 1e6):
        case = _case(g, 6000, mode, length, scale)
        ok = np.abs(case[5]).max(1) > 0
        reported, exact = half_boxes(g, *case)[ok], exact_boxes(*case)[ok]
        assert not (exact & ~reported).any(), (scale, (exact & ~reported).sum(), exact.sum())
        met += exact.sum()
    assert met > 400


@pytest.mark.parametrize("length", [1e6, 1e20, 1e28])
def test_long_directions_report_hardly_more(length):
    """Where the distances are well above the smallest floats, a direction's length changes nothing."""
    g, h = np.random.default_rng(31), np.random.default_rng(31)
    unit, long = _case(g, 20000, "any", 1.0, 1.0), _case(h, 20000, "any", length, 1.0)
    a, b = half_boxes(g, *unit).sum(), half_boxes(h, *long).sum()
    assert abs(int(a) - int(b)) <= 0.005 * a
