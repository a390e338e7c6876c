"""The half-precision node test of the traversal (rt_traverse.cuh,
intersect_children), restated in numpy with the same roundings, is
conservative: it reports every child box that the ray meets in double
precision.  Also how much it reports beyond them.

Nodes of all sizes and aspect ratios, rays from inside and outside, nearly and
exactly parallel to an axis, with and without an end.  The one exception is a
ray with a zero direction component that lies exactly in a box without
thickness along that axis; no triangle of such a box can be hit (it is parallel
to the ray), so it is left out.
"""
import numpy as np
import pytest

f32, f16 = np.float32, np.float16


def half_boxes(p, e, lo, hi, o, d, tmin, tmax):
    """(n, 8) hits; p, o, d (n, 3) float32, e (n, 3) exponents, lo / hi (n, 8, 3) plane bytes."""
    with np.errstate(all="ignore"):
        tiny = f32(1e-20)
        dd = np.where(np.abs(d) > tiny, d, np.where(d < 0, -tiny, tiny)).astype(f32)
        idir = f32(1) / dd
        s = np.ldexp(f32(1), e).astype(f32) * idir
        c = (p - o) * idir
        t0 = np.maximum(np.minimum(c, f32(255) * s + c).max(1), tmin)[:, None]
        c = c - t0
        mx = np.abs(s).max(1, keepdims=True)
        far_out = ~(np.maximum(mx, np.abs(t0)) < f32(1e30))
        lim = f32(1024) * np.maximum(np.maximum(np.abs(s).min(1, keepdims=True), np.abs(t0) * f32(2.0 ** -28)), f32(2.0 ** -90))
        clamped = np.abs(s) > lim
        wide = np.where(mx > lim, f32(0.65 * 2.0 ** -24), f32(0.4 * 2.0 ** -24))
        c = np.where(clamped, c * (lim / np.abs(s)), c)
        s = np.where(clamped, np.copysign(lim, s), s)
        mx = np.minimum(mx, lim)
        k = np.ldexp(f32(1), 117 - ((mx.view(np.int32) & 0x7F800000) >> 23)).astype(f32)
        s = s * (k * f32(2.0 ** 24))
        c = c * k
        b = np.abs(t0) * k * f32(2.0 ** -21) + f32(2.0 ** -23)
        margin = np.abs(s) * wide + b
        sh = s.astype(f16).astype(np.float64)
        cn, cf = ((c - margin).astype(f16).astype(np.float64), (c + margin).astype(f16).astype(np.float64))
        end = ((tmax[:, None] - t0) * (k * f32(1 + 2.0 ** -10)) + b).astype(f16).astype(np.float64)
        neg = (d < 0)[:, None, :]
        qn, qf = np.where(neg, hi, lo) * 2.0 ** -24, np.where(neg, lo, hi) * 2.0 ** -24
        # a product of 8 and 11 bits and the sum are exact in double: one rounding, as the fused operation
        tn = (qn * sh[:, None] + cn[:, None]).astype(f16).astype(np.float64)
        tf = (qf * sh[:, None] + cf[:, None]).astype(f16).astype(np.float64)
        return (np.maximum(tn.max(2), 0) <= np.minimum(tf.min(2), end)) | far_out


def exact_boxes(p, e, lo, hi, o, d, tmin, tmax):
    p, o, d = (x.astype(np.float64) for x in (p, o, d))
    sc = np.ldexp(1.0, e)[:, None]
    a, b = p[:, None] + lo * sc, p[:, None] + hi * sc
    with np.errstate(all="ignore"):
        t1, t2 = (a - o[:, None]) / d[:, None], (b - o[:, None]) / d[:, None]
    zero = np.broadcast_to((d == 0)[:, None], t1.shape)
    inside = (o[:, None] >= a) & (o[:, None] <= b)
    tn = np.where(zero, np.where(inside, -np.inf, np.inf), np.minimum(t1, t2)).max(2)
    tf = np.where(zero, np.where(inside, np.inf, -np.inf), np.maximum(t1, t2)).min(2)
    tn = np.maximum(tn, tmin[:, None])
    in_plane = (zero & (lo == hi)).any(2) | (zero & (sc * 255 < 1e-30)).any(2)
    return (tn <= tf) & (tn < tmax[:, None]) & ~in_plane


def cases(g, n, mode):
    ext = np.exp(g.uniform(np.log(1e-4), np.log(30), (n, 1))) * np.exp(g.normal(0, 0.7, (n, 3)))
    if mode == "flat":
        ext[np.arange(n), g.integers(0, 3, n)] = np.where(g.random(n) < 0.5, 0, 1e-7)
    e = np.maximum(np.where(ext > 0, np.ceil(np.log2(np.maximum(ext, 1e-300) / 255)), -126).astype(int), -126)
    p = g.uniform(-3, 3, (n, 3)).astype(f32)
    top = np.minimum(255, np.floor(ext / np.ldexp(1.0, e))).astype(int)[:, None]
    lo = np.minimum(g.integers(0, 256, (n, 8, 3)), top)
    hi = np.minimum(np.minimum(255, lo + g.integers(0, 90, (n, 8, 3))), np.maximum(top, lo))
    aim = p + g.random((n, 3)) * ext
    if mode == "inside":
        o = (p + g.random((n, 3)) * ext).astype(f32)
    else:
        o = (aim + g.normal(size=(n, 3)) * np.exp(g.uniform(np.log(1e-4), np.log(100), (n, 1)))).astype(f32)
    d = aim - o
    if mode == "axis":
        d[np.arange(n), g.integers(0, 3, n)] *= 10.0 ** g.uniform(-9, -1, n)
        z = g.random(n) < 0.5
        d[np.arange(n)[z], g.integers(0, 3, n)[z]] = 0
    d = (d / np.maximum(np.linalg.norm(d, axis=1, keepdims=True), 1e-30)).astype(f32)
    tmax = np.where(g.random(n) < 0.3, g.uniform(0, 5, n), 3.4e38).astype(f32)
    return p, e, lo, hi, o, d, np.full(n, 1e-4, f32), tmax


@pytest.mark.parametrize("mode", ["any", "inside", "axis", "flat"])
def test_half_precision_boxes_report_every_box_met(mode):
    g = np.random.default_rng(17)
    met = extra = 0
    for _ in range(2):
        c = cases(g, 25000, mode)
        ok = np.abs(c[5]).max(1) > 0
        h, x = half_boxes(*c)[ok], exact_boxes(*c)[ok]
        assert not (x & ~h).any()
        met, extra = met + x.sum(), extra + (h & ~x).sum()
    assert met > 500
    print(f"{mode}: {met} met, {extra} reported beyond them")


def test_distances_beyond_range_report_every_child():
    g = np.random.default_rng(3)
    p, e, lo, hi, o, d, tmin, tmax = cases(g, 64, "any")
    e[:] = 120  # boxes as large as the float range
    assert half_boxes(p, e, lo, hi, o, d, tmin, tmax).all()
