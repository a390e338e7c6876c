"""The quads of the guiding network's dense grid levels (rt_guide.cu,
k_guide_quads): every cell's four corners of a plane, bit for bit the table's
entries, for the resolutions of several finest levels, the hashed levels left
out.  The functions are internal and called by their C++ symbols.
"""
import ctypes as C

import numpy as np
import pytest

import optixrender_b200 as rt

LEVELS, T = 16, 1 << 19


class _NetView(C.Structure):  # rtg::NetView
    _fields_ = [("table", C.c_void_p), ("mlp", C.c_void_p), ("lo", C.c_float * 3), ("inv_ext", C.c_float * 3),
                ("res", C.c_int * LEVELS), ("kappa_hi", C.c_float), ("quads", C.c_void_p),
                ("quad_off", C.c_uint32 * LEVELS)]


@pytest.mark.gpu
@pytest.mark.parametrize("finest", [2, 16, 17, 64, 79, 80, 300])
def test_quads_hold_the_tables_corners(finest):
    torch = pytest.importorskip("torch")
    lib = rt.load_library()
    layout, launch = lib._ZN4rtgh11quad_layoutERN3rtg7NetViewE, lib._ZN4rtgh12launch_quadsERKN3rtg7NetViewEiP11CUstream_st
    layout.restype, launch.restype = C.c_size_t, None
    g = np.random.default_rng(finest)
    table = g.integers(0, 1 << 32, (LEVELS, T), dtype=np.uint64).astype(np.uint32)
    d = torch.from_numpy(table.view(np.int32)).cuda()
    v = _NetView()
    v.table = d.data_ptr()
    lo = min(16, finest)
    for l in range(LEVELS):
        v.res[l] = int(np.floor(lo * (finest / lo) ** (l / (LEVELS - 1)) + 1e-6))
    size = layout(C.byref(v))
    q = torch.full((max(1, size // 4) + 4,), -7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    v.quads = q.data_ptr()
    launch(C.byref(v), C.c_int(148), None)
    torch.cuda.synchronize()
    got = q.cpu().numpy().view(np.uint32)
    assert (got[size // 4:].view(np.int32) == -7).all()  # nothing past the end
    at = 0
    for l in range(LEVELS):
        r = v.res[l]
        if (r + 1) ** 3 > T:
            assert v.quad_off[l] == 0xFFFFFFFF
            continue
        assert v.quad_off[l] == at
        n = r * r * (r + 1)
        t = table[l, :(r + 1) ** 3].reshape(r + 1, r + 1, r + 1)  # z, y, x
        want = np.stack([t[:, :-1, :-1], t[:, :-1, 1:], t[:, 1:, :-1], t[:, 1:, 1:]], -1).reshape(n, 4)
        assert np.array_equal(got[4 * at:4 * (at + n)].reshape(n, 4), want)
        at += n
    assert size == 16 * at
