"""What the scene upload computes on the device: the environment's sampling
cache, equal bit for bit to the host table, and the checks of a device-built
wide BVH, which accept the build and refuse damaged ones.

The functions under test are internal, so they are called by their C++ symbols.
"""
import ctypes as C
import glob
import os

import numpy as np
import pytest

import optixrender_b200 as rt
from optixrender_b200 import scenes


def _image(kind, w, h):
    g = np.random.default_rng(w * 1000 + h)
    img = np.exp(g.normal(0, 3, (h, w, 4))).astype(np.float32)
    if kind == "black-columns":      # their conditional sums are 0 / 0
        img[:, g.random(w) < 0.4] = 0
    elif kind == "black":            # every value is 0 / 0
        img[:] = 0
    elif kind == "one-pixel":
        img[:] = 0
        img[h // 2, w // 3] = 5000
    elif kind == "tiny":             # denormal densities
        img *= np.float32(1e-38)
        img[0, 0] = 1e5
    elif kind == "not-numbers":
        img[h // 2, w // 2] = np.nan
        img[0, w - 1] = np.inf
    return img


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["plain", "black-columns", "black", "one-pixel", "tiny", "not-numbers"])
@pytest.mark.parametrize("size", [(1, 1), (2, 1), (1, 7), (33, 17), (256, 128), (517, 300)])
def test_device_environment_cache_equals_host_cache(kind, size):
    torch = pytest.importorskip("torch")
    lib = rt.load_library()
    f = lib._ZN3rth25env_sampling_cache_deviceEPK6float4iifPS0_P11CUstream_st
    f.restype, f.argtypes = C.c_int, [C.c_void_p, C.c_int, C.c_int, C.c_float, C.c_void_p, C.c_void_p]
    lum = lib._ZN3rth17env_luminance_sumEPKfii
    lum.restype, lum.argtypes = C.c_float, [C.c_void_p, C.c_int, C.c_int]
    w, h = size
    img = _image(kind, w, h)
    want = rt.env_sampling_cache(img)
    d = torch.from_numpy(img).cuda()
    out = torch.empty_like(d)
    torch.cuda.synchronize()
    assert f(d.data_ptr(), w, h, lum(img.ctypes.data, w, h), out.data_ptr(), None) == 0
    got = out.cpu().numpy()
    nan = np.isnan(want)
    assert np.array_equal(nan, np.isnan(got))
    assert np.array_equal(got.view(np.int32)[~nan], want.view(np.int32)[~nan])


class _DeviceBvh(C.Structure):  # rth::DeviceBvh
    _fields_ = [("nodes", C.c_void_p), ("nodes_bytes", C.c_size_t), ("order", C.c_void_p), ("order_bytes", C.c_size_t),
                ("levels", C.POINTER(C.c_int) * 3), ("num_nodes", C.c_int), ("depth", C.c_int)]


class _String(C.Structure):  # an empty std::string
    _fields_ = [("ptr", C.c_void_p), ("size", C.c_size_t), ("local", C.c_char * 16)]


@pytest.mark.gpu
def test_device_check_accepts_the_build_and_refuses_damage():
    torch = pytest.importorskip("torch")
    lib = rt.load_library()
    build = lib._ZN3rth18build_cwbvh_deviceEPKflRNS_9DeviceBvhERNSt7__cxx1112basic_stringIcSt11char_traitsIcESaIcEEEP11CUstream_st
    check = lib._ZN3rth18check_cwbvh_deviceERKNS_9DeviceBvhEPKflRbRNSt7__cxx1112basic_stringIcSt11char_traitsIcESaIcEEEP11CUstream_st
    build.restype = check.restype = C.c_bool
    cudart = C.CDLL(glob.glob(os.path.join(os.path.dirname(torch.__file__), "..", "nvidia", "cuda_runtime", "lib", "libcudart.so*"))[0])
    spec = scenes.spheres(ico_level=3, sphere_tris=False, env_size=(16, 8))
    tri = np.concatenate([m.triangles() for m in spec.meshes]).astype(np.float32)
    n = len(tri)
    d_tv = torch.from_numpy(tri.reshape(-1)).cuda()
    torch.cuda.synchronize()
    b, err = _DeviceBvh(), _String()
    err.ptr = C.addressof(err) + 16
    assert build(C.c_void_p(d_tv.data_ptr()), C.c_int64(n), C.byref(b), C.byref(err), None)
    nodes = np.empty(b.num_nodes * 80, np.uint8)
    order = np.empty(n, np.int32)
    for dst, src in ((nodes, b.nodes), (order, b.order)):
        assert cudart.cudaMemcpy(C.c_void_p(dst.ctypes.data), C.c_void_p(src), C.c_size_t(dst.nbytes), C.c_int(2)) == 0

    def valid(nd, od):
        tn, to = torch.from_numpy(nd).cuda(), torch.from_numpy(od).cuda()
        torch.cuda.synchronize()
        c = _DeviceBvh.from_buffer_copy(b)
        c.nodes, c.order = tn.data_ptr(), to.data_ptr()
        ok = C.c_bool(True)
        assert check(C.byref(c), C.c_void_p(d_tv.data_ptr()), C.c_int64(n), C.byref(ok), C.byref(err), None)
        return ok.value

    assert b.num_nodes > 500 and b.depth > 3
    assert valid(nodes, order)
    g = np.random.default_rng(1)
    rec = nodes.reshape(-1, 80)
    for i in [0, b.num_nodes // 2, b.num_nodes - 1] + list(g.integers(0, b.num_nodes, 5)):
        used = np.flatnonzero(rec[i, 24:32])
        s = int(used[0])
        inner = (rec[i, 15] >> s) & 1
        for what in ("box", "children", "triangles", "meta", "mask"):
            bad = rec.copy()
            if what == "box":        # the slot's x planes: an empty box at the origin
                if not bad[i, 32 + 2 * s:34 + 2 * s].any():
                    continue
                bad[i, 32 + 2 * s:34 + 2 * s] = 0
            elif what == "children":
                if not rec[i, 15]:
                    continue
                bad[i, 16:20] = np.frombuffer(np.uint32(b.num_nodes - 1).tobytes(), np.uint8)
            elif what == "triangles":
                if not any(not (rec[i, 15] >> k) & 1 for k in used):
                    continue
                bad[i, 20:24] = np.frombuffer(np.uint32(n).tobytes(), np.uint8)
            elif what == "meta":
                bad[i, 24 + s] = 0 if inner else 0x5F  # an inner slot without meta, a leaf of no known mask
            else:
                bad[i, 15] ^= np.uint8(1 << s)
            assert not valid(bad.reshape(-1), order), (i, what)
    twice = order.copy()
    twice[5] = twice[6]
    assert not valid(nodes, twice)
    beyond = order.copy()
    beyond[7] = n
    assert not valid(nodes, beyond)
