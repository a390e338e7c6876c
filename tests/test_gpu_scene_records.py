"""The triangle records that a scene upload packs on the device.  Where no mesh
brings normals (texture coordinates), the device derives the face normals
(default coordinates); where any mesh does, the host's arrays, which hold the
derived ones for the meshes without, are uploaded.  Both give the same bits:
the same triangles are rendered with a triangle out of sight that brings its
own normals, coordinates, both or neither.
"""
import numpy as np
import pytest

import optixrender_b200 as rt
from optixrender_b200 import scenes


def _render(own_normals, own_texcoords):
    g = np.random.default_rng(12)
    s = rt.Scene()
    tex = s.add_texture(g.integers(0, 256, (64, 64, 4)).astype(np.uint8))
    n = 3000
    tri = (g.uniform(-1, 1, (n, 1, 3)) + g.normal(0, 0.08, (n, 3, 3))).astype(np.float32)
    tri[::7, 2] = tri[::7, 1] + (g.normal(0, 1e-4, (len(tri[::7]), 3))).astype(np.float32)  # slivers
    s.add_mesh(tri[:1000].reshape(-1, 3), rt.material(rt.MAT_DIFFUSE, texture_ids=[tex]))
    s.add_mesh(tri[1000:].reshape(-1, 3), rt.material(rt.MAT_CONDUCTOR, roughness=0.4, texture_ids=[tex]))
    far = np.float32([[50, 50, -90], [51, 50, -90], [50, 51, -90]])
    s.add_mesh(far, rt.material(rt.MAT_DIFFUSE),
               normals=np.float32([[0.6, 0, -0.8]] * 3) if own_normals else None,
               texcoords=np.float32([[0.1, 0.2], [0.3, 0.9], [0.7, 0.5]]) if own_texcoords else None)
    s.add_env(scenes.sky(32, 16))
    # one bounce: the triangle out of sight can only cast a shadow
    r = rt.Renderer(s, rt.options(width=160, height=120, spp=4, max_depth=1, seed=3))
    r.set_camera(rt.camera(from_=(0.3, 0.4, -3.2), at=(0, 0, 0), up=(0, 1, 0)))
    r.render()
    return [r.download_linear(), r.download_aov(rt.AOV_ALBEDO), r.download_aov(rt.AOV_NORMAL)]


@pytest.mark.gpu
def test_derived_normals_and_coordinates_equal_the_hosts():
    want = _render(False, False)
    assert np.abs(want[2][..., :3]).max() > 0.5 and want[1][..., :3].std() > 0.05  # there is something to see
    for own in ((True, False), (False, True), (True, True)):
        for a, b in zip(_render(*own), want):
            assert np.array_equal(a.view(np.int32), b.view(np.int32)), own
