"""Draws of one flush over the same vertex arrays: with what k_vertex reads
unchanged between them (blend, depth, texture and shading state, other
indices) and changed (matrix, lights, materials, current colour, arrays, a
longer index range), against the oracle.  Lighting is per fragment or off:
bit for bit."""
import ctypes as C

import numpy as np
import pytest

from pixelforge_gb300 import abi as A
from pixelforge_gb300.scenes import Target, _ptr

pytestmark = pytest.mark.gpu


def _render(lib, seed, phong):
    r = np.random.default_rng(seed)
    tg = Target(lib, 72, 56, "fbo")
    n = 60
    pos = r.uniform(-1.2, 1.2, (n, 3)).astype(np.float32)
    other = r.uniform(-1.2, 1.2, (n, 3)).astype(np.float32)
    nrm = r.normal(size=(n, 3)).astype(np.float32)
    uv = r.uniform(0.01, 1.9, (n, 2)).astype(np.float32)
    col = r.integers(0, 256, (n, 4), dtype=np.uint8)
    tex = r.integers(0, 256, (8, 8, 4), dtype=np.uint8)
    idx = [r.integers(0, k, 90).astype(np.uint32) for k in (n // 2, n, n, n // 3, n, n, n, n)]
    try:
        lib.pfClearFramebuffer(tg._fbref, A.PFcolor(5, 6, 7, 255), 1e30)
        lib.pfMatrixMode(A.PF_PROJECTION)
        lib.pfLoadIdentity()
        lib.pfFrustum(-0.1, 0.1, -0.1, 0.1, 0.1, 10.0)
        lib.pfMatrixMode(A.PF_MODELVIEW)
        lib.pfLoadIdentity()
        lib.pfTranslatef(0.0, 0.0, -3.0)
        lib.pfEnable(A.PF_DEPTH_TEST)
        lib.pfDepthFunc(A.PF_LESS)
        lib.pfDisable(A.PF_CULL_FACE)
        th = lib.pfGenTexture(_ptr(tex), 8, 8, A.PF_RGBA, A.PF_UNSIGNED_BYTE)
        lib.pfTextureParameter(th, A.PF_REPEAT, A.PF_NEAREST)
        lib.pfBindTexture(th)
        if phong:
            lib.pfEnable(A.PF_LIGHTING)
            lib.pfLightModel(A.PF_PHONG)
            lib.pfEnableLight(0)
            lib.pfLightfv(0, A.PF_POSITION, _ptr(np.array([2.0, 1.0, 3.0], np.float32)))
        lib.pfEnable(A.PF_VERTEX_ARRAY | A.PF_NORMAL_ARRAY | A.PF_TEXTURE_COORD_ARRAY)
        lib.pfVertexPointer(3, A.PF_FLOAT, 0, _ptr(pos))
        lib.pfNormalPointer(A.PF_FLOAT, 0, _ptr(nrm))
        lib.pfTexCoordPointer(A.PF_FLOAT, 0, _ptr(uv))
        lib.pfColorPointer(4, A.PF_UNSIGNED_BYTE, 0, _ptr(col))
        keep = []

        def draw(k):
            lib.pfDrawElements(A.PF_TRIANGLES, 90, A.PF_UNSIGNED_INT, _ptr(idx[k]))
        steps = [lambda: None, lambda: (lib.pfEnable(A.PF_BLEND), lib.pfBlendFunc(A.PF_BLEND_ADD)),
                 lambda: lib.pfEnable(A.PF_TEXTURE_2D), lambda: lib.pfShadeModel(A.PF_FLAT),
                 lambda: lib.pfColor4ub(10, 200, 30, 128), lambda: lib.pfTranslatef(0.1, -0.05, 0.2),
                 lambda: (lib.pfEnable(A.PF_COLOR_ARRAY), lib.pfDepthFunc(A.PF_GREATER)),
                 lambda: lib.pfMaterialfv(A.PF_FRONT_AND_BACK, A.PF_DIFFUSE,
                                          keep.append(np.array([0.9, 0.2, 0.4, 1.0], np.float32)) or _ptr(keep[-1])),
                 lambda: lib.pfVertexPointer(3, A.PF_FLOAT, 0, _ptr(other)),
                 lambda: lib.pfVertexPointer(3, A.PF_FLOAT, 0, _ptr(pos))]
        for i in r.permutation(len(steps)):
            steps[i]()
            draw(int(r.integers(len(idx))))
            draw(int(r.integers(len(idx))))
        fr = tg.finish()
        lib.pfDeleteTexture(C.byref(C.c_void_p(th)), False)
        return fr
    finally:
        tg.close()


@pytest.mark.parametrize("phong", [False, True])
@pytest.mark.parametrize("seed", range(6))
def test_passes_over_one_mesh_vs_oracle(gpu, oracle, seed, phong):
    a, b = _render(gpu, seed, phong), _render(oracle, seed, phong)
    assert np.array_equal(a.depth.view(np.uint32), b.depth.view(np.uint32))
    assert np.array_equal(a.color, b.color)
    assert gpu.pfGetDeviceStatus() == 0
