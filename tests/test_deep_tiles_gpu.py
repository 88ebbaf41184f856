"""Tiles of many overlapping records whose draws change state in between:
depth tests that hide whole records, unblended fragments replaced before
they are seen, draws that raise depths or blend in the middle, points and
lines among them -- against the oracle, bit for bit, with the fragment
count."""
import ctypes as C

import numpy as np
import pytest

from pixelforge_gb300 import abi as A
from pixelforge_gb300.scenes import Target, _ptr

pytestmark = pytest.mark.gpu

# per scene: the depth functions (-1: no test), blend modes (-1: off) and depth masks its draws choose from
SCENES = {
    "less_opaque": ([A.PF_LESS], [-1], [True]),
    "less_blended": ([A.PF_LESS], [-1, A.PF_BLEND_ALPHA, A.PF_BLEND_ADD], [True]),
    "lequal": ([A.PF_LEQUAL], [-1, A.PF_BLEND_MUL], [True, False]),
    "raised": ([A.PF_LESS, A.PF_GREATER, -1, A.PF_LEQUAL], [-1, A.PF_BLEND_ALPHA], [True, False]),
    "equal": ([A.PF_LESS, A.PF_EQUAL, A.PF_NOTEQUAL, A.PF_GEQUAL], [-1, A.PF_BLEND_SCREEN], [True]),
}


def _scene(lib, name, phong, perspective, w, h, fmt):
    r = np.random.default_rng(sum(map(ord, name)) + 2 * phong + perspective)
    funcs, blends, masks = SCENES[name]
    tg = Target(lib, w, h, "fbo", fmt=fmt)
    keep = []
    try:
        lib.pfClearFramebuffer(tg._fbref, A.PFcolor(9, 8, 7, 255), 1e30 if perspective else 1.0)
        if perspective:
            lib.pfMatrixMode(A.PF_PROJECTION)
            lib.pfLoadIdentity()
            lib.pfFrustum(-0.1, 0.1, -0.1, 0.1, 0.1, 10.0)
            lib.pfMatrixMode(A.PF_MODELVIEW)
            lib.pfLoadIdentity()
            lib.pfTranslatef(0.0, 0.0, -2.0)
        if phong:
            lib.pfEnable(A.PF_LIGHTING)
            lib.pfLightModel(A.PF_PHONG)
            for i in range(2):
                lib.pfEnableLight(i)
                p = np.array([2.0 - 4 * i, 1.5, 3.0], np.float32)
                lib.pfLightfv(i, A.PF_POSITION, _ptr(p))
        tex = r.integers(0, 256, (16, 16, 4), dtype=np.uint8)
        th = lib.pfGenTexture(_ptr(tex), 16, 16, A.PF_RGBA, A.PF_UNSIGNED_BYTE)
        lib.pfTextureParameter(th, A.PF_REPEAT, A.PF_NEAREST)
        lib.pfBindTexture(th)
        lib.pfEnable(A.PF_VERTEX_ARRAY | A.PF_COLOR_ARRAY | A.PF_NORMAL_ARRAY | A.PF_TEXTURE_COORD_ARRAY)
        lib.pfDisable(A.PF_CULL_FACE)
        for k in range(14):
            f, b, m = (int(r.choice(funcs)), int(r.choice(blends)), bool(r.choice(masks)))
            (lib.pfEnable if f >= 0 else lib.pfDisable)(A.PF_DEPTH_TEST)
            if f >= 0:
                lib.pfDepthFunc(f)
            (lib.pfEnable if b >= 0 else lib.pfDisable)(A.PF_BLEND)
            if b >= 0:
                lib.pfBlendFunc(b)
            lib.pfDepthMask(m)
            (lib.pfEnable if r.random() < 0.5 else lib.pfDisable)(A.PF_TEXTURE_2D)
            # nearly flat layers (hidden whole tiles at a time), slanted ones, small ones
            n = int(r.integers(5, 50))
            size = r.choice([0.3, 1.0, 3.0], (n, 1, 1))
            pos = r.uniform(-0.8, 0.8, (n, 1, 3)) + r.uniform(-1, 1, (n, 3, 3)) * size
            z = r.uniform(0.1, 0.9, (n, 1)) + r.choice([0.0, 0.01, 0.3], (n, 1)) * r.uniform(-1, 1, (n, 3))
            pos[:, :, 2] = np.clip(z, 0.05, 0.95)
            arr = [np.ascontiguousarray(pos.reshape(-1, 3), np.float32), r.integers(0, 256, (3 * n, 4), dtype=np.uint8),
                   r.normal(size=(3 * n, 3)).astype(np.float32), r.uniform(0.0, 1.9, (3 * n, 2)).astype(np.float32)]
            keep.append(arr)
            lib.pfVertexPointer(3, A.PF_FLOAT, 0, _ptr(arr[0]))
            lib.pfColorPointer(4, A.PF_UNSIGNED_BYTE, 0, _ptr(arr[1]))
            lib.pfNormalPointer(A.PF_FLOAT, 0, _ptr(arr[2]))
            lib.pfTexCoordPointer(A.PF_FLOAT, 0, _ptr(arr[3]))
            lib.pfDrawArrays(A.PF_TRIANGLES, 0, 3 * n)
            if k % 4 == 3 and not perspective:
                lib.pfDisable(A.PF_TEXTURE_2D)
                lib.pfDrawArrays(A.PF_POINTS if k % 8 == 3 else A.PF_LINES, 0, min(3 * n, 12))
        fr = tg.finish()
        lib.pfDeleteTexture(C.byref(C.c_void_p(th)), False)
        return fr
    finally:
        tg.close()


@pytest.mark.parametrize("fmt", [(A.PF_RGBA, A.PF_UNSIGNED_BYTE), (A.PF_RGB, A.PF_UNSIGNED_SHORT_5_6_5)])
@pytest.mark.parametrize("size", [(8, 8), (37, 21)])
@pytest.mark.parametrize("perspective", [False, True])
@pytest.mark.parametrize("phong", [False, True])
@pytest.mark.parametrize("name", list(SCENES))
def test_deep_tiles_vs_oracle(gpu, oracle, name, phong, perspective, size, fmt):
    a = _scene(gpu, name, phong, perspective, *size, fmt)
    b = _scene(oracle, name, phong, perspective, *size, fmt)
    assert np.array_equal(a.depth.view(np.uint32), b.depth.view(np.uint32))
    assert np.array_equal(a.color, b.color)
    if "fragments" in b.stats:
        assert a.stats["fragments"] == b.stats["fragments"]
    assert gpu.pfGetDeviceStatus() == 0
