"""Triangles whose edge functions leave 32 bits: two of them are exactly
-2^31 at the origin of a tile and the third is positive on all of it, so that
the wrapped values, not the geometry, decide each pixel -- against the oracle,
bit for bit, with the fragment count."""
import numpy as np
import pytest

from pixelforge_gb300 import abi as A
from pixelforge_gb300.scenes import Target, _ptr

pytestmark = pytest.mark.gpu

W = H = 129
# corners relative to the tile's origin
CORNERS = {"front": ((32768, -100), (-32768, -100), (0, 65536)),
           "back": ((512, 512), (0, 512), (-4194304, -8388608))}


def _ndc(pixel, flip):
    """A coordinate that projects exactly onto a pixel (a viewport of 129)."""
    want, one, half = np.float32(pixel), np.float32(1), np.float32(0.5)
    h = np.float32((pixel - 0.5) / 64.0 - 1.0)
    h = -h if flip else h
    for c in [h, *(np.nextafter(h, np.float32(s) * np.float32(np.inf), dtype=np.float32) for s in (-1, 1))]:
        t = (one - c) if flip else (c + one)
        if np.trunc(t * half * np.float32(128) + half) == want:
            return c
    raise AssertionError(pixel)


def _edges(corners, x, y):
    """The three edge functions at a pixel in 64 bits and wrapped to 32."""
    (x1, y1), (x2, y2), (x3, y3) = corners
    area = ((x2 - x1) * (y3 - y1) - (x3 - x1) * (y2 - y1) + 2**31) % 2**32 - 2**31
    s = 1 if area < 0 else -1
    w = [s * ((x - px) * (qy - py) + (y - py) * (px - qx)) for (px, py), (qx, qy) in
         (((x2, y2), (x3, y3)), ((x3, y3), (x1, y1)), ((x1, y1), (x2, y2)))]
    return [(v + 2**31) % 2**32 - 2**31 for v in w]


def _scene(lib, corners, fmt):
    r = np.random.default_rng(5)
    tg = Target(lib, W, H, "fbo", fmt=fmt)
    try:
        lib.pfClearFramebuffer(tg._fbref, A.PFcolor(9, 8, 7, 255), 1.0)
        lib.pfDisable(A.PF_CULL_FACE)
        lib.pfShadeModel(A.PF_FLAT)
        lib.pfEnable(A.PF_VERTEX_ARRAY | A.PF_COLOR_ARRAY)
        pos = np.array([(_ndc(x, False), _ndc(y, True), 0.5) for x, y in corners], np.float32)
        col = r.integers(0, 256, (3, 4), dtype=np.uint8)
        lib.pfVertexPointer(3, A.PF_FLOAT, 0, _ptr(pos))
        lib.pfColorPointer(4, A.PF_UNSIGNED_BYTE, 0, _ptr(col))
        lib.pfDrawArrays(A.PF_TRIANGLES, 0, 3)
        return tg.finish()
    finally:
        tg.close()


@pytest.mark.parametrize("fmt", [(A.PF_RGBA, A.PF_UNSIGNED_BYTE), (A.PF_RGB, A.PF_UNSIGNED_SHORT_5_6_5)])
@pytest.mark.parametrize("tile", [(0, 0), (8, 8), (64, 24)])
@pytest.mark.parametrize("face", list(CORNERS))
def test_lowest_edge_value_vs_oracle(gpu, oracle, face, tile, fmt):
    corners = [(x + tile[0], y + tile[1]) for x, y in CORNERS[face]]
    assert sorted(_edges(corners, *tile))[:2] == [-2**31, -2**31]
    got, ref = _scene(gpu, corners, fmt), _scene(oracle, corners, fmt)
    assert np.array_equal(got.color, ref.color)
    assert np.array_equal(got.depth.view(np.uint32), ref.depth.view(np.uint32))
    if "fragments" in ref.stats:
        assert got.stats["fragments"] == ref.stats["fragments"]
    assert gpu.pfGetDeviceStatus() == 0
