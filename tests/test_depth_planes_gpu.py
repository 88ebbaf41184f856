"""Fragments counted at set-up and records dropped by their depth planes:
triangles around the sizes where the counting and the bound change, with
horizontal and vertical edges, cut by the framebuffer's edges and not, in
launches of few and of many triangles a tile, with depths of either sign --
against the oracle, bit for bit, with the fragment count."""
import numpy as np
import pytest

from pixelforge_gb300 import abi as A
from pixelforge_gb300.scenes import Target, _ptr

pytestmark = pytest.mark.gpu


def _scene(lib, side, n, sign, fmt):
    r = np.random.default_rng(1000 * side + n + (sign > 0))
    w, h = 149, 77
    tg = Target(lib, w, h, "fbo", fmt=fmt)
    try:
        lib.pfClearFramebuffer(tg._fbref, A.PFcolor(9, 8, 7, 255), 1e30)
        lib.pfEnable(A.PF_DEPTH_TEST | A.PF_VERTEX_ARRAY | A.PF_COLOR_ARRAY)
        lib.pfDepthFunc(A.PF_LESS if n % 2 else A.PF_LEQUAL)
        lib.pfDisable(A.PF_CULL_FACE)
        # corners in pixels from a first one anywhere, some outside the framebuffer
        px = r.integers(-6, [w + 6, h + 6], (n, 1, 2)) + r.integers(-side, side + 1, (n, 3, 2))
        flat = r.random(n)
        px[flat < 0.25, 1, 1] = px[flat < 0.25, 0, 1]                    # a horizontal edge
        px[flat > 0.75, 2, 0] = px[flat > 0.75, 1, 0]                    # a vertical one
        z = sign * (r.uniform(0.2, 0.9, (n, 1)) + r.choice([0.0, 0.09], (n, 1)) * r.uniform(-1, 1, (n, 3)))
        pos = np.empty((n, 3, 3), np.float32)
        pos[:, :, 0] = 2.0 * (px[:, :, 0] + 0.25) / (w - 1) - 1.0
        pos[:, :, 1] = 1.0 - 2.0 * (px[:, :, 1] + 0.25) / (h - 1)
        pos[:, :, 2] = z
        pos = np.ascontiguousarray(pos.reshape(-1, 3))
        col = r.integers(0, 256, (3 * n, 4), dtype=np.uint8)
        lib.pfVertexPointer(3, A.PF_FLOAT, 0, _ptr(pos))
        lib.pfColorPointer(4, A.PF_UNSIGNED_BYTE, 0, _ptr(col))
        lib.pfDrawArrays(A.PF_TRIANGLES, 0, 3 * n)
        return tg.finish()
    finally:
        tg.close()


@pytest.mark.parametrize("fmt", [(A.PF_RGBA, A.PF_UNSIGNED_BYTE), (A.PF_BGRA, A.PF_UNSIGNED_BYTE)])
@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("side,n", [(2, 60), (2, 2500), (4, 2500), (5, 300), (16, 300), (17, 301), (16, 1501), (90, 37), (90, 700)])
def test_counted_and_dropped(gpu, oracle, side, n, sign, fmt):
    got, ref = _scene(gpu, side, n, sign, fmt), _scene(oracle, side, n, sign, fmt)
    assert np.array_equal(got.depth.view(np.uint32), ref.depth.view(np.uint32))
    assert np.array_equal(got.color, ref.color)
    if "fragments" in ref.stats:
        assert got.stats["fragments"] == ref.stats["fragments"]
        assert ref.stats["fragments"] > 100
    assert gpu.pfGetDeviceStatus() == 0
