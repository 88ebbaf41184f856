"""pfClear keeps pixels 0..7 (context.c:680-745): the caller's values of them,
as they are at each flush, for every pixel size, main buffers and framebuffer
objects, with a draw over them, against the oracle, byte for byte."""
import numpy as np
import pytest

from pixelforge_gb300 import abi as A
from pixelforge_gb300.scenes import Target, _ptr

pytestmark = pytest.mark.gpu

FORMATS = {"rgba8": (A.PF_RGBA, A.PF_UNSIGNED_BYTE), "rgb8": (A.PF_RGB, A.PF_UNSIGNED_BYTE),
           "rgb565": (A.PF_RGB, A.PF_UNSIGNED_SHORT_5_6_5), "rgba16f": (A.PF_RGBA, A.PF_HALF_FLOAT),
           "rgba32f": (A.PF_RGBA, A.PF_FLOAT), "bgra8": (A.PF_BGRA, A.PF_UNSIGNED_BYTE)}


def _frames(lib, kind, fmt, w, h):
    r = np.random.default_rng(w * h)
    tg = Target(lib, w, h, kind, fmt=fmt)
    out = []
    try:
        pos = np.array([(-1, 1, 0.5), (-1, 0.2, 0.5), (0.6, 1, 0.5), (0.9, -1, 0.3), (0.9, 1, 0.3), (-0.2, 1, 0.3)], np.float32)
        col = r.integers(0, 256, (6, 4), dtype=np.uint8)
        lib.pfEnable(A.PF_DEPTH_TEST)
        lib.pfDepthFunc(A.PF_LEQUAL)
        lib.pfDisable(A.PF_CULL_FACE)
        lib.pfEnable(A.PF_VERTEX_ARRAY | A.PF_COLOR_ARRAY)
        lib.pfVertexPointer(3, A.PF_FLOAT, 0, _ptr(pos))
        lib.pfColorPointer(4, A.PF_UNSIGNED_BYTE, 0, _ptr(col))
        for frame in range(4):
            if kind == "main":      # the caller's own bytes, changed between frames (finite halves and floats)
                if fmt[1] == A.PF_HALF_FLOAT:
                    tg.main.reshape(-1, tg.bpp)[:8].view(np.float16)[...] = r.uniform(0, 1, (8, tg.bpp // 2))
                elif fmt[1] == A.PF_FLOAT:
                    tg.main.reshape(-1, tg.bpp)[:8].view(np.float32)[...] = r.uniform(0, 1, (8, tg.bpp // 4))
                else:
                    tg.main.reshape(-1, tg.bpp)[:8] = r.integers(0, 256, (8, tg.bpp))
            lib.pfClearColor(10 * frame, 20, 30, 255)
            lib.pfClearDepth(1.0)
            lib.pfClear(A.PF_COLOR_BUFFER_BIT | A.PF_DEPTH_BUFFER_BIT)
            if frame % 2:
                lib.pfEnable(A.PF_BLEND)
                lib.pfBlendFunc(A.PF_BLEND_AVERAGE)
            else:
                lib.pfDisable(A.PF_BLEND)
            if frame != 2:          # (a clear alone in the third)
                lib.pfDrawArrays(A.PF_TRIANGLES, 0, 6)
            if frame == 3:          # two clears and draws of one flush
                lib.pfClear(A.PF_COLOR_BUFFER_BIT | A.PF_DEPTH_BUFFER_BIT)
                lib.pfDrawArrays(A.PF_TRIANGLES, 3, 3)
            fr = tg.finish()
            out.append((fr.color, fr.depth))
        return out
    finally:
        tg.close()


@pytest.mark.parametrize("w,h", [(8, 1), (16, 5), (40, 24)])
@pytest.mark.parametrize("kind", ["main", "fbo"])
@pytest.mark.parametrize("fmt", list(FORMATS))
def test_kept_pixels_vs_oracle(gpu, oracle, fmt, kind, w, h):
    a, b = _frames(gpu, kind, FORMATS[fmt], w, h), _frames(oracle, kind, FORMATS[fmt], w, h)
    for (ca, da), (cb, db) in zip(a, b):
        assert np.array_equal(ca, cb)
        assert da is None or np.array_equal(da.view(np.uint32), db.view(np.uint32))
    assert gpu.pfGetDeviceStatus() == 0
