"""Copies of one PFframebuffer name the same pixels: what is drawn through one
is there for a pfClear through the other, which keeps pixels 0..7 as they are
at that moment (context.c:680-745), in one flush, against the oracle, byte for
byte."""
import ctypes as C

import numpy as np
import pytest

from pixelforge_gb300 import abi as A
from pixelforge_gb300.scenes import Target, _ptr

pytestmark = pytest.mark.gpu

FORMATS = {"rgba8": (A.PF_RGBA, A.PF_UNSIGNED_BYTE), "rgba16f": (A.PF_RGBA, A.PF_HALF_FLOAT),
           "bgra8": (A.PF_BGRA, A.PF_UNSIGNED_BYTE)}


def _render(lib, fmt, first):
    tg = Target(lib, 24, 16, "fbo", fmt=FORMATS[fmt])
    copy = A.PFframebuffer()
    C.memmove(C.byref(copy), C.byref(tg.fb), C.sizeof(copy))
    pos = np.array([(-1.2, 1.5, 0.5), (-1.2, 0.1, 0.5), (0.1, 1.5, 0.5), (0.9, -1, 0.3), (0.9, 1, 0.3), (-0.2, 1, 0.3)], np.float32)
    col = np.random.default_rng(3).integers(0, 256, (6, 4), dtype=np.uint8)
    try:
        lib.pfDisable(A.PF_CULL_FACE)
        lib.pfEnable(A.PF_DEPTH_TEST | A.PF_VERTEX_ARRAY | A.PF_COLOR_ARRAY)
        lib.pfDepthFunc(A.PF_LEQUAL)
        lib.pfVertexPointer(3, A.PF_FLOAT, 0, _ptr(pos))
        lib.pfColorPointer(4, A.PF_UNSIGNED_BYTE, 0, _ptr(col))
        lib.pfClearFramebuffer(tg._fbref, A.PFcolor(200, 90, 30, 255), 0.8)
        if first == "draw":
            lib.pfDrawArrays(A.PF_TRIANGLES, 0, 3)
            lib.pfClearFramebuffer(tg._fbref, A.PFcolor(7, 8, 9, 255), 0.9)
        lib.pfBindFramebuffer(C.byref(copy))
        lib.pfClearColor(10, 20, 30, 255)
        lib.pfClearDepth(1.0)
        lib.pfClear(A.PF_COLOR_BUFFER_BIT | A.PF_DEPTH_BUFFER_BIT)
        lib.pfEnable(A.PF_BLEND)
        lib.pfBlendFunc(A.PF_BLEND_AVERAGE)
        lib.pfDrawArrays(A.PF_TRIANGLES, 3, 3)
        fr = tg.finish()
        lib.pfBindFramebuffer(tg._fbref)
        return fr
    finally:
        tg.close()


@pytest.mark.parametrize("first", ["clear", "draw"])
@pytest.mark.parametrize("fmt", list(FORMATS))
def test_kept_pixels_of_a_copy_vs_oracle(gpu, oracle, fmt, first):
    a, b = _render(gpu, fmt, first), _render(oracle, fmt, first)
    assert np.array_equal(a.color, b.color)
    assert np.array_equal(a.depth.view(np.uint32), b.depth.view(np.uint32))
    assert gpu.pfGetDeviceStatus() == 0
