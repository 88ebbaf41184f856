"""k_items' binning: launches of one item to several items a warp, triangles
from a pixel to many tile rows, in one framebuffer and over several, against
the oracle (depth and smooth-shaded colour bit-exact: nothing here reaches
powf)."""
import ctypes as C

import numpy as np
import pytest

from pixelforge_gb300 import abi as A
from pixelforge_gb300.scenes import Target, _ptr

pytestmark = pytest.mark.gpu


def _mixed(seed, n):
    """Points to image-wide triangles, some degenerate, some off screen, in
    runs of one size (whole warps of tiny or wide ones) and interleaved."""
    r = np.random.default_rng(seed)
    size = np.where(r.random(n) < 0.5, r.choice([0.004, 0.03, 0.2, 1.0, 2.5], n), np.repeat([0.01, 1.5], (n + 1) // 2)[:n])
    pos = r.uniform(-1.05, 1.05, (n, 1, 3)) + r.uniform(-1, 1, (n, 3, 3)) * size[:, None, None]
    pos[:, :, 2] = r.uniform(0.1, 0.9, (n, 3))
    pos[r.random(n) < 0.03, 2] = pos[r.random(n) < 0.03, 0][:1] if n > 200 else 0.5
    return np.ascontiguousarray(pos.reshape(-1, 3), np.float32), r.integers(0, 256, (n * 3, 4), dtype=np.uint8)


def _render(lib, n, w, h, cull):
    pos, col = _mixed(100 + n, n)
    tg = Target(lib, w, h, "fbo")
    try:
        lib.pfClearFramebuffer(tg._fbref, A.PFcolor(3, 5, 7, 255), 1.0)
        lib.pfEnable(A.PF_DEPTH_TEST)
        lib.pfDepthFunc(A.PF_LESS)
        if not cull:
            lib.pfDisable(A.PF_CULL_FACE)
        lib.pfEnable(A.PF_VERTEX_ARRAY | A.PF_COLOR_ARRAY)
        lib.pfVertexPointer(3, A.PF_FLOAT, 0, _ptr(pos))
        lib.pfColorPointer(4, A.PF_UNSIGNED_BYTE, 0, _ptr(col))
        lib.pfDrawArrays(A.PF_TRIANGLES, 0, 3 * n)
        return tg.finish()
    finally:
        tg.close()


# item counts on both sides of each change of the items a warp sets up (the
# launch halves 32 while fewer than 12 warps an SM would run)
@pytest.mark.parametrize("n,w,h,cull", [
    (1, 9, 9, True), (2, 64, 64, False), (31, 200, 120, True), (33, 7, 300, True), (1823, 257, 129, True),
    (3647, 320, 200, True), (3649, 320, 200, True), (7301, 131, 77, False), (14600, 200, 201, True),
    (29300, 96, 64, True), (60000, 64, 96, True)])
def test_binning_vs_oracle(gpu, oracle, n, w, h, cull):
    a, b = _render(gpu, n, w, h, cull), _render(oracle, n, w, h, cull)
    assert np.array_equal(a.depth.view(np.uint32), b.depth.view(np.uint32))
    assert np.array_equal(a.color, b.color)
    assert gpu.pfGetDeviceStatus() == 0
    if "fragments" in b.stats:
        assert a.stats["fragments"] == b.stats["fragments"]


def test_binning_several_framebuffers_in_a_warp(gpu, oracle):
    """Triangles of framebuffers of different widths set up by one warp."""
    sizes = [(40, 300), (300, 40), (8, 8), (129, 65), (64, 64)]

    def scene(lib, batch):
        out, ctxs = [], []
        if batch:
            b = lib.pfgbBatchCreate()
            lib.pfgbBatchBegin(b)
        for k, (w, h) in enumerate(sizes):
            buf = np.zeros((h, w, 4), np.uint8)
            ctx = lib.pfCreateContext(_ptr(buf), w, h, A.PF_RGBA, A.PF_UNSIGNED_BYTE)
            lib.pfMakeCurrent(ctx)
            pos, col = _mixed(7 + k, 7)
            lib.pfClearDepth(1.0)
            lib.pfClear(A.PF_COLOR_BUFFER_BIT | A.PF_DEPTH_BUFFER_BIT)
            lib.pfEnable(A.PF_DEPTH_TEST)
            lib.pfDepthFunc(A.PF_LESS)
            lib.pfEnable(A.PF_VERTEX_ARRAY | A.PF_COLOR_ARRAY)
            lib.pfVertexPointer(3, A.PF_FLOAT, 0, _ptr(pos))
            lib.pfColorPointer(4, A.PF_UNSIGNED_BYTE, 0, _ptr(col))
            lib.pfDrawArrays(A.PF_TRIANGLES, 0, 21)
            out.append(buf)
            ctxs.append((ctx, pos, col))
        if batch:
            lib.pfgbBatchEnd(b)
            lib.pfgbBatchDelete(b)
        for ctx, _, _ in ctxs:
            lib.pfMakeCurrent(ctx)
            lib.pfDeleteContext(ctx)
        return out

    for x, y in zip(scene(gpu, True), scene(oracle, False)):
        assert np.array_equal(x, y)
