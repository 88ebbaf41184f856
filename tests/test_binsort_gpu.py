"""k_binsort's item maps: bins of 128 entries to thousands, items of a launch
on both sides of the maps' sizes (2,048, 4,096 ... 65,536 and above, where
bins are merge-sorted), several targets, and launches that clip, against the
oracle bit for bit (a bin out of submission order would show in blended
colours and equal depths)."""
import numpy as np
import pytest

from pixelforge_gb300 import abi as A
from pixelforge_gb300.scenes import Target, _ptr

pytestmark = pytest.mark.gpu


def _soup(seed, n, every, clip):
    """n triangles of which every `every`-th is visible, all over the image
    and behind one another at few distinct depths."""
    r = np.random.default_rng(seed)
    pos = r.uniform(-0.9, 0.9, (n, 3, 3)).astype(np.float32)
    pos[:, :, 2] = r.integers(1, 6, (n, 1)) / 8.0
    hidden = np.arange(n) % every != 0
    pos[hidden] = pos[hidden][:, :1]                    # a point: culled
    if clip:
        pos[::37, 0, 2] = 3.0                           # behind the camera of the perspective view
    return np.ascontiguousarray(pos.reshape(-1, 3)), r.integers(0, 256, (3 * n, 4), dtype=np.uint8)


def _render(lib, n, every, w, h, clip):
    tg = Target(lib, w, h, "fbo")
    try:
        lib.pfClearFramebuffer(tg._fbref, A.PFcolor(1, 2, 3, 255), 1e30)
        if clip:
            lib.pfMatrixMode(A.PF_PROJECTION)
            lib.pfLoadIdentity()
            lib.pfFrustum(-0.1, 0.1, -0.1, 0.1, 0.1, 10.0)
            lib.pfMatrixMode(A.PF_MODELVIEW)
            lib.pfLoadIdentity()
            lib.pfTranslatef(0.0, 0.0, -2.0)
        pos, col = _soup(n + every, n, every, clip)
        lib.pfEnable(A.PF_DEPTH_TEST)
        lib.pfDepthFunc(A.PF_LEQUAL)
        lib.pfEnable(A.PF_BLEND)
        lib.pfBlendFunc(A.PF_BLEND_ALPHA)
        lib.pfDisable(A.PF_CULL_FACE)
        lib.pfEnable(A.PF_VERTEX_ARRAY | A.PF_COLOR_ARRAY)
        lib.pfVertexPointer(3, A.PF_FLOAT, 0, _ptr(pos))
        lib.pfColorPointer(4, A.PF_UNSIGNED_BYTE, 0, _ptr(col))
        half = n // 2
        lib.pfDrawArrays(A.PF_TRIANGLES, 0, 3 * half)
        lib.pfDrawArrays(A.PF_TRIANGLES, 3 * half, 3 * (n - half))
        return tg.finish()
    finally:
        tg.close()


# culling off: two items a triangle
@pytest.mark.parametrize("n,every,w,h,clip", [
    (300, 1, 24, 16, False), (895, 1, 16, 16, False), (1025, 1, 17, 9, False), (5000, 3, 24, 24, False),
    (16000, 7, 16, 24, False), (32760, 23, 16, 16, False), (32768, 23, 16, 16, False), (33000, 23, 16, 16, False),
    (700, 1, 24, 24, True), (40000, 41, 16, 16, True)])
def test_sorted_bins_vs_oracle(gpu, oracle, n, every, w, h, clip):
    a, b = _render(gpu, n, every, w, h, clip), _render(oracle, n, every, w, h, clip)
    assert np.array_equal(a.depth.view(np.uint32), b.depth.view(np.uint32))
    assert np.array_equal(a.color, b.color)
    assert gpu.pfGetDeviceStatus() == 0


def test_batch_of_uneven_targets(gpu, oracle):
    """Targets whose items start anywhere in the launch's numbering."""
    sizes = [(16, 16, 700), (24, 8, 5), (8, 24, 3000), (16, 24, 400), (40, 40, 9000)]

    def scene(lib, batch):
        out, keep = [], []
        if batch:
            b = lib.pfgbBatchCreate()
            lib.pfgbBatchBegin(b)
        for k, (w, h, n) in enumerate(sizes):
            buf = np.zeros((h, w, 4), np.uint8)
            ctx = lib.pfCreateContext(_ptr(buf), w, h, A.PF_RGBA, A.PF_UNSIGNED_BYTE)
            lib.pfMakeCurrent(ctx)
            pos, col = _soup(90 + k, n, 1, False)
            lib.pfClearDepth(1.0)
            lib.pfClear(A.PF_COLOR_BUFFER_BIT | A.PF_DEPTH_BUFFER_BIT)
            lib.pfEnable(A.PF_BLEND)
            lib.pfBlendFunc(A.PF_BLEND_ALPHA)
            lib.pfEnable(A.PF_VERTEX_ARRAY | A.PF_COLOR_ARRAY)
            lib.pfVertexPointer(3, A.PF_FLOAT, 0, _ptr(pos))
            lib.pfColorPointer(4, A.PF_UNSIGNED_BYTE, 0, _ptr(col))
            lib.pfDrawArrays(A.PF_TRIANGLES, 0, 3 * n)
            out.append(buf)
            keep.append((ctx, pos, col))
        if batch:
            lib.pfgbBatchEnd(b)
            lib.pfgbBatchDelete(b)
        for ctx, _, _ in keep:
            lib.pfMakeCurrent(ctx)
            lib.pfDeleteContext(ctx)
        return out

    for x, y in zip(scene(gpu, True), scene(oracle, False)):
        assert np.array_equal(x, y)
