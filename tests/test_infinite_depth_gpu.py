"""Depth buffers that hold infinities, the largest value and zeros under more
than a tile's batch of triangles, with depths of either sign: flat layers,
slanted ones, and perspective geometry before and behind the middle of the
depth range (where depths change their sign), against the oracle, bit for
bit, with the fragment count."""
import numpy as np
import pytest

from pixelforge_gb300 import abi as A
from pixelforge_gb300.scenes import FLT_MAX, Target, _ptr

pytestmark = pytest.mark.gpu

INF = float("inf")
W, H, N = 45, 29, 600
FORMATS = {"rgba8": (A.PF_RGBA, A.PF_UNSIGNED_BYTE), "rgb565": (A.PF_RGB, A.PF_UNSIGNED_SHORT_5_6_5),
           "bgra8": (A.PF_BGRA, A.PF_UNSIGNED_BYTE)}


def _scene(lib, clear, depths, func, fmt):
    r = np.random.default_rng(sum(map(ord, depths)) + func)
    tg = Target(lib, W, H, "fbo", fmt=FORMATS[fmt])
    try:
        if clear == "holes":        # the caller's own buffer: finite but for a few pixels
            lib.pfClearFramebuffer(tg._fbref, A.PFcolor(9, 8, 7, 255), 0.5)
            lib.pfFinish()
            z = np.ctypeslib.as_array(tg.fb.zbuffer, shape=(H, W))
            z[r.random((H, W)) < 0.05] = INF
        elif clear == "pfClear":
            lib.pfClearDepth(INF)
            lib.pfClear(A.PF_COLOR_BUFFER_BIT | A.PF_DEPTH_BUFFER_BIT)
        else:
            lib.pfClearFramebuffer(tg._fbref, A.PFcolor(9, 8, 7, 255), clear)
        lib.pfEnable(A.PF_DEPTH_TEST | A.PF_VERTEX_ARRAY | A.PF_COLOR_ARRAY)
        lib.pfDepthFunc(func)
        lib.pfDisable(A.PF_CULL_FACE)
        pos = r.uniform(-1.0, 1.0, (N, 1, 3)) * [1.0, 1.0, 0.0] + r.uniform(-1.6, 1.6, (N, 3, 3)) * [1.0, 1.0, 0.0]
        slant = r.choice([0.0, 0.05], (N, 1)) * r.uniform(-1, 1, (N, 3))
        if depths.startswith("perspective"):
            lib.pfMatrixMode(A.PF_PROJECTION)
            lib.pfLoadIdentity()
            lib.pfFrustum(-0.1, 0.1, -0.1, 0.1, 0.1, 10.0)
            lib.pfMatrixMode(A.PF_MODELVIEW)
            lib.pfLoadIdentity()
            # (clip z changes its sign at a distance of 0.198)
            near, far = (0.11, 0.19) if depths.endswith("near") else (0.25, 6.0)
            dist = r.uniform(near, far, (N, 1)) * (1.0 + 0.2 * slant)
            dist = np.clip(dist, near, far)
            pos[:, :, :2] = np.clip(pos[:, :, :2], -1.0, 1.0) * (0.98 * dist[:, :, None])
            pos[:, :, 2] = -dist
        else:
            pos[:, :, 2] = (1.0 if depths == "positive_z" else -1.0) * (r.uniform(0.2, 0.9, (N, 1)) + slant)
        pos = np.ascontiguousarray(pos.reshape(-1, 3), np.float32)
        col = r.integers(0, 256, (3 * N, 4), dtype=np.uint8)
        lib.pfVertexPointer(3, A.PF_FLOAT, 0, _ptr(pos))
        lib.pfColorPointer(4, A.PF_UNSIGNED_BYTE, 0, _ptr(col))
        lib.pfDrawArrays(A.PF_TRIANGLES, 0, 3 * N)
        return tg.finish()
    finally:
        tg.close()


@pytest.mark.parametrize("fmt", list(FORMATS))
@pytest.mark.parametrize("func", [A.PF_LESS, A.PF_LEQUAL])
@pytest.mark.parametrize("depths", ["positive_z", "negative_z", "perspective_near", "perspective_far"])
@pytest.mark.parametrize("clear", [INF, "pfClear", "holes", FLT_MAX, 0.0, -INF])
def test_infinite_depths_vs_oracle(gpu, oracle, clear, depths, func, fmt):
    got, ref = _scene(gpu, clear, depths, func, fmt), _scene(oracle, clear, depths, func, fmt)
    assert np.array_equal(got.depth.view(np.uint32), ref.depth.view(np.uint32))
    assert np.array_equal(got.color, ref.color)
    if "fragments" in ref.stats:
        assert got.stats["fragments"] == ref.stats["fragments"]
    assert gpu.pfGetDeviceStatus() == 0
