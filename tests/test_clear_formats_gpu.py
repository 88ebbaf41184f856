"""A clear or a fill folded into the draw that follows, over tiles that stay
empty: every accepted pixel format, rows that are whole tiles and rows that
are not, rows that start on 16 bytes and rows that do not, and a batch whose
targets differ in format, against the oracle, byte for byte."""
import numpy as np
import pytest

from fbscenes import FB_ACCEPTED
from pixelforge_gb300 import abi as A
from pixelforge_gb300.scenes import Target, _ptr

pytestmark = pytest.mark.gpu

SIZES = [(64, 24), (61, 19), (20, 16), (36, 9), (8, 8)]


def _draw(lib, fill, tg, at):
    """A clear, then a triangle of a few pixels, so that all other tiles are empty."""
    if fill and tg.kind == "fbo":
        lib.pfClearFramebuffer(tg._fbref, A.PFcolor(201, 78, 33, 170), 0.75)
    else:
        lib.pfClearColor(201, 78, 33, 170)
        lib.pfClearDepth(0.75)
        lib.pfClear(A.PF_COLOR_BUFFER_BIT | A.PF_DEPTH_BUFFER_BIT)
    lib.pfEnable(A.PF_VERTEX_ARRAY)
    lib.pfDisable(A.PF_CULL_FACE)
    pos = (np.array([(0, 0, 0.1), (0.2, 0, 0.1), (0, 0.4, 0.1)], np.float32) + np.array([*at, 0], np.float32)).astype(np.float32)
    lib.pfVertexPointer(3, A.PF_FLOAT, 0, _ptr(pos))
    lib.pfColor4ub(10, 250, 120, 255)
    lib.pfDrawArrays(A.PF_TRIANGLES, 0, 3)
    return pos


def _frames(lib, fmt, kind):
    out = []
    for i, (w, h) in enumerate(SIZES):
        r = np.random.default_rng(w)
        init = None
        if fmt[1] == A.PF_UNSIGNED_BYTE:
            init = r.integers(0, 256, (h, w, A.pixel_bytes(*fmt)), dtype=np.uint8)
        tg = Target(lib, w, h, kind, init=init, fmt=fmt)
        try:
            for fill in (False, True):
                _draw(lib, fill, tg, (-0.9 if i % 2 else 0.6, 0.3))
                fr = tg.finish()
                out += [fr.color] + ([fr.depth.view(np.uint32)] if fr.depth is not None else [])
        finally:
            tg.close()
    return out


@pytest.mark.parametrize("kind", ["main", "fbo"])
@pytest.mark.parametrize("fmt", FB_ACCEPTED)
def test_folded_clear_vs_oracle(gpu, oracle, fmt, kind):
    a, b = _frames(gpu, fmt, kind), _frames(oracle, fmt, kind)
    assert len(a) == len(b)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
    assert gpu.pfGetDeviceStatus() == 0


def test_folded_clears_of_a_batch_of_formats(gpu, oracle):
    def one(lib, batch):
        tgs, keep = [Target(lib, *SIZES[i % len(SIZES)], "main", fmt=f) for i, f in enumerate(FB_ACCEPTED)], []
        try:
            b = lib.pfgbBatchCreate() if batch else None
            if batch:
                lib.pfgbBatchBegin(b)
            for tg in tgs:
                lib.pfMakeCurrent(tg.ctx)
                keep.append(_draw(lib, False, tg, (0.2, -0.4)))
            if batch:
                lib.pfgbBatchEnd(b)
                lib.pfgbBatchDelete(b)
            return [tg.main.copy() for tg in tgs]
        finally:
            for tg in tgs:
                lib.pfMakeCurrent(tg.ctx)
                tg.close()
    for x, y in zip(one(gpu, True), one(oracle, False)):
        assert np.array_equal(x, y)
    assert gpu.pfGetDeviceStatus() == 0
