"""The row pipeline of BGRA / unsigned-byte framebuffers against the oracle,
bit for bit: rows narrower than a half, records wider than a batch's 96
halves (384 pixels), rows too wide for shared memory, hundreds of records a
row with state changes in between (blend modes in both channel orders,
points and lines, lighting per fragment), and the fragment count."""
import numpy as np
import pytest

from pixelforge_gb300 import abi as A
from test_deep_tiles_gpu import SCENES, _scene

pytestmark = pytest.mark.gpu

BGRA8 = (A.PF_BGRA, A.PF_UNSIGNED_BYTE)


@pytest.mark.parametrize("size", [(3, 9), (37, 21), (383, 4), (389, 4), (1201, 3), (2051, 3)])
@pytest.mark.parametrize("phong", [False, True])
@pytest.mark.parametrize("name", list(SCENES))
def test_rows_vs_oracle(gpu, oracle, name, phong, size):
    a = _scene(gpu, name, phong, False, *size, BGRA8)
    b = _scene(oracle, name, phong, False, *size, BGRA8)
    assert np.array_equal(a.depth.view(np.uint32), b.depth.view(np.uint32))
    assert np.array_equal(a.color, b.color)
    if "fragments" in b.stats:
        assert a.stats["fragments"] == b.stats["fragments"]
    assert gpu.pfGetDeviceStatus() == 0
