"""Two draws of one flush over the same vertex arrays with the lighting
changed between them: the second must not read the vertices that the first
one lit.  Each draw in a flush of its own is the bar, bit for bit, and the
oracle, to the last place of its Gouraud colours; that each change is seen in
the picture is checked on the oracle alone."""
import numpy as np
import pytest

from pixelforge_gb300 import abi as A
from pixelforge_gb300.scenes import Target, _ptr

pytestmark = pytest.mark.gpu

COLOR_TOL = 1
SIDE = 40
_keep = []


def _v(*x):
    _keep.append(np.array(x, np.float32))
    return _ptr(_keep[-1])


STEPS = {
    "position": lambda lib: lib.pfLightfv(0, A.PF_POSITION, _v(-3.0, 2.0, 1.0)),
    "diffuse": lambda lib: lib.pfLightfv(0, A.PF_DIFFUSE, _v(0.2, 0.9, 0.1)),
    "specular": lambda lib: lib.pfLightfv(0, A.PF_SPECULAR, _v(0.9, 0.1, 0.1)),
    "ambient": lambda lib: lib.pfLightfv(0, A.PF_AMBIENT, _v(0.5, 0.1, 0.5)),
    "attenuation": lambda lib: lib.pfLightf(0, A.PF_LINEAR_ATTENUATION, 0.3),
    "spot": lambda lib: (lib.pfLightfv(0, A.PF_SPOT_DIRECTION, _v(-0.5, -0.3, -0.8)), lib.pfLightf(0, A.PF_SPOT_INNER_CUTOFF, 15.0),
                         lib.pfLightf(0, A.PF_SPOT_OUTER_CUTOFF, 40.0)),
    "second": lambda lib: (lib.pfEnableLight(3), lib.pfLightfv(3, A.PF_POSITION, _v(-2.0, -2.0, 2.0))),
    "none": lambda lib: lib.pfDisableLight(0),
    "material_diffuse": lambda lib: lib.pfMaterialfv(A.PF_FRONT_AND_BACK, A.PF_DIFFUSE, _v(0.3, 0.9, 0.5)),
    "material_specular": lambda lib: lib.pfMaterialf(A.PF_FRONT_AND_BACK, A.PF_SPECULAR, 0.1),
    "material_ambient": lambda lib: lib.pfMaterialfv(A.PF_FRONT_AND_BACK, A.PF_AMBIENT, _v(0.1, 0.2, 0.9)),
    "emission": lambda lib: lib.pfMaterialfv(A.PF_FRONT_AND_BACK, A.PF_EMISSION, _v(0.2, 0.1, 0.4)),
    "shininess": lambda lib: lib.pfMaterialf(A.PF_FRONT_AND_BACK, A.PF_SHININESS, 3.0),
    "to_phong": lambda lib: lib.pfLightModel(A.PF_PHONG),
    "to_gouraud": lambda lib: lib.pfLightModel(A.PF_GOURAUD),
    "off": lambda lib: lib.pfDisable(A.PF_LIGHTING),
    "camera": lambda lib: lib.pfTranslatef(0.02, 0.05, -0.1),
    # (the product of the matrices stays, the eye moves)
    "eye": lambda lib: (lib.pfTranslatef(0.0, 0.0, -2.0), lib.pfMatrixMode(A.PF_PROJECTION), lib.pfTranslatef(0.0, 0.0, 2.0),
                        lib.pfMatrixMode(A.PF_MODELVIEW)),
    "normals": lambda lib: lib.pfDisable(A.PF_NORMAL_ARRAY),
}


def _render(lib, step, apart, first_model=A.PF_GOURAUD):
    r = np.random.default_rng(21)
    n = 48
    pos = r.uniform(-1.1, 1.1, (n, 3)).astype(np.float32)
    nrm = r.normal(size=(n, 3)) * 0.4 + [0.3, 0.2, 1.0]
    nrm = (nrm / np.linalg.norm(nrm, axis=1, keepdims=True)).astype(np.float32)
    idx = [r.integers(0, n, 60).astype(np.uint32) for _ in range(2)]
    tg = Target(lib, SIDE, SIDE, "fbo")
    try:
        lib.pfClearFramebuffer(tg._fbref, A.PFcolor(5, 6, 7, 255), 1e30)
        lib.pfMatrixMode(A.PF_PROJECTION)
        lib.pfLoadIdentity()
        lib.pfFrustum(-0.05, 0.05, -0.05, 0.05, 0.1, 10.0)
        lib.pfMatrixMode(A.PF_MODELVIEW)
        lib.pfLoadIdentity()
        lib.pfTranslatef(0.0, 0.0, -3.0)
        lib.pfDisable(A.PF_CULL_FACE)
        lib.pfEnable(A.PF_LIGHTING | A.PF_VERTEX_ARRAY | A.PF_NORMAL_ARRAY)
        lib.pfLightModel(first_model)
        lib.pfEnableLight(0)
        lib.pfLightfv(0, A.PF_POSITION, _v(2.0, 1.0, 4.0))
        lib.pfMaterialf(A.PF_FRONT_AND_BACK, A.PF_DIFFUSE, 0.8)
        lib.pfMaterialf(A.PF_FRONT_AND_BACK, A.PF_SPECULAR, 0.9)
        lib.pfMaterialf(A.PF_FRONT_AND_BACK, A.PF_SHININESS, 16.0)
        lib.pfVertexPointer(3, A.PF_FLOAT, 0, _ptr(pos))
        lib.pfNormalPointer(A.PF_FLOAT, 0, _ptr(nrm))
        lib.pfColor4ub(220, 200, 180, 255)
        lib.pfDrawElements(A.PF_TRIANGLES, 60, A.PF_UNSIGNED_INT, _ptr(idx[0]))
        if apart:
            lib.pfFinish()
        if step:
            STEPS[step](lib)
        lib.pfDrawElements(A.PF_TRIANGLES, 60, A.PF_UNSIGNED_INT, _ptr(idx[1]))
        return tg.finish()
    finally:
        tg.close()


@pytest.mark.parametrize("model,step", [(m, s) for m in ("gouraud", "phong") for s in STEPS
                                        if s != "to_" + m and (m, s) != ("phong", "emission")])    # (which has no emission)
def test_lighting_changed_between_draws(gpu, oracle, step, model):
    first = A.PF_GOURAUD if model == "gouraud" else A.PF_PHONG
    ref = _render(oracle, step, False, first)
    assert np.abs(ref.color.astype(int) - _render(oracle, None, False, first).color).max() > 4 * COLOR_TOL
    got, apart = _render(gpu, step, False, first), _render(gpu, step, True, first)
    assert np.array_equal(got.color, apart.color)
    assert np.array_equal(got.depth.view(np.uint32), apart.depth.view(np.uint32))
    assert np.abs(got.color.astype(int) - ref.color).max() <= COLOR_TOL
    assert np.array_equal(got.depth.view(np.uint32), ref.depth.view(np.uint32))
    assert gpu.pfGetDeviceStatus() == 0
