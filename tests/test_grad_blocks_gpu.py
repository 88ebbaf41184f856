"""The differentiable kernels' block lists against the FP64 oracle: images of
odd sizes, tile lists of several staged chunks, and blocks whose visible
fragments fill the list, are split by pixel rows, or are walked pixel by
pixel.  Bars as in test_grad_gpu.py: images within 2e-5 absolute, gradients
within 1e-4 of the FP64 adjoint, norm-wise per group."""
import numpy as np
import pytest

from pixelforge_gb300.fit import FitScene, look_at, perspective, to_device
from pixelforge_gb300.grad import GradScene, Mesh, PARAM_NAMES

pgref = pytest.importorskip("pgref")
torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _layers(n):
    """n quads facing the camera, far to near: every one is visible."""
    z = np.linspace(-1.0, 1.0, n) if n > 1 else np.zeros(1)
    quad = np.array([(-0.8, -0.6), (0.8, -0.6), (0.8, 0.6), (-0.8, 0.6)])
    pos = np.concatenate([np.concatenate([quad, np.full((4, 1), k)], 1) for k in z])
    nrm = np.tile([0.0, 0.0, 1.0], (4 * n, 1))
    uv = np.tile([(0.11, 0.07), (0.93, 0.07), (0.93, 0.89), (0.11, 0.89)], (n, 1))
    tri = np.concatenate([np.array([(0, 1, 2), (0, 2, 3)]) + 4 * k for k in range(n)])
    return Mesh(pos.astype(np.float32), nrm.astype(np.float32), uv.astype(np.float32), tri.astype(np.uint32))


def _check(mesh, mvp, eyes, w, h, tex, wrap, filt, opacity, seed):
    rng = np.random.default_rng(seed)
    nv = len(mesh.positions)
    params = {"texture": rng.uniform(0.2, 0.9, (tex, tex, 4)).astype(np.float32),
              "colors": rng.uniform(0.2, 0.9, (nv, 3)).astype(np.float32),
              "alphas": (opacity * rng.uniform(0.6, 1.0, nv)).astype(np.float32),
              "material": np.array([0.8, 0.5, 12.0], np.float32),
              "light": np.array([0.3, 0.5, 0.8], np.float32)}
    kw = dict(filter=filt, wrap=wrap, cull=-1, ambient=0.2)
    gs = GradScene(mesh, mvp, eyes, w, h, (tex, tex), **kw)
    rs = pgref.RefScene(mesh, mvp, eyes, w, h, (tex, tex), **kw)
    try:
        ts = to_device(params)
        img = gs.render(*ts)
        _, ref = rs.forward(rs.pack(params))
        assert np.abs(img.detach().cpu().numpy() - ref).max() <= 2e-5
        target = torch.from_numpy(rng.uniform(0.0, 1.0, gs.image_shape()).astype(np.float32)).cuda()
        ((img - target) ** 2).mean().backward()
        gref = rs.unpack(rs.gradient(rs.pack(params), target.cpu().numpy(), 1.0 / target.numel()))
        for k, t in zip(PARAM_NAMES, ts):
            g = t.grad.detach().cpu().numpy().astype(np.float64)
            err = np.linalg.norm(g - gref[k]) / max(np.linalg.norm(gref[k]), 1e-30)
            assert err <= 1e-4, f"{k}: relative error {err:.2e} against the FP64 adjoint"
    finally:
        gs.close()


# a block of 64 pixels lists 128 fragments: 2 layers fill it, 3 and 4 split
# it by rows, more are walked pixel by pixel (4 at a time)
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 9, 33, 70])
@pytest.mark.parametrize("w,h,filt,wrap", [(20, 12, 1, 0), (37, 29, 0, 1)])
def test_layers(n, w, h, filt, wrap):
    eyes = np.array([[0.0, 0.0, 3.0], [0.4, 0.3, 3.0]])
    mvp = np.stack([(look_at(e) @ perspective(60.0, w / h, 0.1, 100.0)).reshape(16) for e in eyes])
    _check(_layers(n), mvp.astype(np.float32), eyes.astype(np.float32), w, h, 16, wrap, filt, min(1.0, 3.0 / n), 50 + n)


# triangles from a pixel to below it: tile lists of one to many chunks of 64
@pytest.mark.parametrize("subdiv,w,h", [(1, 64, 64), (3, 61, 43), (4, 48, 40), (5, 45, 37), (5, 130, 97)])
def test_dense_meshes(subdiv, w, h):
    fs = FitScene(subdiv=subdiv, n_views=2, size=64, tex_size=24)
    _, eyes = fs.cameras()
    mvp = np.stack([(look_at(e) @ perspective(60.0, w / h, 0.1, 100.0)).reshape(16) for e in eyes.astype(np.float64)])
    _check(fs.mesh(), mvp.astype(np.float32), eyes, w, h, 24, 2, 1, 0.8, subdiv)
