"""Performance cases: passes of the library's public entry points over the
range of calls its users make.

A case is a dict of plain values; its ``kind`` says which entry point it
drives:

  static  pfgbDrawTrianglesStatic, the allocation-free call on device buffers
  soup    one context, a triangle soup through pfDrawArrays into a framebuffer
          object whose colour and depth the caller reads
  sphere  one context, a textured Gouraud-lit UV sphere drawn opaque and then
          blended, into the caller's buffer, in one of the pixel formats
  phong   one context, a displaced icosphere lit per fragment, with device fog
  batch   many contexts of uneven sizes rendered as one pfgbBatch
  grad    the differentiable renderer: images of many views, and optionally
          the gradients of a loss with respect to every parameter

``prepare`` makes what a program has in hand before it draws (contexts,
textures, vertex arrays, device tensors), ``run`` draws one frame and returns
the buffers it lands in.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

from pixelforge_gb300 import abi as A, load_library
from pixelforge_gb300.fit import look_at, fibonacci_sphere, perspective
from pixelforge_gb300.grad import GradScene, Mesh
from pixelforge_gb300.scenes import icosphere, uv_sphere

# name -> (format, type, bytes per pixel)
FORMATS = {"rgba8": (A.PF_RGBA, A.PF_UNSIGNED_BYTE, 4), "bgra8": (A.PF_BGRA, A.PF_UNSIGNED_BYTE, 4),
           "rgb565": (A.PF_RGB, A.PF_UNSIGNED_SHORT_5_6_5, 2), "rgba16f": (A.PF_RGBA, A.PF_HALF_FLOAT, 8)}
FILTERS = {"nearest": A.PF_NEAREST, "bilinear": A.PF_BILINEAR}
WRAPS = {"repeat": A.PF_REPEAT, "mirror": A.PF_MIRRORED_REPEAT, "clamp": A.PF_CLAMP_TO_EDGE}
BLENDS = {"none": None, "alpha": A.PF_BLEND_ALPHA, "add": A.PF_BLEND_ADD, "mul": A.PF_BLEND_MUL}
COLOR_DEPTH = A.PF_COLOR_BUFFER_BIT | A.PF_DEPTH_BUFFER_BIT
STATIC_FAR = 16.0
SOUP_AREA = 11.0 / 144.0       # mean area of a triangle of three uniform points, as a share of the square


def listed():
    return [
        # the smallest call: a handful of triangles into a thumbnail, latency and launches only
        dict(name="static_64", kind="static", width=64, height=64, ntris=64),
        # the same entry point at its limits: a frame path that may not allocate
        dict(name="static_512", kind="static", width=512, height=512, ntris=8192),
        # one small context of many (an environment, an icon): host arrays, textured and blended
        dict(name="soup_64_textured", kind="soup", width=64, height=64, ntris=400, blend="alpha", texture=64,
             filt="bilinear", wrap="repeat"),
        # overlapping triangles with colour and depth read back: heavy overdraw in a small image
        dict(name="soup_256", kind="soup", width=256, height=256, ntris=2000, blend="none", texture=0,
             filt="nearest", wrap="repeat"),
        # a frame of the textured sphere from host arrays, as a program written for the CPU library sends it
        dict(name="sphere_1080_host", kind="sphere", width=1920, height=1080, segments=256, rings=128, texture=1024,
             filt="bilinear", wrap="repeat", format="rgba8", device=False),
        # the same frame with arrays, indices and texture already in device memory
        dict(name="sphere_1080", kind="sphere", width=1920, height=1080, segments=256, rings=128, texture=1024,
             filt="bilinear", wrap="repeat", format="rgba8", device=True),
        # a window's native pixel order
        dict(name="sphere_1080_bgra8", kind="sphere", width=1920, height=1080, segments=256, rings=128, texture=1024,
             filt="bilinear", wrap="repeat", format="bgra8", device=True),
        # half-float output at an odd size, nearest texels
        dict(name="sphere_odd_rgba16f", kind="sphere", width=1365, height=767, segments=100, rings=51, texture=500,
             filt="nearest", wrap="mirror", format="rgba16f", device=True),
        # a dense mesh lit per fragment, 30 % of it additive, then fog
        dict(name="phong_1080", kind="phong", width=1920, height=1080, subdiv=8, texture=2048, lights=8),
        # many contexts of uneven sizes and loads in one launch of each kernel
        dict(name="batch_64", kind="batch", contexts=64, max_side=512, tri_median=2000),
        # one iteration of an inverse-rendering fit: images and all gradients
        dict(name="grad_64x512", kind="grad", views=64, width=512, height=512, subdiv=5, texture=512, filt="bilinear",
             wrap="repeat", backward=True),
        # evaluation of a few views at an odd size, forward only
        dict(name="grad_eval_odd", kind="grad", views=5, width=301, height=203, subdiv=4, texture=200, filt="bilinear",
             wrap="mirror", backward=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["static", "soup", "soup", "sphere", "sphere", "phong", "batch", "grad", "grad"])
    filt, wrap = rng.choice(list(FILTERS)), rng.choice(list(WRAPS))
    if kind == "static":
        return dict(kind=kind, width=rng.randint(33, 512), height=rng.randint(33, 512), ntris=_log(rng, 16, 8192))
    if kind == "soup":
        w, h = _log(rng, 48, 1280), _log(rng, 48, 1024)
        most = int(5e7 / (SOUP_AREA * w * h))          # covered pixels of all triangles
        return dict(kind=kind, width=w, height=h, ntris=_log(rng, 32, max(64, min(20000, most))),
                    blend=rng.choice(list(BLENDS)), texture=rng.choice([0, 64, 255, 512]), filt=filt, wrap=wrap)
    if kind == "sphere":
        return dict(kind=kind, width=_log(rng, 160, 1920), height=_log(rng, 120, 1080), segments=_log(rng, 16, 256),
                    rings=_log(rng, 8, 128), texture=_log(rng, 64, 1024), filt=filt, wrap=wrap,
                    format=rng.choice(["rgba8", "rgba8", "rgba8", "bgra8", "rgb565", "rgba16f"]),
                    device=rng.random() < 0.6)
    if kind == "phong":
        return dict(kind=kind, width=_log(rng, 320, 1920), height=_log(rng, 200, 1080), subdiv=rng.randint(4, 7),
                    texture=_log(rng, 128, 2048), lights=rng.randint(1, 8))
    if kind == "batch":
        return dict(kind=kind, contexts=_log(rng, 4, 48), max_side=rng.choice([128, 256, 384, 512]),
                    tri_median=_log(rng, 200, 2000))
    w = _log(rng, 64, 512)
    # (taller images would clip the sphere at the sides, which the differentiable path refuses)
    return dict(kind="grad", views=_log(rng, 1, 64), width=w, height=rng.randint(w // 2, min(512, int(1.3 * w))),
                subdiv=rng.randint(2, 5), texture=_log(rng, 32, 512), filt=filt, wrap=wrap, backward=rng.random() < 0.6)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _uniform(g, shape, lo, hi):
    return torch.rand(shape, generator=g, device="cuda") * (hi - lo) + lo


def _bytes(g, shape):
    """RGBA8 noise, alpha 255."""
    t = torch.randint(0, 256, (*shape, 4), generator=g, device="cuda", dtype=torch.uint8)
    t[..., 3] = 255
    return t


def _smooth(g, size, channels):
    """Smooth value noise in [0, 1], (size, size, channels)."""
    lattice = torch.rand((1, channels, 33, 33), generator=g, device="cuda")
    t = torch.nn.functional.interpolate(lattice, size=(size, size), mode="bilinear", align_corners=True)
    return t[0].permute(1, 2, 0).contiguous()


_icosphere = functools.lru_cache(maxsize=None)(icosphere)
_uv_sphere = functools.lru_cache(maxsize=None)(uv_sphere)


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _dp(t):
    return C.c_void_p(t.data_ptr())


def _hp(a):
    return C.c_void_p(a.ctypes.data)


def _static_inputs(case, seed):
    """Small triangles scattered through the view volume of a perspective camera."""
    g, n = _gen(seed), case["ntris"]
    centre = torch.cat([_uniform(g, (n, 1, 1), -0.5, 0.5), _uniform(g, (n, 1, 1), -0.4, 0.4),
                        torch.zeros((n, 1, 1), device="cuda")], -1)
    pos = centre + torch.cat([_uniform(g, (n, 3, 2), -0.07, 0.07), _uniform(g, (n, 3, 1), -0.9, 0.9)], -1)
    col = torch.randint(0, 256, (n * 3, 4), generator=g, device="cuda", dtype=torch.uint8)
    l, t, near, far = 0.06, 0.045, 0.1, 10.0
    m = np.zeros(16, np.float32)
    m[0], m[5], m[10], m[11] = near / l, near / t, -(far + near) / (far - near), -1.0
    m[14] = -2.0 * far * near / (far - near)
    m[14] += -2.0 * m[10]                              # the camera two units back
    m[15] = 2.0
    return pos.contiguous(), col, m


def _soup_inputs(case, seed):
    """Triangles with corners anywhere in the image, as numpy arrays."""
    g, n = _gen(seed), case["ntris"] * 3
    pos = torch.cat([_uniform(g, (n, 2), -1.0, 1.0), _uniform(g, (n, 1), 0.1, 0.9)], -1)
    col = torch.randint(0, 256, (n, 4), generator=g, device="cuda", dtype=torch.uint8)
    uv = _uniform(g, (n, 2), 0.0, 2.0)
    tex = _bytes(g, (case["texture"], case["texture"])) if case["texture"] else None
    return pos.cpu().numpy(), col.cpu().numpy(), uv.cpu().numpy(), None if tex is None else tex.cpu().numpy()


# ---------------------------------------------------------------------------
# pf* contexts
# ---------------------------------------------------------------------------
class _Context:
    """A context on a buffer of its own, deleted with the object."""

    def __init__(self, lib, w, h, fmt="rgba8"):
        f, t, bpp = FORMATS[fmt]
        self.lib, self.w, self.h = lib, w, h
        # (room behind the pixels: pfClear's tail writes past those of packed formats)
        self.backing = np.zeros(h * w * bpp * (4 if bpp == 2 else 1), np.uint8)
        self.buf = self.backing[:h * w * bpp].reshape(h, w, bpp)
        self.ctx = lib.pfCreateContext(_hp(self.buf), w, h, f, t)
        if not self.ctx:
            raise RuntimeError("pfCreateContext failed")
        lib.pfMakeCurrent(self.ctx)
        self.fb, self.textures, self.keep = None, [], []

    def framebuffer(self):
        """A bound framebuffer object; its colour and depth as numpy views."""
        lib = self.lib
        self.fb = lib.pfGenFramebuffer(self.w, self.h, A.PF_RGBA, A.PF_UNSIGNED_BYTE)
        self.fbref = C.pointer(self.fb)
        lib.pfBindFramebuffer(self.fbref)
        lib.pfEnable(A.PF_FRAMEBUFFER)
        base = lib.pfGetTexturePixels(self.fb.texture, None, None, None, None)
        self.color = np.ctypeslib.as_array(C.cast(base, C.POINTER(C.c_uint8)), shape=(self.h, self.w, 4))
        self.depth = np.ctypeslib.as_array(self.fb.zbuffer, shape=(self.h, self.w))

    def texture(self, t, filt, wrap):
        lib = self.lib
        h, w = t.shape[:2]
        if isinstance(t, torch.Tensor):
            th = lib.pfGenTextureDevice(_dp(t), w, h)
        else:
            th = lib.pfGenTexture(_hp(t), w, h, A.PF_RGBA, A.PF_UNSIGNED_BYTE)
        self.textures.append(th)
        self.keep.append(t)
        lib.pfTextureParameter(th, WRAPS[wrap], FILTERS[filt])
        lib.pfBindTexture(th)
        lib.pfEnable(A.PF_TEXTURE_2D)

    def arrays(self, pos=None, normal=None, uv=None, color=None):
        lib = self.lib
        for a, host, dev, bit, args in (
                (pos, lib.pfVertexPointer, lib.pfVertexPointerDevice, A.PF_VERTEX_ARRAY, (3, A.PF_FLOAT, 0)),
                (normal, lib.pfNormalPointer, lib.pfNormalPointerDevice, A.PF_NORMAL_ARRAY, (A.PF_FLOAT, 0)),
                (uv, lib.pfTexCoordPointer, lib.pfTexCoordPointerDevice, A.PF_TEXTURE_COORD_ARRAY, (A.PF_FLOAT, 0)),
                (color, lib.pfColorPointer, lib.pfColorPointerDevice, A.PF_COLOR_ARRAY, (4, A.PF_UNSIGNED_BYTE, 0))):
            if a is None:
                continue
            self.keep.append(a)
            lib.pfEnable(bit)
            if isinstance(a, torch.Tensor):
                dev(*args, _dp(a))
            else:
                host(*args, _hp(a))

    def camera(self, fov_deg, near, far, distance):
        lib = self.lib
        top = near * math.tan(math.radians(fov_deg) / 2)
        right = top * self.w / self.h
        lib.pfMatrixMode(A.PF_PROJECTION)
        lib.pfLoadIdentity()
        lib.pfFrustum(-right, right, -top, top, near, far)
        lib.pfMatrixMode(A.PF_MODELVIEW)
        lib.pfLoadIdentity()
        lib.pfTranslatef(0.0, 0.0, -distance)
        lib.pfEnable(A.PF_DEPTH_TEST)
        lib.pfDepthFunc(A.PF_LESS)

    def __del__(self):
        lib = self.lib
        if not getattr(self, "ctx", None):
            return
        lib.pfMakeCurrent(self.ctx)
        if self.fb is not None:
            lib.pfDisable(A.PF_FRAMEBUFFER)
            lib.pfBindFramebuffer(None)
            lib.pfDeleteFramebuffer(self.fbref)
        for th in self.textures:
            lib.pfDeleteTexture(C.byref(C.c_void_p(th)), False)
        lib.pfDeleteContext(self.ctx)
        self.ctx = None


class _State:
    """What one case keeps between its passes."""


def _soup_state(case, seed, lib):
    pos, col, uv, tex = _soup_inputs(case, seed)
    c = _Context(lib, case["width"], case["height"])
    c.framebuffer()
    lib.pfEnable(A.PF_DEPTH_TEST)
    lib.pfDepthFunc(A.PF_LESS)
    if BLENDS[case["blend"]] is not None:
        lib.pfEnable(A.PF_BLEND)
        lib.pfBlendFunc(BLENDS[case["blend"]])
    if tex is not None:
        c.texture(tex, case["filt"], case["wrap"])
    c.arrays(pos, None, uv if tex is not None else None, col)
    return c


def _soup_frame(c, ntris):
    lib = c.lib
    lib.pfMakeCurrent(c.ctx)
    lib.pfClearFramebuffer(c.fbref, A.PFcolor(20, 30, 40, 255), 1.0)
    lib.pfDrawArrays(A.PF_TRIANGLES, 0, ntris * 3)
    lib.pfFinish()
    return {"color": c.color, "depth": c.depth}


def _sphere_state(case, seed, lib):
    g = _gen(seed)
    pos, uv, idx = _uv_sphere(case["segments"], case["rings"])
    tex = _bytes(g, (case["texture"], case["texture"]))
    c = _Context(lib, case["width"], case["height"], case["format"])
    c.camera(60.0, 0.1, 100.0, 3.0)
    spin = torch.rand(2, generator=g, device="cuda").tolist()
    lib.pfRotatef(360.0 * spin[0], 0.0, 1.0, 0.0)
    lib.pfRotatef(60.0 * spin[1], 1.0, 0.0, 0.0)
    lib.pfEnable(A.PF_LIGHTING)
    lib.pfLightModel(A.PF_GOURAUD)
    lib.pfEnableLight(0)
    light = np.array([-577.0, 577.0, 577.0], np.float32)
    lib.pfLightfv(0, A.PF_POSITION, _hp(light))
    lib.pfMaterialf(A.PF_FRONT_AND_BACK, A.PF_DIFFUSE, 0.8)
    lib.pfMaterialf(A.PF_FRONT_AND_BACK, A.PF_SPECULAR, 0.5)
    lib.pfMaterialf(A.PF_FRONT_AND_BACK, A.PF_SHININESS, 32.0)
    if case["device"]:
        pos, uv, idx = _dev(pos), _dev(uv), _dev(idx.view(np.int32))
    else:
        tex, pos, uv, idx = tex.cpu().numpy(), pos.copy(), uv.copy(), idx.copy()
    c.texture(tex, case["filt"], case["wrap"])
    c.arrays(pos, pos, uv)
    c.idx, c.nverts = idx, len(pos)
    return c


def _elements(c, idx):
    if isinstance(idx, torch.Tensor):
        c.lib.pfDrawElementsDevice(A.PF_TRIANGLES, idx.numel(), c.nverts, _dp(idx))
    else:
        c.lib.pfDrawElements(A.PF_TRIANGLES, idx.size, A.PF_UNSIGNED_INT, _hp(idx))


def _sphere_frame(c):
    lib = c.lib
    lib.pfMakeCurrent(c.ctx)
    lib.pfClear(COLOR_DEPTH)
    lib.pfColor4ub(255, 255, 255, 255)
    _elements(c, c.idx)
    lib.pfPushMatrix()                                   # a translucent shell around it
    lib.pfScalef(1.05, 1.05, 1.05)
    lib.pfColor4f(1.0, 1.0, 1.0, 0.5)
    lib.pfEnable(A.PF_BLEND)
    lib.pfBlendFunc(A.PF_BLEND_ALPHA)
    lib.pfDepthMask(False)
    _elements(c, c.idx)
    lib.pfDepthMask(True)
    lib.pfDisable(A.PF_BLEND)
    lib.pfPopMatrix()
    lib.pfFinish()
    return c.buf


@functools.lru_cache(maxsize=2)
def _phong_mesh(subdiv):
    """Device copies of the undisplaced mesh: directions, texture coordinates, faces."""
    v, f = _icosphere(subdiv)
    v = torch.from_numpy(v).cuda()
    u = 0.5 + torch.atan2(v[:, 2], v[:, 0]) / (2 * math.pi)
    w = torch.arccos(v[:, 1].clamp(-1, 1)) / math.pi
    # (1.9, not 2: no vertex sits on the mirrored edge itself)
    return v, (torch.stack([u, w], 1) * 1.9).float().contiguous(), torch.from_numpy(f.astype(np.int32)).cuda()


def _phong_state(case, seed, lib):
    g = _gen(seed)
    v, uv, faces = _phong_mesh(case["subdiv"])
    pos = (v * (1.0 + 0.04 * torch.randn((len(v), 1), generator=g, device="cuda"))).float().contiguous()
    add = torch.rand(len(faces), generator=g, device="cuda") < 0.3
    tex = (_smooth(g, case["texture"], 4) * 255).to(torch.uint8)
    tex[..., 3] = 255
    c = _Context(lib, case["width"], case["height"])
    c.camera(60.0, 0.1, 6.0, 3.0)
    lib.pfEnable(A.PF_LIGHTING)
    lib.pfLightModel(A.PF_PHONG)
    lights = torch.randn((case["lights"], 3), generator=g, device="cuda")
    lights = (4.0 * lights / lights.norm(dim=1, keepdim=True)).cpu().numpy()
    tints = _uniform(g, (case["lights"], 3), 0.3, 1.0).cpu().numpy()
    for i in range(case["lights"]):
        lib.pfEnableLight(i)
        lib.pfLightfv(i, A.PF_POSITION, _hp(np.ascontiguousarray(lights[i])))
        lib.pfLightfv(i, A.PF_DIFFUSE, _hp(np.ascontiguousarray(tints[i])))
    lib.pfMaterialf(A.PF_FRONT_AND_BACK, A.PF_DIFFUSE, 0.9)
    lib.pfMaterialf(A.PF_FRONT_AND_BACK, A.PF_SPECULAR, 0.3)
    lib.pfMaterialf(A.PF_FRONT_AND_BACK, A.PF_SHININESS, 24.0)
    c.texture(tex, "nearest", "mirror")
    c.arrays(pos, v.float().contiguous(), uv)
    c.nverts = len(pos)
    c.opaque, c.additive = faces[~add].contiguous(), faces[add].contiguous()
    c.fog = A.PFhookfog(0.1, 6.0, 0.3, 0.9, A.PFcolor(160, 170, 190, 255))
    return c


def _phong_frame(c):
    lib = c.lib
    lib.pfMakeCurrent(c.ctx)
    lib.pfClear(COLOR_DEPTH)
    _elements(c, c.opaque)
    lib.pfEnable(A.PF_BLEND)
    lib.pfBlendFunc(A.PF_BLEND_ADD)
    _elements(c, c.additive)
    lib.pfDisable(A.PF_BLEND)
    lib.pfPostProcessDevice(A.PF_HOOK_FOG_LINEAR, C.c_void_p(C.addressof(c.fog)), C.sizeof(c.fog))
    lib.pfFinish()
    return c.buf


def _batch_sizes(case):
    """Sides and triangle counts of a batch's contexts: sides evenly from 64
    up, counts lognormal (sigma 1) by quantile, paired at random."""
    n = case["contexts"]
    q = torch.linspace(0.5 / n, 1 - 0.5 / n, n, dtype=torch.float64)
    counts = (case["tri_median"] * torch.exp(math.sqrt(2.0) * torch.erfinv(2 * q - 1))).clamp(100, 50000).int().tolist()
    sides = [64 * (1 + i % (case["max_side"] // 64)) for i in range(n)]
    p = np.random.default_rng(n).permutation(n)
    return [sides[i] for i in p], counts


class _BatchHandle:
    def __init__(self, lib):
        self.lib, self.b = lib, lib.pfgbBatchCreate()

    def __del__(self):
        self.lib.pfgbBatchDelete(self.b)


def _batch_state(case, seed, lib):
    g = _gen(seed)
    s = _State()
    s.batch, s.contexts = _BatchHandle(lib), []
    sides, counts = _batch_sizes(case)
    modes = list(BLENDS)
    for i, (side, n) in enumerate(zip(sides, counts)):
        c = _Context(lib, side, side)
        m = 3 * n
        lib.pfEnable(A.PF_DEPTH_TEST)
        lib.pfDepthFunc(A.PF_LESS)
        lib.pfClearDepth(1.0)
        blend = BLENDS[modes[i % 4]]
        if blend is not None:
            lib.pfEnable(A.PF_BLEND)
            lib.pfBlendFunc(blend)
        c.texture(_bytes(g, (256, 256)), list(FILTERS)[i // 4 % 2], list(WRAPS)[i // 8 % 3])
        c.arrays(torch.cat([_uniform(g, (m, 2), -1.0, 1.0), _uniform(g, (m, 1), 0.1, 0.9)], -1), None,
                 _uniform(g, (m, 2), 0.0, 2.0), _bytes(g, (m,)))
        c.nverts = m
        s.contexts.append(c)
    return s


def _batch_frame(s):
    lib = s.batch.lib
    lib.pfgbBatchBegin(s.batch.b)
    for c in s.contexts:
        lib.pfMakeCurrent(c.ctx)
        lib.pfClear(COLOR_DEPTH)
        lib.pfDrawArrays(A.PF_TRIANGLES, 0, c.nverts)
    lib.pfgbBatchEnd(s.batch.b)
    return [c.buf for c in s.contexts]


# ---------------------------------------------------------------------------
# differentiable renderer
# ---------------------------------------------------------------------------
def _grad_geometry(case):
    v, f = _icosphere(case["subdiv"])
    u = 0.5 + np.arctan2(v[:, 2], v[:, 0]) / (2 * np.pi)
    t = 0.5 - np.arcsin(np.clip(v[:, 1], -1, 1)) / np.pi
    eyes = fibonacci_sphere(case["views"], 3.0)
    proj = perspective(60.0, case["width"] / case["height"], 0.1, 100.0)
    mvp = np.stack([(look_at(e) @ proj).reshape(16) for e in eyes]).astype(np.float32)
    pos = v.astype(np.float32)
    return Mesh(pos, pos.copy(), np.stack([u, t], 1).astype(np.float32), f.astype(np.uint32)), mvp, eyes.astype(np.float32)


def _grad_params(case, seed):
    """Texture, vertex colours and alphas, material, light; and dLoss/dImage."""
    g, nv = _gen(seed), 10 * 4 ** case["subdiv"] + 2
    light = torch.randn(3, generator=g, device="cuda")
    light[1] = light[1].abs() + 0.5
    params = [_smooth(g, case["texture"], 4), _uniform(g, (nv, 3), 0.3, 1.0), _uniform(g, (nv,), 0.6, 1.0),
              torch.tensor([0.8, 0.5, 32.0], device="cuda"), light / light.norm()]
    shape = (case["views"], case["height"], case["width"], 3)
    d_image = torch.randn(shape, generator=g, device="cuda") / math.sqrt(np.prod(shape)) if case["backward"] else None
    return params, d_image


def _grad_state(case, seed):
    s = _State()
    mesh, mvp, eyes = _grad_geometry(case)
    s.scene = GradScene(mesh, mvp, eyes, case["width"], case["height"], (case["texture"], case["texture"]),
                        filter=FILTERS[case["filt"]], wrap=WRAPS[case["wrap"]], cull=1, ambient=0.2)
    s.params, s.d_image = _grad_params(case, seed)
    for p in s.params:
        p.requires_grad_(case["backward"])
    return s


def _grad_pass(s):
    image = s.scene.render(*s.params)
    if s.d_image is None:
        return [image]
    return [image, *torch.autograd.grad(image, s.params, s.d_image)]


# ---------------------------------------------------------------------------
def prepare(case, seed):
    lib, kind = load_library(), case["kind"]
    if kind == "grad":
        s = _grad_state(case, seed)
    else:
        s = _State()
        if kind == "static":
            s.pos, s.col, s.mvp = _static_inputs(case, seed)
            s.color = torch.zeros((case["height"], case["width"]), dtype=torch.int32, device="cuda")
            s.depth = torch.zeros((case["height"], case["width"]), device="cuda")
        elif kind == "batch":
            s = _batch_state(case, seed, lib)
        else:
            s.context = {"soup": _soup_state, "sphere": _sphere_state, "phong": _phong_state}[kind](case, seed, lib)
    s.case, s.lib = case, lib
    torch.cuda.synchronize()            # the pf* kernels run on streams of their own
    return s


def run(state):
    case = state.case
    kind = case["kind"]
    if kind == "static":
        state.color.fill_(0)
        state.depth.fill_(STATIC_FAR)
        rc = state.lib.pfgbDrawTrianglesStatic(
            _dp(state.pos), _dp(state.col), case["ntris"], _hp(state.mvp), _dp(state.color), _dp(state.depth),
            case["width"], case["height"], A.PF_LESS, 1, C.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc:
            raise RuntimeError(f"pfgbDrawTrianglesStatic: {rc}")
        return {"color": state.color, "depth": state.depth}
    if kind == "soup":
        return _soup_frame(state.context, case["ntris"])
    if kind == "sphere":
        return _sphere_frame(state.context)
    if kind == "phong":
        return _phong_frame(state.context)
    if kind == "batch":
        return _batch_frame(state)
    return _grad_pass(state)


def work(case):
    """Bytes: inputs read once, images written once.  Flops: about 60 per
    transformed vertex and 30 per covered pixel (weights, depth, colour),
    250 per pixel and light of per-fragment lighting."""
    k = case["kind"]
    if k == "batch":
        sides, counts = _batch_sizes(case)
        verts = 3 * sum(counts)
        frags = sum(0.5 * SOUP_AREA * s * s * n for s, n in zip(sides, counts))
        return {"bytes": verts * 24 + sum(4 * s * s + 256 * 256 * 4 for s in sides), "flops": 60.0 * verts + 30.0 * frags}
    pixels = case["width"] * case["height"]
    if k == "static":
        n = case["ntris"]
        return {"bytes": n * 48 + 8 * pixels, "flops": 180.0 * n + 30.0 * 0.5 * n * pixels * 0.0009}
    if k == "soup":
        n = case["ntris"]
        return {"bytes": n * 3 * (16 + (8 if case["texture"] else 0)) + case["texture"] ** 2 * 4 + 8 * pixels,
                "flops": 180.0 * n + 30.0 * 0.5 * n * SOUP_AREA * pixels}
    if k == "sphere":
        nv, nt = (case["rings"] + 1) * (case["segments"] + 1), 2 * case["rings"] * case["segments"]
        return {"bytes": nv * 20 + nt * 12 + case["texture"] ** 2 * 4 + FORMATS[case["format"]][2] * pixels,
                "flops": 120.0 * nv + 30.0 * 2 * 0.29 * case["height"] ** 2}
    nv, nt = 10 * 4 ** case["subdiv"] + 2, 20 * 4 ** case["subdiv"]
    if k == "phong":
        disc = 0.29 * case["height"] ** 2
        return {"bytes": nv * 32 + nt * 12 + case["texture"] ** 2 * 4 + 4 * pixels,
                "flops": 60.0 * nv + (30.0 + 250.0 * case["lights"]) * disc}
    views, disc = case["views"], 0.29 * min(case["height"], case["width"]) ** 2
    one = {"bytes": nv * 32 + nt * 12 + nv * 16 + case["texture"] ** 2 * 16 + 12 * pixels * views,
           "flops": views * (100.0 * nv + 80.0 * disc)}
    if case["backward"]:
        one = {"bytes": 2 * one["bytes"], "flops": 3 * one["flops"]}
    return one


# ---------------------------------------------------------------------------
# the same results in 64 bits: coverage from the integer corners the pipeline
# defines, depth and shading in double precision
# ---------------------------------------------------------------------------
def _corners(pos, m, w, h, perspective_divide):
    """Clip positions (float64) and integer pixel corners (from float32, as
    they are defined) of points under the row-vector matrix m."""
    m32 = torch.as_tensor(m, device="cuda", dtype=torch.float32)
    def clip(p, mm):
        return [((mm[i] * p[..., 0] + mm[4 + i] * p[..., 1]) + mm[8 + i] * p[..., 2]) + mm[12 + i] for i in range(4)]
    h32, h64 = clip(pos, m32), clip(pos.double(), m32.double())
    inv = 1.0 / h32[3] if perspective_divide else torch.ones_like(h32[3])
    sx = ((h32[0] * inv + 1.0) * 0.5 * float(w - 1)) + 0.5
    sy = ((1.0 - h32[1] * inv) * 0.5 * float(h - 1)) + 0.5
    return h32, h64, sx.trunc().long(), sy.trunc().long()


def _exact_depth(pos, m, w, h, perspective_divide, clear):
    """Nearest depth of front-facing triangles (T, 3, 3), LESS."""
    _, hc, x, y = _corners(pos, m, w, h, perspective_divide)
    z = 1.0 / hc[2] if perspective_divide else hc[2]
    area = (x[:, 1] - x[:, 0]) * (y[:, 2] - y[:, 0]) - (x[:, 2] - x[:, 0]) * (y[:, 1] - y[:, 0])
    keep = area < 0
    x, y, z, area = x[keep], y[keep], z[keep], area[keep]
    py, px = torch.meshgrid(torch.arange(h, device="cuda"), torch.arange(w, device="cuda"), indexing="ij")
    px, py = px.reshape(1, -1), py.reshape(1, -1)
    best = torch.full((h * w,), float(clear), dtype=torch.float64, device="cuda")
    step = max(1, 20_000_000 // (h * w))
    for b in range(0, len(x), step):
        X, Y, Z = x[b:b + step, :, None], y[b:b + step, :, None], z[b:b + step, :, None]
        ws = [(px - X[:, i]) * (Y[:, j] - Y[:, i]) + (py - Y[:, i]) * (X[:, i] - X[:, j]) for i, j in ((1, 2), (2, 0), (0, 1))]
        box = (px >= X.amin(1)) & (px < X.amax(1)) & (py >= Y.amin(1)) & (py <= Y.amax(1))
        cover = box & (ws[0] >= 0) & (ws[1] >= 0) & (ws[2] >= 0) & ((ws[0] | ws[1] | ws[2]) > 0)
        total = (ws[0] + ws[1] + ws[2]).double()
        d = total / (ws[0] * Z[:, 0] + ws[1] * Z[:, 1] + ws[2] * Z[:, 2])
        best = torch.minimum(best, torch.where(cover, d, float("inf")).amin(0))
    return best.reshape(h, w)


def _texel_index(u, size, wrap):
    """Texel column of float32 coordinates, as the sampler rounds them."""
    if wrap == "repeat":
        return ((u - u.trunc()) * float(size - 1)).round().abs().long()
    if wrap == "mirror":
        u = u.abs()
        u = u - torch.floor(u / 2.0) * 2.0
        u = torch.where(u > 1.0, 1.0 - (u - 1.0), u)
    else:
        u = u.clamp(0.0, 1.0)
    return (u * float(size - 1) + 0.5).round().long()


def _exact_grad(case, seed):
    mesh, mvp, eyes = _grad_geometry(case)
    params, d_image = _grad_params(case, seed)
    tex, col, alpha, mat, light = ps = [p.double().requires_grad_(case["backward"]) for p in params]
    W, H, V, ts = case["width"], case["height"], case["views"], case["texture"]
    pos, faces = _dev(mesh.positions), _dev(mesh.indices.astype(np.int64))
    uv32, nv = _dev(mesh.texcoords), len(mesh.positions)
    # covered (pixel, triangle) pairs of every view, in submission order
    frags = []
    for v in range(V):
        h32, h64, x, y = _corners(pos, mvp[v], W, H, True)
        x, y = x[faces], y[faces]
        area = (x[:, 1] - x[:, 0]) * (y[:, 2] - y[:, 0]) - (x[:, 2] - x[:, 0]) * (y[:, 1] - y[:, 0])
        t = torch.nonzero(area < 0)[:, 0]
        x, y = x[t], y[t]
        x0, x1, y0, y1 = x.amin(1).clamp(min=0), x.amax(1).clamp(max=W), y.amin(1).clamp(min=0), y.amax(1).clamp(max=H - 1)
        bw, bh = (x1 - x0).clamp(min=0), (y1 - y0 + 1).clamp(min=0)
        n = bw * bh
        r = torch.repeat_interleave(torch.arange(len(t), device="cuda"), n)
        k = torch.arange(len(r), device="cuda") - torch.repeat_interleave(n.cumsum(0) - n, n)
        px, py = x0[r] + k % bw[r], y0[r] + k // bw[r]
        X, Y = x[r], y[r]
        w = torch.stack([(px - X[:, i]) * (Y[:, j] - Y[:, i]) + (py - Y[:, i]) * (X[:, i] - X[:, j])
                         for i, j in ((1, 2), (2, 0), (0, 1))], 1)
        c = torch.nonzero((w >= 0).all(1) & (w > 0).any(1))[:, 0]
        r, w, pix, X, Y = r[c], w[c], py[c] * W + px[c], X[c], Y[c]
        # the depth test and texel choice are those of single precision
        f = faces[t[r]]
        wn = w.float() * (1.0 / w.sum(1).float())[:, None]
        hz = (1.0 / h32[2])[f]
        z = 1.0 / ((hz[:, 0] * wn[:, 0] + hz[:, 1] * wn[:, 1]) + hz[:, 2] * wn[:, 2])
        su = uv32[f] * hz[..., None]
        tu = ((su[:, 0] * wn[:, :1] + su[:, 1] * wn[:, 1:2]) + su[:, 2] * wn[:, 2:]) * z[:, None]
        b = w.double() / w.sum(1, keepdim=True)
        hz = (1.0 / h64[2])[f]
        tu64 = (uv32.double()[f] * hz[..., None] * b[..., None]).sum(1) / (hz * b).sum(1, keepdim=True)
        order = torch.argsort(pix, stable=True)
        frags.append([q[order] for q in (pix + v * W * H, z, f + v * nv, b, tu, tu64)])
    pix, z, f, b, tu, tu64 = [torch.cat(q) for q in zip(*frags)]
    del frags
    start = torch.ones_like(pix, dtype=torch.bool)
    start[1:] = pix[1:] != pix[:-1]
    first = torch.nonzero(start)[:, 0]
    rank = torch.arange(len(pix), device="cuda") - torch.repeat_interleave(first, torch.diff(first, append=torch.tensor([len(pix)], device="cuda")))
    # vertex lighting
    p, N = pos.double(), _dev(mesh.normals).double()
    N = N / N.norm(dim=1, keepdim=True)
    L = light / light.norm()
    E = torch.from_numpy(eyes).cuda().double()[:, None, :] - p
    Hh = L + E / E.norm(dim=2, keepdim=True)
    Hh = Hh / Hh.norm(dim=2, keepdim=True)
    nl, nh = (N @ L).clamp(min=0.0), (N * Hh).sum(2)
    spec = torch.where(nh > 0, nh.clamp(min=1e-300) ** mat[2], 0.0)
    lit = (col * mat[0] * (0.2 + nl)[:, None] + mat[1] * spec[..., None]).clamp(max=1.0)
    lit = torch.cat([lit, alpha[None, :, None].expand(V, nv, 1)], 2).reshape(V * nv, 4)
    image = torch.zeros((V * H * W, 3), dtype=torch.float64, device="cuda")
    nearest = torch.full((V * H * W,), float(np.finfo(np.float32).max), device="cuda")
    for k in range(int(rank.max()) + 1):
        i = torch.nonzero(rank == k)[:, 0]
        i = i[z[i] < nearest[pix[i]]]
        nearest[pix[i]] = z[i]
        c = (lit[f[i]] * b[i][..., None]).sum(1)
        at = [[_texel_index(tu[i][:, a] + d, ts, case["wrap"]) for a in (0, 1)] for d in (0.0, float(np.float32(1.0) / np.float32(ts)))]
        flat = tex.reshape(-1, 4)

        def texel(xx, yy):
            o = yy * ts + xx
            return flat[o.clamp(max=ts * ts - 1)] * (o < ts * ts)[:, None]
        s = texel(at[0][0], at[0][1])
        if case["filt"] == "bilinear":
            q = [(tu64[i][:, a] * ts - at[0][a]).clamp(0.0, 1.0)[:, None] for a in (0, 1)]
            top = s + q[0] * (texel(at[1][0], at[0][1]) - s)
            bottom = texel(at[0][0], at[1][1])
            bottom = bottom + q[0] * (texel(at[1][0], at[1][1]) - bottom)
            s = top + q[1] * (bottom - top)
        a = (s[:, 3] * c[:, 3])[:, None]
        old = image[pix[i]]
        image = image.index_put((pix[i],), a * s[:, :3] * c[:, :3] + (1.0 - a) * old)
    image = image.reshape(V, H, W, 3)
    if not case["backward"]:
        return [image]
    return [image.detach(), *torch.autograd.grad(image, ps, d_image.double())]


def exact(case, seed):
    if case["kind"] == "static":
        pos, _, m = _static_inputs(case, seed)
        return {"color": None, "depth": _exact_depth(pos, m, case["width"], case["height"], True, STATIC_FAR)}
    if case["kind"] == "soup":
        pos = torch.from_numpy(_soup_inputs(case, seed)[0]).cuda().reshape(-1, 3, 3)
        m = np.diag([1.0, 1.0, -1.0, 1.0]).astype(np.float32).reshape(16)
        return {"color": None, "depth": _exact_depth(pos, m, case["width"], case["height"], False, 1.0)}
    if case["kind"] == "grad":
        return _exact_grad(case, seed)
    return None
