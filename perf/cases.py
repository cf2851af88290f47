"""The work that users of the cloud framework have it do, as cases that can be timed and compared.

A renderer calls the cloud pass once a frame (whole frames, one pixel in 16 with the previous frame reprojected,
small probes, batches of views), darkens its meshes with the cloud shadow, runs the post chain to 8 bits, generates
the noise textures when a scene is loaded, and fits the learned sun cone.  Sizes are the ones this repository's
benchmark and tests use (3840x2160 down to 256x256), and odd ones beside them.  `exact` restates each pass in plain
torch, in 64 bits, with exact filter weights.
"""
import ctypes as C
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "project-marshmallow_gb300"))
import marshmallow as mm  # noqa: E402
from marshmallow import lib as L  # noqa: E402

F64 = torch.float64
FORMATS = {"unorm8": L.FORMAT_UNORM8, "fp16": L.FORMAT_FP16, "bf16": L.FORMAT_BF16}
NOISE = {"low_res": (L.NOISE_LOWRES, 3, 4), "hi_res": (L.NOISE_HIRES, 3, 4), "curl": (L.NOISE_CURL2D, 2, 2),
         "weather": (L.NOISE_WEATHER, 2, 4)}


def listed():
    return [
        # The headline workload: every pixel of a 3840x2160 frame.
        {"name": "march_uhd", "kind": "march", "width": 3840, "height": 2160, "pitch": 15.0, "sun": 30.0, "format": "unorm8"},
        # The same at the reference application's own size.
        {"name": "march_hd", "kind": "march", "width": 1920, "height": 1080, "pitch": 15.0, "sun": 30.0, "format": "unorm8"},
        # A window of odd size over FP16 density textures (the reduced-precision option), a low sun.
        {"name": "march_odd_fp16", "kind": "march", "width": 1367, "height": 771, "pitch": 10.0, "sun": 12.0, "format": "fp16"},
        # A small camera or light probe: the smallest launch, bound by the latency of its longest rays.
        {"name": "march_256", "kind": "march", "width": 256, "height": 256, "pitch": 15.0, "sun": 30.0, "format": "unorm8"},
        # The reference application's per-frame compute work: the previous frame reprojected, 1 pixel in 16 marched.
        {"name": "frame_hd", "kind": "frame", "width": 1920, "height": 1080, "pitch": 15.0, "sun": 30.0, "turn": 0.5},
        # Reprojection by itself (a paused or interleaved march), a quick turn of the camera.
        {"name": "reproject", "kind": "reproject", "width": 2880, "height": 1620, "pitch": 15.0, "sun": 30.0, "turn": 4.0},
        # Cloud shadows on the meshes of a 3840x2160 G-buffer, the lit colour darkened in place.
        {"name": "shadow_uhd", "kind": "shadow", "width": 3840, "height": 2160, "pitch": -12.0, "sun": 45.0},
        # The post chain of a finished frame to the swapchain's 8 bits, with the mesh layer.
        {"name": "post_uhd", "kind": "post", "width": 3840, "height": 2160, "pitch": 15.0, "sun": 20.0, "mesh": True},
        # The same passes one by one, for a host that keeps the reference's framebuffers.
        {"name": "post_passes_hd", "kind": "post_passes", "width": 1920, "height": 1080, "pitch": 15.0, "sun": 20.0},
        # A scene is loaded: the four noise textures of a seed at their default sizes.
        {"name": "textures", "kind": "noise", "low_res": 128, "hi_res": 32, "curl": 128, "weather": 512},
        # Fitting the learned sun cone: training steps, then predictions for held-out samples.
        {"name": "fit", "kind": "fit", "batch": 131072, "steps": 8, "held_out": 262144},
        # Cube-map faces and cameras of uneven size in one call.
        {"name": "views", "kind": "views", "faces": 512, "cameras": 6, "largest": 1280, "sun": 30.0},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def size(lo=192):
        w = log(lo, 3840)
        return w, max(96, min(2160, int(w / rng.choice([16 / 9, 16 / 9, 4 / 3, 1.0, 2.35]))))

    kind = rng.choice(["march", "march", "march", "frame", "reproject", "shadow", "post", "post_passes", "noise", "fit", "views"])
    pitch, sun = round(rng.uniform(5.0, 25.0), 2), round(rng.uniform(5.0, 85.0), 2)
    if kind == "noise":
        return {"kind": kind, "low_res": log(24, 128), "hi_res": log(16, 64), "curl": log(33, 256), "weather": log(65, 1024)}
    if kind == "fit":
        return {"kind": kind, "batch": 128 * log(8, 1024), "steps": rng.choice([2, 4, 8]), "held_out": log(1000, 262144)}
    if kind == "views":
        return {"kind": kind, "faces": log(64, 512), "cameras": rng.randint(1, 6), "largest": log(400, 1280), "sun": sun}
    w, h = size()
    case = {"kind": kind, "width": w, "height": h, "pitch": -pitch if kind == "shadow" else pitch, "sun": sun}
    if kind == "march":
        case["format"] = rng.choice(["unorm8", "unorm8", "fp16", "bf16"])
    elif kind in ("frame", "reproject"):
        case["turn"] = round(rng.uniform(0.05, 6.0), 2)
    elif kind == "post":
        case["mesh"] = rng.choice([True, False])
    return case


# ------------------------------------------------------------------------------------------------ inputs and passes

class State:
    """What a program keeps between calls; its handles are given back with it."""

    def __init__(self, **have):
        self.__dict__.update(have)

    def __del__(self):
        for name in ("textures", "renderer"):
            if name in self.__dict__:
                self.__dict__[name].close()
        if "net" in self.__dict__:
            L.load().mm_mlp_destroy(self.net)


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _smooth(g, h, w, channels, cells):
    """A smooth field in [0, 1] of `cells` bumps across."""
    low = torch.rand((1, channels, max(2, cells * h // max(1, w) + 2), cells + 2), generator=g, device="cuda")
    return torch.nn.functional.interpolate(low, size=(h, w), mode="bicubic", align_corners=True)[0].clamp(0, 1).permute(1, 2, 0)


def _cloud_frame(seed, h, w):
    """A frame as the march leaves it: sky with clouds, the sun's glow in alpha, depth +inf in clear sky."""
    g = _generator(seed)
    cover = (_smooth(g, h, w, 1, 24) * 1.6 - 0.4).clamp(0, 0.999)
    sky = torch.tensor([0.10, 0.22, 0.45], device="cuda") * (0.6 + 0.8 * torch.linspace(0, 1, h, device="cuda")[:, None, None])
    rgb = sky * (1 - cover) + (0.2 + 2.5 * _smooth(g, h, w, 1, 40)) * cover
    glow = _smooth(g, h, w, 1, 4) ** 3
    rgba = torch.cat([rgb, glow * (1 - cover)], 2).float().contiguous()
    depth = 1.0e5 + 8.0e4 * _smooth(g, h, w, 1, 16)[..., 0]
    return rgba, torch.where(cover[..., 0] > 0.02, depth, math.inf).float().contiguous()


def _camera(case, seed, w, h, **more):
    r = random.Random(seed)
    at = dict(yaw=r.uniform(0.0, 360.0), time=r.uniform(0.0, 2.0), pitch=case.get("pitch", 15.0), sun_elevation=case["sun"],
              phase=seed % 16)
    at.update(more)
    return mm.scene.uniforms(w, h, **at), at


def _target(h, w):
    return torch.zeros((h, w, 4), device="cuda"), torch.zeros((h, w), device="cuda")


def _samples(g, n):
    """Features as the deferred cone records hold them (heights, densities, fractions, sun direction) and a
    transmittance that depends on them."""
    x = torch.rand((n, 16), generator=g, device="cuda")
    x[:, 13:] = torch.nn.functional.normalize(x[:, 13:] - 0.3, dim=1)
    t = torch.exp(-2.0 * x[:, 1] * x[:, 2] - (1.5 * x[:, 3:9].mean(1)) * (1.2 - x[:, 0]) - 0.3 * torch.sin(9.0 * x[:, 10]))
    return x.bfloat16().contiguous(), t.clamp(0, 1).contiguous()


WARM_STEPS, WARM_LR, LR = 32, 1e-5, 1e-3


def _train(net, x, t, batch, steps, lr, history=None):
    L.check(L.load().mm_mlp_train(net, x.data_ptr(), t.data_ptr(), x.shape[0], batch, steps, lr,
                                  history.ctypes.data if history is not None else None,
                                  torch.cuda.current_stream().cuda_stream), "mm_mlp_train")


def prepare(case, seed):
    kind = case["kind"]
    if kind == "noise":
        bufs = {k: torch.empty((case[k],) * dims + (ch,), dtype=torch.uint8, device="cuda") for k, (_, dims, ch) in NOISE.items()}
        return State(kind=kind, seed=seed & 0xFFFFFFFF, bufs=bufs)
    if kind == "fit":
        g = _generator(seed)
        batch = case["batch"]
        x, t = _samples(g, 3 * batch)
        held, _ = _samples(g, case["held_out"])
        net = C.c_void_p()
        L.check(L.load().mm_mlp_create(seed & 0xFFFFFFFF, C.byref(net)), "mm_mlp_create")
        _train(net, x, t, batch, WARM_STEPS, WARM_LR)  # the learning rate is warmed up before the fit proper
        return State(kind=kind, net=net, x=x, t=t, held=held, y=torch.empty(held.shape[0], device="cuda"), batch=batch,
                     steps=case["steps"])
    renderer = mm.render.Renderer()
    if kind == "views":
        r = random.Random(seed)
        views = mm.scene.cubemap_views(case["faces"], time=r.uniform(0.0, 2.0), sun_elevation=case["sun"])
        for k in range(case["cameras"]):
            w = case["largest"] - 61 * k
            h = w * 9 // 16
            views.append((w, h, mm.scene.uniforms(w, h, yaw=r.uniform(0.0, 360.0), pitch=r.uniform(5.0, 25.0),
                                                  time=r.uniform(0.0, 2.0), sun_elevation=case["sun"])))
        return State(kind=kind, renderer=renderer, textures=mm.render.Textures(seed & 0xFFFFFFFF), views=views,
                     out=[_target(h, w) for w, h, _ in views])
    w, h = case["width"], case["height"]
    if kind == "shadow":
        u, _ = _camera(case, seed, w, h, eye=(0.0, 150.0, 0.0))
        world = mm.scene.terrain_gbuffer_cuda(u, w, h)
        lit = 0.1 + 0.9 * _smooth(_generator(seed), h, w, 4, 32)
        return State(kind=kind, renderer=renderer, textures=mm.render.Textures(seed & 0xFFFFFFFF), u=u, world=world,
                     lit=lit.float().contiguous(), color=torch.empty((h, w, 4), device="cuda"),
                     shadow=torch.empty((h, w), device="cuda"))
    u, at = _camera(case, seed, w, h)
    if kind == "march":
        textures = mm.render.Textures(seed & 0xFFFFFFFF)
        fmt = FORMATS[case["format"]]
        if fmt != L.FORMAT_UNORM8:
            textures.set_density_format(fmt)
        return State(kind=kind, renderer=renderer, textures=textures, u=u, fmt=fmt, out=_target(h, w))
    if kind in ("frame", "reproject"):
        before = mm.scene.uniforms(w, h, **dict(at, yaw=at["yaw"] - case["turn"]))
        u.camera_prev.view, u.camera_prev.proj = before.camera.view, before.camera.proj
        u.camera_prev.camera_position = before.camera.camera_position
        have = dict(kind=kind, renderer=renderer, u=u, prev=_cloud_frame(seed, h, w), out=_target(h, w))
        return State(textures=mm.render.Textures(seed & 0xFFFFFFFF), **have) if kind == "frame" else State(**have)
    # post chain and passes: the sun stands in the view, a little off the centre
    u, _ = _camera(case, seed, w, h, yaw=random.Random(seed).uniform(-25.0, 25.0))
    clouds, _ = _cloud_frame(seed, h, w)
    have = dict(kind=kind, renderer=renderer, u=u, clouds=clouds, out8=torch.empty((h, w, 4), dtype=torch.uint8, device="cuda"))
    if kind == "post":
        have["mesh"] = None
        if case["mesh"]:
            g = _generator(seed + 1)
            have["mesh"] = torch.cat([_smooth(g, h, w, 3, 32), (_smooth(g, h, w, 1, 8) > 0.7).float()], 2).contiguous()
    else:
        have.update(rays=torch.empty((h, w, 4), device="cuda"), blurred=torch.empty((h, w, 4), device="cuda"))
    return State(**have)


def run(s):
    kind = s.kind
    if kind == "march":
        s.renderer.march(s.u, s.textures, *s.out, density_format=s.fmt)
        return {"rgba": s.out[0], "depth": s.out[1]}
    if kind == "frame":
        s.renderer.frame(s.u, s.textures, s.prev, s.out)
        return {"rgba": s.out[0], "depth": s.out[1]}
    if kind == "reproject":
        s.renderer.reproject(s.u, s.prev, s.out)
        return {"rgba": s.out[0], "depth": s.out[1]}
    if kind == "views":
        s.renderer.march_batch(s.views, s.textures, s.out)
        return [{"rgba": c, "depth": d} for c, d in s.out]
    if kind == "shadow":
        s.color.copy_(s.lit)  # the mesh pass draws the lit colour anew each frame
        s.renderer.mesh_shadow(s.u, s.textures, s.world, shadow=s.shadow, rgba=s.color)
        return {"shadow": s.shadow, "color": s.color}
    if kind == "post":
        s.renderer.post_chain(s.u, s.clouds, s.out8, mesh=s.mesh)
        return {"out8": s.out8}
    if kind == "post_passes":
        s.renderer.god_rays(s.u, s.clouds, s.rays)
        s.renderer.radial_blur(s.u, s.rays, s.blurred)
        s.renderer.tonemap(s.blurred, s.out8)
        return {"rays": s.rays, "blurred": s.blurred, "out8": s.out8}
    lib, stream = L.load(), torch.cuda.current_stream().cuda_stream
    if kind == "noise":
        for k, (code, dims, _) in NOISE.items():
            b = s.bufs[k]
            n = b.shape[0]
            desc = L.NoiseDesc(code, s.seed, n, n, n if dims == 3 else 1)
            L.check(lib.mm_noise_fill(C.byref(desc), b.data_ptr(), b.numel(), stream), "mm_noise_fill")
        return s.bufs
    _train(s.net, s.x, s.t, s.batch, s.steps, LR)
    params = np.empty(lib.mm_mlp_param_count(), np.float32)
    L.check(lib.mm_mlp_get_params(s.net, params.ctypes.data, params.size), "mm_mlp_get_params")
    L.check(lib.mm_mlp_forward(s.net, s.held.data_ptr(), s.held.shape[0], s.y.data_ptr(), stream), "mm_mlp_forward")
    return {"params": params, "held_out": s.y}


def work(case):
    """Bytes: each input read once, each output written once.  Flops: of the arithmetic a pass needs by its
    definition; a marched ray takes about 56 coverage samples and 39 eroded ones (the 3840x2160 sweep's mean)."""
    kind = case["kind"]
    n = case.get("width", 0) * case.get("height", 0)
    scene = 128 ** 3 * 4 + 32 ** 3 * 4 + 128 * 128 * 2 + 512 * 512 * 4
    ray = 56 * 90 + 39 * 60 + 600
    if kind == "march":
        return {"bytes": 20 * n + scene, "flops": ray * n}
    if kind == "frame":
        return {"bytes": 40 * n + scene, "flops": ray * n / 16 + 130 * n}
    if kind == "reproject":
        return {"bytes": 40 * n, "flops": 130 * n}
    if kind == "views":
        n = 6 * case["faces"] ** 2 + sum((case["largest"] - 61 * k) ** 2 * 9 // 16 for k in range(case["cameras"]))
        return {"bytes": 20 * n + scene, "flops": ray * n}
    if kind == "shadow":  # the colour drawn anew and darkened, the position read, the shadow written
        return {"bytes": (16 + 16 + 16 + 4) * n, "flops": 6 * 100 * n}
    if kind == "post":
        return {"bytes": (16 + 4 + (16 if case["mesh"] else 0)) * n, "flops": 300 * n}
    if kind == "post_passes":
        return {"bytes": (32 + 32 + 20) * n, "flops": 300 * n}
    if kind == "noise":  # nine to twelve octaves of 27 distances per 3D texel
        out = 4 * case["low_res"] ** 3 + 4 * case["hi_res"] ** 3 + 2 * case["curl"] ** 2 + 4 * case["weather"] ** 2
        return {"bytes": out, "flops": case["low_res"] ** 3 * 12 * 27 * 9 + case["hi_res"] ** 3 * 9 * 27 * 9}
    macs = 16 * 64 + 64 * 64 + 64 * 64 + 64
    return {"bytes": 36 * (case["batch"] * case["steps"] + case["held_out"]),
            "flops": 2 * macs * (3 * case["batch"] * case["steps"] + case["held_out"])}


# ------------------------------------------------------------------------------------------------ 64-bit restatement
# Vectors are (3, N) tensors.  Line numbers of the shaders stand beside the kernels; here only the formulas.

def _dot(a, b):
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]


def _normal(a):
    return a / _dot(a, a).sqrt()


def _col(*v):
    return torch.tensor(v, dtype=F64, device="cuda")[:, None]


def _remap(v, a, b, c, d):
    return c + (v - a) / (b - a) * (d - c)


def _remap01(v, a):
    return torch.nan_to_num((v - a) / (1 - a), nan=0.0).clamp(0, 1)


def _texels(textures, name):
    return torch.from_numpy(textures.host(name)).to("cuda", F64) / 255


def _fetch(t, *at):
    """LINEAR / REPEAT fetch of t (..., z, y, x, channel) at normalized (u, v[, w])."""
    dims = t.shape[:-1][::-1]  # x, y[, z]
    flat = t.reshape(-1, t.shape[-1])
    corners = [(0, None)]
    stride = 1
    for n, u in zip(dims, at):
        x = u * n - 0.5
        i = x.floor()
        a = x - i
        i = i.long()
        lo, hi = i.remainder(n) * stride, (i + 1).remainder(n) * stride
        corners = [(c + e, f if w is None else w * f) for c, w in corners for e, f in ((lo, 1 - a), (hi, a))]
        stride *= n
    return sum(flat[c] * w[:, None] for c, w in corners).T


class _Scene:
    R, THICK = 1.0e6, 20000.0

    def __init__(self, u, textures):
        self.u = u
        self.tex = {k: _texels(textures, k) for k in ("weather", "curl", "low_res", "hi_res")}
        self.cam = _col(*u.camera.camera_position[:3])
        self.centre = _col(u.camera.camera_position[0], -self.R * 0.995, u.camera.camera_position[2])
        self.sun = _normal(_col(*u.sun.direction_basis[4:7]))
        self.wind, self.time = _col(*u.sky.wind[:3]), u.sky.wind[3]
        basis = torch.tensor(list(u.sun.direction_basis), dtype=F64, device="cuda").reshape(4, 4)[:3, :3]
        taps = _col(0, .6, 0), _col(0, .5, .05), _col(.1, .75, 0), _col(.2, 2.5, .3), _col(0, 6, 0), _col(-.1, 1, -.2)
        self.taps = [basis.T @ v for v in taps]

    def geo(self, pos):
        d = pos - self.centre
        rh = ((_dot(d, d).sqrt() - self.R).abs() / self.THICK).clamp(0, 1)
        return rh, pos + 20 * (self.wind + rh * _col(0.1, 0.05, 0.0)) * (self.time + rh * 200)

    def test(self, rh, sp):
        proj = self.R * _normal(sp - self.centre) + self.centre - self.cam
        info = _fetch(self.tex["weather"], 9e-6 * proj[0], 9e-6 * proj[2])
        dn = _fetch(self.tex["low_res"], 2e-5 * sp[0], 2e-5 * sp[1], 2e-5 * sp[2])
        kind = info[2]
        up = rh / 0.2
        cumulus = (up * _remap(rh, 0.7, 0.9, 1, 0)).clamp(min=0)
        strato = (up * _remap(rh, 0.2, 0.7, 1, 0)).clamp(min=0)
        stratus = (rh / 0.1 * _remap(rh, 0.2, 0.3, 1, 0)).clamp(min=0)
        d1 = torch.lerp(stratus, strato, (2 * kind).clamp(0, 1))
        d2 = torch.lerp(strato, cumulus, (2 * kind - 1).clamp(0, 1))
        density = torch.lerp(d1, d2, kind) * _remap01(dn[0], 0.3)
        cover = rh ** _remap(info[0].clamp(max=0.85), 0.7, 0.8, 1, 0.8).clamp(0.8, 1)
        erosion = _remap01(0.625 * dn[1] + 0.25 * dn[2] + 0.125 * dn[3], cover)
        return torch.where(density < 1e-4, 0.0, _remap01(density, erosion))

    def hires(self, rh, sp, strength, low):
        c = _fetch(self.tex["curl"], 1e-4 * sp[0], 1e-4 * sp[2])
        q = sp + 1.9 * strength * torch.stack([2 * c[0] - 1, 2 * c[1] - 1, -torch.ones_like(c[0])])
        dn = _fetch(self.tex["hi_res"], 4e-4 * q[0], 4e-4 * q[1], 4e-4 * q[2])
        e = 0.625 * dn[0] + 0.25 * dn[1] + 0.125 * dn[2]
        return _remap01(low, torch.lerp(e, 1 - e, (10 * rh).clamp(0, 1)))

    def shell(self, rd, w):
        ro = (self.cam - self.centre) / w
        a, b, c = _dot(rd, rd), 2 * _dot(rd, ro), _dot(ro, ro) - 0.25
        disc = b * b - 4 * a * c
        s = disc.clamp(min=0).sqrt()
        t = (-s - b) / a * 0.5
        t = torch.where(t < 0, (s - b) / a * 0.5, t)
        q = (ro + rd * t) * w + self.centre - ro
        return torch.where((disc >= 0) & (t >= 0), _dot(q, q).sqrt(), 0.0)

    def sky(self, rd):
        u = self.u
        beta_r, beta_m, e = _col(*u.sky.beta_r[:3]), _col(*u.sky.beta_v[:3]), u.sun.intensity
        zenith = rd[1].clamp(min=0).acos()
        inverse = 1 / (zenith.cos() + 0.15 * (93.885 - zenith * 180 / 3.14159265) ** -1.253)
        fex = (-beta_r * 8.4e3 * inverse + beta_m * 1.25e3 * inverse).exp()
        cos = _dot(self.sun, rd)
        betas = (beta_r * 0.05968310365946075 * (1 + (cos * 0.5 + 0.5) ** 2) + beta_m * self.phase(cos, u.sky.mie_directional)) / (beta_r + beta_m)
        dark = min(1.0, max(0.0, (1 - float(self.sun[1])) ** 5))
        light = (e * betas * (1 - fex)) ** 1.5 * torch.lerp(torch.ones_like(fex), (e * betas * fex) ** 0.5, dark)
        return (light + 0.1 * fex) * 0.04 + _col(0, 0.0003, 0.00075)

    @staticmethod
    def phase(cos, g):
        return 0.07957747154594767 * (1 - g * g) / (1 - 2 * g * cos + g * g) ** 1.5

    def march(self, width, height, px, py):
        """rgba (N, 4) and depth (N) of the pixels (px, py) of a width x height frame, the sun above the horizon."""
        u = self.u
        v = list(u.camera.view)
        aspect, tan = u.camera.camera_params[0], u.camera.camera_params[1]
        sx, sy = 2 * px.to(F64) / width - 1, 2 * py.to(F64) / height - 1
        rd = _normal(-_col(v[2], v[6], v[10]) + aspect * tan * sx * _col(v[0], v[4], v[8]) - tan * sy * _col(v[1], v[5], v[9]))
        to_sun = _dot(self.sun, rd).clamp(min=0)
        edge = ((to_sun - 0.9999566769464484) / 0.00003).clamp(0, 1)
        disk = torch.maximum(edge * edge * (3 - 2 * edge), to_sun ** 768)
        bg = self.sky(rd)
        alpha = torch.maximum((0.18 * to_sun) ** 4, disk)
        accum, trans = torch.zeros_like(alpha), torch.ones_like(alpha)
        depth = torch.full_like(alpha, math.inf)
        t, t1 = self.shell(rd, 2 * self.R), self.shell(rd, 2 * self.R * 1.02)
        cos = _dot(rd, self.sun)
        glow = torch.maximum(self.phase(cos, 0.6), 0.7 * self.phase(cos, 0.89))
        ray = torch.nonzero((rd[1] >= 0) & (t < t1))[:, 0]
        now = dict(t=t[ray], t1=t1[ray], step=torch.full_like(t[ray], 0.05 * self.THICK), far=torch.ones_like(ray, dtype=torch.bool),
                   misses=torch.zeros_like(ray), steps=torch.zeros_like(ray), accum=accum[ray], trans=trans[ray], depth=depth[ray])
        d = rd[:, ray]
        while ray.numel():
            s = now
            pos = self.cam + s["t"] * d
            rh, sp = self.geo(pos)
            low = self.test(rh, sp)
            hit = low > 0
            turn, near = hit & s["far"], torch.nonzero(hit & ~s["far"])[:, 0]
            counted = ~hit  # samples that count as a step and are checked for the end
            s["misses"] = torch.where(hit, 0, s["misses"] + (~s["far"]).long())
            back = ~hit & ~s["far"] & (s["misses"] >= 10)
            if near.numel():
                step = s["step"][near]
                fine = self.hires(rh[near], sp[:, near], step, low[near])
                keep = fine >= 1e-4
                at, fine, step = near[keep], fine[keep], step[keep]
                counted[at] = True
                if at.numel():
                    shade = torch.zeros_like(fine)
                    for tap in self.taps:
                        h2, p2 = self.geo(pos[:, at] + 3 * step * tap)
                        l2 = self.test(h2, p2)
                        shade += torch.where(l2 > 0, self.hires(h2, p2, step, l2), 0.0)
                    beers = (-shade).exp()
                    beers = torch.lerp(beers, torch.maximum(beers, 0.7 * (-0.25 * shade).exp()), 0.5 - 0.5 * cos[ray[at]])
                    h = rh[at]
                    lit = 0.09 + low[at] ** _remap(h, 0.3, 0.85, 0.5, 2.0).clamp(0.5, 2.0)
                    lit = lit * _remap(h, 0.07, 0.34, 0.1, 1.0).clamp(0.1, 1.0) ** 0.8
                    s["trans"][at] = torch.lerp(lit * glow[ray[at]] * beers, s["trans"][at], s["accum"][at])
                    s["depth"][at] = torch.minimum(s["depth"][at], s["t"][at])
                    s["accum"][at] += fine
            full = counted & (s["accum"] > 0.99)
            s["steps"] += (counted & ~full).long()
            s["accum"] = torch.where(full, 1.0, s["accum"])
            s["t"] = torch.where(turn, s["t"] - s["step"], s["t"])
            s["step"] = torch.where(turn, s["step"] * 0.3, torch.where(back, s["step"] / 0.3, s["step"]))
            s["far"] = (s["far"] & ~turn) | back
            s["t"] = s["t"] + s["step"]
            live = ~full & (s["steps"] <= 100) & (s["t"] < s["t1"])
            over = torch.nonzero(~live)[:, 0]
            if over.numel():
                accum[ray[over]], trans[ray[over]], depth[ray[over]] = s["accum"][over], s["trans"][over], s["depth"][over]
                ray, d = ray[live], d[:, live]
                now = {k: x[live] for k, x in s.items()}
        up = rd[1] >= 0
        f = (rd[1] / 0.1).clamp(0, 1)
        cover = torch.where(up, accum * f * f * (3 - 2 * f), 0.0).clamp(max=0.999)
        cloud = _col(*u.sun.color[:3]) * (u.sun.intensity * trans.clamp(min=0) + 0.08 * bg * (-trans).exp())
        return torch.cat([torch.lerp(bg, cloud, cover), (alpha * (1 - cover))[None]]).T, depth


def _grid(w, h, x0=0, y0=0, every=1):
    y, x = torch.meshgrid(torch.arange(y0, h, every, device="cuda"), torch.arange(x0, w, every, device="cuda"), indexing="ij")
    return x.reshape(-1), y.reshape(-1)


def _exact_march(u, textures, w, h):
    rgba, depth = _Scene(u, textures).march(w, h, *_grid(w, h))
    return {"rgba": rgba.reshape(h, w, 4), "depth": depth.reshape(h, w)}


def _exact_reproject(u, prev, w, h):
    v, p = list(u.camera.view), list(u.camera_prev.view)
    aspect, tan = u.camera.camera_params[0], u.camera.camera_params[1]
    x, y = _grid(w, h)
    su, sv = x.to(F64) / w, y.to(F64) / h
    rd = _normal(-_col(v[2], v[6], v[10]) + aspect * tan * (2 * su - 1) * _col(v[0], v[4], v[8]) - tan * (2 * sv - 1) * _col(v[1], v[5], v[9]))
    cam = _col(*u.camera.camera_position[:3])
    centre = _col(u.camera.camera_position[0], -995000.0, u.camera.camera_position[2])
    ro = (cam - centre) / 2e6
    b, c = 2 * _dot(rd, ro), float(_dot(ro, ro)) - 0.25
    hit = (ro + rd * ((b * b - 4 * c).sqrt() - b) * 0.5) * 2e6 + centre  # the camera stands inside the sphere
    q = [p[r] * hit[0] + p[4 + r] * hit[1] + p[8 + r] * hit[2] + p[12 + r] for r in range(3)]
    ou, ov = q[0] / -q[2] / tan / aspect * 0.5 + 0.5, -q[1] / -q[2] / tan * 0.5 + 0.5
    rgba, depth = prev[0].to(F64).reshape(-1, 4), prev[1].to(F64).reshape(-1)

    def at(k):
        tx = ((ou - (ou - su) * k) * w).round().clamp(0, w - 1).long()
        return ((ov - (ov - sv) * k) * h).round().clamp(0, h - 1).long() * w + tx

    out = sum(rgba[at(k / 9 - 0.5)] for k in range(10)) / 10
    out[:, 3] = rgba[at(0.0), 3]
    return {"rgba": out.reshape(h, w, 4), "depth": depth[at(0.0)].reshape(h, w)}


def _exact_shadow(s):
    h, w = s.shadow.shape
    u, low, weather = s.u, _texels(s.textures, "low_res"), _texels(s.textures, "weather")
    covered = torch.nonzero(s.world[..., 3].reshape(-1) != 0)[:, 0]
    wc = s.world.reshape(-1, 4)[covered, :3].T.to(F64)
    v, db = list(u.camera.view), _col(*u.sun.direction_basis[4:7])
    light = _normal(sum(_col(v[4 * k], v[4 * k + 1], v[4 * k + 2]) * db[k] for k in range(3)))
    light = -light if float(light[1]) < -0.05 else light
    radius, thick = 5.0e5, 1.0e4
    cam = _col(*u.camera.camera_position[:3])
    centre = _col(u.camera.camera_position[0], -495000.0, u.camera.camera_position[2])
    ro = (wc - centre) / 1e6
    a, b, c = _dot(db, db), 2 * _dot(db, ro), _dot(ro, ro) - 0.25
    disc = b * b - 4 * a * c
    root = disc.clamp(min=0).sqrt()
    t = (-root - b) / a * 0.5
    t = torch.where(t < 0, (root - b) / a * 0.5, t)
    q = (ro + db * t) * 1e6 + centre - ro
    t = torch.where((disc >= 0) & (t >= 0), _dot(q, q).sqrt(), 0.0)
    wind, time = _col(*u.sky.wind[:3]), u.sky.wind[3]
    most = torch.zeros_like(t)
    for _ in range(6):
        pos = wc * 4 + light * t
        d = pos - centre
        rh = ((_dot(d, d).sqrt() - radius).abs() / thick).clamp(0, 1)
        pos = pos + 20 * (wind + rh * _col(0.0, 0.2, 0.0)) * (time + rh * 200)
        proj = radius * _normal(pos - centre) + centre - cam
        info, n = _fetch(weather, 1e-5 * proj[0], 1e-5 * proj[2]), _fetch(low, *(5.7e-5 * pos))
        strato = (rh / 0.2 * _remap(rh, 0.2, 0.7, 1, 0)).clamp(min=0)
        stratus = (rh / 0.1 * _remap(rh, 0.2, 0.3, 1, 0)).clamp(min=0)
        d1 = torch.lerp(stratus, strato, (2 * info[2]).clamp(0, 1))
        d2 = torch.lerp(strato, stratus, (2 * info[2] - 1).clamp(0, 1))
        density = torch.lerp(d1, d2, info[2]) * _remap01(n[0], 0.3)
        cover = rh ** _remap(info[0].clamp(max=0.85), 0.7, 0.8, 1, 0.6).clamp(0.6, 1)
        got = _remap01(density, _remap01(0.625 * n[1] + 0.25 * n[2] + 0.125 * n[3], cover))
        most = torch.where(most == 1, most, torch.maximum(most, torch.where(density < 1e-4, 0.0, got)))
        most = torch.where(most > 0.99, 1.0, most)
        t = t + 0.1 * thick
    shadow = torch.zeros(h * w, dtype=F64, device="cuda")
    shadow[covered] = most
    color = s.lit.to(F64).reshape(-1, 4)
    color[covered, :3] = (color[covered, :3] * (1 - 2 * most)[:, None]).clamp(min=0)
    color[covered, 3] = 1.0
    return {"shadow": shadow.reshape(h, w), "color": color.reshape(h, w, 4)}


def _exact_passes(s):
    u = s.u
    h, w = s.out8.shape[:2]
    proj, view = (torch.tensor(list(m), dtype=F64).reshape(4, 4).T for m in (u.camera.proj, u.camera.view))
    q = proj @ view @ torch.tensor(list(u.sun.location), dtype=F64)
    sun = float(q[0] / q[3]), float(q[1] / q[3])
    x, y = _grid(w, h)
    px, py = 2 * (x + 0.5).to(F64) / w - 1, 2 * (y + 0.5).to(F64) / h - 1

    def tap(plane, nx, ny):  # bilinear, clamped to the edge
        fx, fy = (0.5 * nx + 0.5) * w - 0.5, (0.5 * ny + 0.5) * h - 0.5
        x0, y0 = fx.floor(), fy.floor()
        ax, ay = fx - x0, fy - y0
        xs, ys = [(x0 + k).clamp(0, w - 1).long() for k in (0, 1)], [(y0 + k).clamp(0, h - 1).long() * w for k in (0, 1)]
        return torch.lerp(torch.lerp(plane[ys[0] + xs[0]], plane[ys[0] + xs[1]], ax),
                          torch.lerp(plane[ys[1] + xs[0]], plane[ys[1] + xs[1]], ax), ay)

    src = s.clouds.to(F64).reshape(-1, 4)
    dx, dy = (px - sun[0]) * 0.09375, (py - sun[1]) * 0.09375
    term = src[:, 3] * 0.5
    for k in range(8):
        term = term + tap(src[:, 3], px - (k + 1) * dx, py - (k + 1) * dy) * 0.5 * 0.125 * 0.99 ** k
    rays = src.clone()
    rays[:, 3] = term * 0.9
    blur = sum(tap(rays[:, 3], px + 1.5 * k * (sun[0] - px), py + 1.5 * k * (sun[1] - py)) * 1.1
               for k in (-.08, -.05, -.03, -.02, -.01, .01, .02, .03, .05, .08)) / 10
    light = torch.tensor(list(u.sun.color)[:3], dtype=F64, device="cuda") * u.sun.intensity
    out = torch.cat([light * blur[:, None] + 0.5 * rays[:, :3], torch.ones_like(blur)[:, None]], 1)
    return {"rays": rays.reshape(h, w, 4), "blurred": out.reshape(h, w, 4), "out8": None}


def _exact_fit(case, seed):
    g = _generator(seed)
    x, t = _samples(g, 3 * case["batch"])
    held, _ = _samples(g, case["held_out"])
    x, t, held = x.to(F64), t.to(F64), held.to(F64)
    net, n = C.c_void_p(), L.load().mm_mlp_param_count()
    first = np.empty(n, np.float32)
    L.check(L.load().mm_mlp_create(seed & 0xFFFFFFFF, C.byref(net)), "mm_mlp_create")  # the network's first weights
    L.load().mm_mlp_get_params(net, first.ctypes.data, n)
    L.load().mm_mlp_destroy(net)
    p = torch.from_numpy(first).to("cuda", F64)
    m, v = torch.zeros_like(p), torch.zeros_like(p)

    def forward(p, x):
        for o, i in ((64, 16), (64, 64), (64, 64)):
            wgt, bias, p = p[:o * i].reshape(o, i), p[o * i:o * i + o], p[o * i + o:]
            x = (x @ wgt.T + bias).relu()
        return torch.sigmoid(x @ p[:64] + p[64])

    cursor, k, batch = 0, 0, case["batch"]
    for steps, lr in ((WARM_STEPS, WARM_LR), (case["steps"], LR)):
        cursor = 0
        for _ in range(steps):
            cursor = 0 if cursor + batch > x.shape[0] else cursor
            p = p.detach().requires_grad_(True)
            loss = (forward(p, x[cursor:cursor + batch]) - t[cursor:cursor + batch]).square().mean()
            grad, = torch.autograd.grad(loss, p)
            k, cursor = k + 1, cursor + batch
            m, v = 0.9 * m + 0.1 * grad, 0.999 * v + 0.001 * grad * grad
            p = p.detach() - lr * (m / (1 - 0.9 ** k)) / ((v / (1 - 0.999 ** k)).sqrt() + 1e-8)
    return {"params": p.cpu().numpy(), "held_out": forward(p, held).detach()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "fit":
        return _exact_fit(case, seed)
    if kind in ("noise", "post"):
        return None  # bytes
    s = prepare(case, seed)
    if kind == "march":
        return _exact_march(s.u, s.textures, case["width"], case["height"])
    if kind == "views":
        return [_exact_march(u, s.textures, w, h) for w, h, u in s.views]
    if kind == "shadow":
        return _exact_shadow(s)
    if kind == "post_passes":
        return _exact_passes(s)
    w, h = case["width"], case["height"]
    out = _exact_reproject(s.u, s.prev, w, h)
    if kind == "frame":
        phase = int(s.u.sun.color[3])
        x0, y0 = phase % 4, phase // 4
        rgba, depth = _Scene(s.u, s.textures).march(w, h, *_grid(w, h, x0, y0, 4))
        out["rgba"][y0::4, x0::4] = rgba.reshape(-1, len(range(x0, w, 4)), 4)
        out["depth"][y0::4, x0::4] = depth.reshape(-1, len(range(x0, w, 4)))
    return out
