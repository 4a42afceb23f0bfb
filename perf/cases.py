"""The work a user of this framework has it do, as measurable cases.

A case is a dict of plain values; its "kind" names the entry points it goes through:

  frame      one ray-cast (or slicing) frame into device memory: set_view + render_device
  fit        forward with tape, image residual and adjoint of every view: a TF / filter fit step
  batch      several volumes x views in one persistent launch: batch_render
  licvolume  LIC-volume precompute and a frame that ray-casts it
  animation  a new field from device memory, then a direct-volume frame of it
  gradients  noise gradients (quantised RGBA) of a noise volume in device memory

`exact` restates each kind in 64 bits with torch alone.
"""
import math

import numpy as np
import torch
import torch.nn.functional as F

from vectorvisualization_gb300 import capi

F32 = np.float32


# --------------------------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------------------------
def _case(kind, **kw):
    c = dict(kind=kind, field="vortex", nx=64, ny=64, nz=64, storage="f32", noise="dense", mx=64, my=64, mz=64,
             w=256, h=256, integrator="heun", lb=32, lf=32, h_lic=0.01, spacing=1.0 / 128.0, filter="gaussian",
             illum="none", tf_index="magnitude", tf="default", freq=1.0, low_res=False, technique="raycast",
             schedule="queue", ortho=False, tilt=20.0, turn=30.0, distance=2.3, views=1, volumes=1)
    c.update(kw)
    return c


def _dims(prefix, *v):
    v = v * 3 if len(v) == 1 else v
    return {prefix + a: int(x) for a, x in zip("xyz", v)}


def listed():
    return [
        # the low-resolution preview the renderer draws while the view is being dragged: the
        # smallest call, where the launches count
        _case("frame", name="preview", w=128, h=128, low_res=True, tf_index="dir_z", **_dims("n", 64), **_dims("m", 64)),
        # the plain method: 64^3 ABC flow in FP32, sparse noise, Euler, orthographic
        _case("frame", name="abc_ortho", field="abc", noise="sparse", integrator="euler", lb=20, lf=20, filter="box",
              ortho=True, w=256, h=256, **_dims("n", 64), **_dims("m", 64)),
        # the mid-size lit frame, FP16 storage (the reference's own texel format)
        _case("frame", name="lit_f16", storage="f16", lb=40, lf=40, h_lic=0.005, spacing=1.0 / 256.0, illum="gradient",
              freq=4.0, w=1024, h=1024, **_dims("n", 256), **_dims("m", 256)),
        # the same volume at the default FP32 storage, a window half as wide
        _case("frame", name="lit_f32", storage="f32", lb=40, lf=40, h_lic=0.005, spacing=1.0 / 256.0, illum="gradient",
              freq=4.0, w=512, h=512, **_dims("n", 256), **_dims("m", 256)),
        # a measured data set: odd uneven extents, 8-bit storage, a noise file of another odd
        # size, uneven streamline lengths, a 16:9 window
        _case("frame", name="ragged_u8", storage="u8", lb=25, lf=38, h_lic=0.008, spacing=1.0 / 160.0, filter="cos2",
              freq=2.0, tf="random", w=853, h=481, tilt=-35.0, turn=75.0, **_dims("n", 181, 97, 133),
              **_dims("m", 100, 75, 90)),
        # the slicing technique, lit, BF16 storage
        _case("frame", name="slicing_bf16", field="spectral", technique="slicing", storage="bf16", lb=30, lf=30,
              filter="triangle", illum="gradient", w=800, h=600, tilt=10.0, turn=140.0, **_dims("n", 160), **_dims("m", 128)),
        # a batch of uneven volumes, several views each, in one launch
        _case("batch", name="batch", storage="f16", volumes=8, views=3, w=512, h=512, **_dims("m", 128)),
        # one step of a transfer-function / filter fit: four views, forward and adjoint
        _case("fit", name="fit", storage="f16", views=4, lb=30, lf=30, tf="random", w=512, h=512, distance=2.4,
              **_dims("n", 128), **_dims("m", 128)),
        # the large turbulence frame of an orbit: 512^3, RK4, lit, 2048^2
        _case("frame", name="orbit", field="spectral", storage="f16", integrator="rk4", lb=60, lf=60,
              h_lic=1.0 / 512.0, spacing=1.0 / 512.0, illum="gradient", schedule="static", tilt=25.0, turn=45.0,
              distance=2.2, w=2048, h=2048, **_dims("n", 512), **_dims("m", 512)),
        # LIC volume precomputed for a static view, then ray-cast
        _case("licvolume", name="licvolume", storage="f16", field="spectral", lb=30, lf=30, h_lic=0.005,
              spacing=1.0 / 256.0, w=1024, h=1024, **_dims("n", 256), **_dims("m", 256)),
        # the animation loop: the next time step (on the device already) and a direct-volume frame
        _case("animation", name="animation", storage="f16", technique="volume", spacing=1.0 / 512.0, w=1600, h=1200,
              **_dims("n", 512)),
        # noise preparation: central-difference gradients of the turbulence orbit's noise
        _case("gradients", name="gradients", sobel=False, **_dims("m", 512)),
    ]


#: sample-steps (times four for FP32 texels) of the largest drawn ray-cast
_DRAW_STEPS = 1.5e10


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["frame"] * 6 + ["batch", "fit", "licvolume", "animation", "gradients"])
    cube = rng.random() < 0.5
    n = [log(33, 320)] * 3 if cube else [log(33, 320) for _ in range(3)]
    m = [rng.choice([32, 64, 128, 256])] * 3 if rng.random() < 0.6 else [log(20, 200) for _ in range(3)]
    w, h = log(64, 1200), log(64, 1200)
    steps = rng.choice([16, 20, 32, 40, 60])
    c = _case(kind, field=rng.choice(["abc", "vortex", "vortex", "spectral"]) if cube else rng.choice(["abc", "vortex"]),
              storage=rng.choice(["f32", "f16", "f16", "bf16", "u8"]), noise=rng.choice(["dense", "dense", "sparse"]),
              w=w, h=h, integrator=rng.choice(["euler", "heun", "heun", "heun", "rk4"]), lb=steps,
              lf=steps if rng.random() < 0.7 else log(5, 60), h_lic=rng.choice([0.004, 0.006, 0.01]),
              spacing=1.0 / rng.choice([96, 128, 200, 256]), filter=rng.choice(["box", "triangle", "cos2", "gaussian"]),
              illum=rng.choice(["none", "none", "gradient", "gradient", "zoeckler", "mallo"]),
              tf_index=rng.choice(["dir_z", "magnitude"]), tf=rng.choice(["default", "random"]),
              freq=rng.choice([1.0, 2.0, 4.0]), tilt=round(rng.uniform(-60, 60), 2), turn=round(rng.uniform(0, 360), 2),
              distance=round(rng.uniform(1.9, 2.8), 2), ortho=rng.random() < 0.15,
              low_res=kind == "frame" and rng.random() < 0.1, **_dims("n", *n), **_dims("m", *m))
    if kind == "frame":
        c["technique"] = rng.choice(["raycast"] * 4 + ["slicing", "volume"])
        c["schedule"] = rng.choice(["queue", "queue", "static"])
    elif kind == "batch":
        c.update(volumes=rng.randint(2, 10), views=rng.randint(1, 4), illum=rng.choice(["none", "gradient"]), ortho=False)
    elif kind == "fit":
        c.update(views=rng.randint(1, 4), illum=rng.choice(["none", "none", "gradient"]), tf="random", w=min(w, 600),
                 h=min(h, 600))
    elif kind == "licvolume":
        c.update(illum="none", storage=rng.choice(["f16", "u8"]))
    elif kind == "animation":
        c.update(technique="volume", illum="none")
    elif kind == "gradients":
        c.update(sobel=rng.random() < 0.3, **_dims("m", *[log(24, 400) for _ in range(3)]))
    while _units(c) > _DRAW_STEPS and min(c["w"], c["h"]) > 48:
        c["w"], c["h"] = c["w"] * 3 // 4, c["h"] * 3 // 4
    while kind == "licvolume" and _units(c) > _DRAW_STEPS:
        c.update({k: v * 3 // 4 for k, v in c.items() if k in ("nx", "ny", "nz")})
    return c


# --------------------------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------------------------
def _rand(gen, *shape):
    return torch.rand(*shape, generator=gen, device="cuda", dtype=torch.float32)


def _field(kind, n, gen):
    """(nz, ny, nx, 3) float32 vectors on the device."""
    nx, ny, nz = n
    z, y, x = (((torch.arange(k, device="cuda", dtype=torch.float32) + 0.5) / k) for k in (nz, ny, nx))
    if kind == "abc":  # Arnold-Beltrami-Childress flow, phases and amplitudes from the seed
        p, a = 2 * math.pi * _rand(gen, 3).cpu(), (1.0 + 0.8 * _rand(gen, 3)).cpu()
        X, Y, Z = (2 * math.pi * v + float(q) for v, q in zip((x, y, z), p))
        X, Y, Z = X[None, None, :], Y[None, :, None], Z[:, None, None]
        one = torch.ones(nz, ny, nx, device="cuda")
        return torch.stack([(a[0] * torch.sin(Z) + a[2] * torch.cos(Y)) * one,
                            (a[1] * torch.sin(X) + a[0] * torch.cos(Z)) * one,
                            (a[2] * torch.sin(Y) + a[1] * torch.cos(X)) * one], dim=-1).contiguous()
    if kind == "vortex":  # drift and eight Gaussian vortices
        c, R = _rand(gen, 8, 3).cpu(), (0.05 + 0.15 * _rand(gen, 8)).cpu()
        s = torch.randn(8, generator=gen, device="cuda").cpu()
        a = torch.randn(8, 3, generator=gen, device="cuda").cpu()
        a = a / a.norm(dim=1, keepdim=True)
        v = torch.zeros(nz, ny, nx, 3, device="cuda")
        v[..., 0] = 0.2
        for i in range(8):
            dx, dy, dz = x[None, None, :] - float(c[i, 0]), y[None, :, None] - float(c[i, 1]), z[:, None, None] - float(c[i, 2])
            g = float(s[i]) * torch.exp(-(dx * dx + dy * dy + dz * dz) / float(R[i]) ** 2)
            ax, ay, az = (float(q) for q in a[i])
            v[..., 0] += g * (ay * dz - az * dy)
            v[..., 1] += g * (az * dx - ax * dz)
            v[..., 2] += g * (ax * dy - ay * dx)
        return v
    # divergence-free random phases, E(k) ~ k^-5/3 on 2 <= k <= 64, unit RMS
    k1 = torch.fft.fftfreq(nx, 1.0 / nx, device="cuda")
    kr = torch.fft.rfftfreq(nx, 1.0 / nx, device="cuda")
    K = [kr[None, None, :], k1[None, :, None], k1[:, None, None]]
    k2 = K[0] ** 2 + K[1] ** 2 + K[2] ** 2
    amp = torch.where((k2 >= 4.0) & (k2 <= 4096.0), k2.clamp(min=1e-6) ** (-11.0 / 12.0), torch.zeros_like(k2))
    u = [torch.complex(torch.randn(k2.shape, generator=gen, device="cuda"),
                       torch.randn(k2.shape, generator=gen, device="cuda")) * amp for _ in range(3)]
    dot = (K[0] * u[0] + K[1] * u[1] + K[2] * u[2]) / k2.clamp(min=1e-6)
    v = torch.empty(nz, ny, nx, 3, device="cuda")
    for i in range(3):
        v[..., i] = torch.fft.irfftn(u[i] - K[i] * dot, s=(nz, ny, nx))
    return v / v.square().sum(-1).mean().sqrt()


def _noise(kind, m, gen):
    """(mz, my, mx) uint8 noise on the device."""
    shape = (m[2], m[1], m[0])
    if kind == "sparse":
        return ((_rand(gen, *shape) < 0.05) * 255).to(torch.uint8)
    return torch.randint(0, 256, shape, generator=gen, device="cuda", dtype=torch.uint8)


def _tf(kind, gen):
    i = np.arange(256, dtype=F32)
    if kind == "default":  # rgb identity, alpha and opacity max(0, i - 20)
        a = np.where(i < 20, 0, i - 20).astype(F32) / F32(255)
        return np.stack([i / F32(255)] * 3 + [a], axis=1), a.copy()
    k = _rand(gen, 8, 5).cpu().numpy()
    t = (np.arange(256) + 0.5) / 256
    v = np.stack([np.interp(t, np.linspace(0, 1, 8), k[:, q]) for q in range(5)], axis=1).astype(F32)
    return np.ascontiguousarray(v[:, :4]), np.ascontiguousarray(v[:, 4])


def _quat(tilt, turn):
    a, b = math.radians(tilt) / 2, math.radians(turn) / 2
    sx, cx, sy, cy = math.sin(a), math.cos(a), math.sin(b), math.cos(b)
    return tuple(float(F32(v)) for v in (sx * cy, cx * sy, sx * sy, cx * cy))  # tilt about x after turn about y


def _angles(c, k, gen_turns):
    """Tilt, turn and distance of view k of a case."""
    if c["views"] == 1 and c["kind"] != "batch":
        return c["tilt"], c["turn"], c["distance"]
    t = gen_turns[k % len(gen_turns)]
    return 80.0 * (t[0] - 0.5), 360.0 * t[1], c["distance"] * (0.9 + 0.2 * t[2])


def _view(c, tilt, turn, distance):
    v = capi.view_default()
    if c["ortho"]:
        v.projection = capi.ORTHOGRAPHIC
        return v  # along +z over the unit square
    for i, q in enumerate(_quat(tilt, turn)):
        v.quat[i] = q
    v.distance = distance
    return v


_ILLUM = {"none": capi.ILLUM_NONE, "gradient": capi.ILLUM_GRADIENT, "zoeckler": capi.ILLUM_ZOECKLER, "mallo": capi.ILLUM_MALLO}
_INTEG = {"euler": capi.EULER, "heun": capi.HEUN, "rk4": capi.RK4}


def _params(c):
    p = capi.params_default()
    p.step_size_vol, p.step_size_lic, p.freq_scale = c["spacing"], c["h_lic"], c["freq"]
    p.steps_backward, p.steps_forward = c["lb"], c["lf"]
    p.integrator, p.illum = _INTEG[c["integrator"]], _ILLUM[c["illum"]]
    p.tf_index = capi.TF_INDEX_MAGNITUDE if c["tf_index"] == "magnitude" else capi.TF_INDEX_DIR_Z
    p.low_res = int(c["low_res"])
    p.schedule = capi.SCHEDULE[c["schedule"]]
    p.technique = capi.TECHNIQUE[c["technique"]]
    return p


def _inputs(c, seed):
    """What a program reads from its files, in the order the seed gives it."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 13)
    d = {}
    if c["kind"] == "gradients":
        d["noise"] = _noise(c["noise"], (c["mx"], c["my"], c["mz"]), gen)
        return d
    d["turns"] = _rand(gen, 64, 3).cpu().tolist()
    d["tf"] = _tf(c["tf"], gen)
    if c["kind"] != "animation":
        d["noise"] = _noise(c["noise"], (c["mx"], c["my"], c["mz"]), gen)
    if c["kind"] == "batch":
        d["fields"], d["L"], d["filters"] = [], [], []
        u = _rand(gen, c["volumes"], 6).cpu().tolist()
        for q in u:  # extents 64, 80, ..., 192 per axis, L in 15..60, mixed filters
            n = [64 + 16 * min(8, int(9 * x)) for x in q[:3]]
            d["fields"].append(_field("abc" if q[3] < 0.5 else "vortex", n, gen))
            d["L"].append(15 + min(45, int(46 * q[4])))
            d["filters"].append(("box", "triangle", "cos2")[min(2, int(3 * q[5]))])
    else:
        n = (c["nx"], c["ny"], c["nz"])
        d["field"] = _field(c["field"], n, gen)
        if c["kind"] == "fit":
            d["target"] = 0.5 * _rand(gen, c["views"], c["h"], c["w"], 4)
    return d


class _Stream:
    """A program's own stream (batches do not run on the legacy default one)."""

    def __init__(self):
        self.s = torch.cuda.Stream()

    @property
    def ptr(self):
        return self.s.cuda_stream


def prepare(case, seed):
    c = dict(case)
    d = _inputs(c, seed)
    if c["kind"] == "gradients":
        return {"c": c, "noise": d["noise"], "rgba": torch.empty(*d["noise"].shape, 4, dtype=torch.uint8, device="cuda"),
                "mode": capi.NOISE_GRAD_SOBEL if c["sobel"] else capi.NOISE_GRAD_CENTRAL}
    ctx = capi.Context(0)
    s = {"c": c, "ctx": ctx}
    w, h = c["w"], c["h"]
    ctx.set_tf(*d["tf"])
    ctx.set_filter_table(capi.make_filter_table(c["filter"], 256))
    lit = c["illum"] == "gradient"
    noise = d.get("noise")
    if noise is None:
        noise = torch.zeros(8, 8, 8, dtype=torch.uint8)
    ctx.upload_noise(noise.cpu().numpy(), capi.NOISE_GRAD_CENTRAL if lit else capi.NOISE_SCALAR)
    p = _params(c)
    if c["kind"] == "batch":
        s["stream"] = _Stream()
        vids = [ctx.upload_field_device(f.data_ptr(), f.shape[2::-1], storage=c["storage"]) for f in d["fields"]]
        torch.cuda.synchronize()
        s["out"] = torch.empty(c["volumes"] * c["views"], h, w, 4, device="cuda")
        s["jobs"] = []
        for i, vid in enumerate(vids):
            q = capi.Params.from_buffer_copy(p)
            q.steps_backward = q.steps_forward = d["L"][i]
            table = capi.make_filter_table(d["filters"][i], 256)
            for k in range(c["views"]):
                j = i * c["views"] + k
                s["jobs"].append(capi.make_job(vid, s["out"][j].data_ptr(), w, h, _view(c, *_angles(c, j, d["turns"])),
                                               q, table))
        ctx.set_params(p)
        return s
    s["vid"] = ctx.upload_field_device(d["field"].data_ptr(), (c["nx"], c["ny"], c["nz"]), storage=c["storage"])
    s["views"] = [_view(c, *_angles(c, k, d["turns"])) for k in range(c["views"])]
    s["out"] = torch.empty(c["views"], h, w, 4, device="cuda")
    if c["kind"] == "fit":
        p.record_tape = 1
        s["target"], s["residual"] = d["target"], torch.empty(h, w, 4, device="cuda")
        s["grads"] = [torch.zeros(c["views"], k, device="cuda") for k in (1024, 256, c["lb"] + c["lf"] + 1)]
    if c["kind"] == "animation":
        s["field"] = d["field"]
    if c["kind"] == "licvolume":
        p.technique = capi.TECHNIQUE["licvolume"]
    ctx.set_params(p)
    torch.cuda.synchronize()
    return s


# --------------------------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------------------------
def run(s):
    c = s["c"]
    kind, w, h = c["kind"], c["w"], c["h"]
    if kind == "gradients":
        capi.noise_gradients_device(s["noise"].data_ptr(), (c["mx"], c["my"], c["mz"]), s["mode"], s["rgba"].data_ptr(),
                                    stream=torch.cuda.current_stream().cuda_stream)
        return s["rgba"]
    ctx = s["ctx"]
    if kind == "batch":
        ctx.batch_render(s["jobs"], s["stream"].ptr)
        return s["out"]
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "licvolume":
        ctx.compute_lic_volume(s["vid"], (c["nx"], c["ny"], c["nz"]))
    elif kind == "animation":
        ctx.update_field_device(s["vid"], s["field"].data_ptr(), (c["nx"], c["ny"], c["nz"]), stream)
    for k, view in enumerate(s["views"]):
        ctx.set_view(view)
        ctx.render_device(s["vid"], s["out"][k].data_ptr(), w, h, stream=stream)
        if kind == "fit":
            torch.sub(s["out"][k], s["target"][k], out=s["residual"])
            ctx.render_adjoint(s["vid"], s["residual"].data_ptr(), w, h, *(g[k].data_ptr() for g in s["grads"]),
                               stream=stream)
    return {"image": s["out"], "tf": s["grads"][0], "opacity": s["grads"][1], "taps": s["grads"][2]} if kind == "fit" else s["out"]


# --------------------------------------------------------------------------------------------
# rays, restated in double
# --------------------------------------------------------------------------------------------
def _geometry(n):
    n = np.array(n, np.float64)
    return n / n.max(), n.max() / n, n / n.max()  # extent, scale, scale_inv (unit slice distances)


def _rays(c, n, angles, w, h):
    """Affine pixel-ray coefficients (origin: o0 + u o1 + v o2, direction alike), clamped to t >= 0?"""
    ext = _geometry(n)[0]
    z = np.zeros(3)
    if c["ortho"]:
        return (z, np.array([1.0 / w, 0, 0]), np.array([0, 1.0 / h, 0])), (np.array([0, 0, 1.0]), z, z), False
    tilt, turn, distance = angles
    x, y, zq, q = _quat(tilt, turn)
    k = math.sqrt(x * x + y * y + zq * zq + q * q)
    x, y, zq, q = x / k, y / k, zq / k, q / k
    R = np.array([[1 - 2 * (y * y + zq * zq), 2 * (x * y - zq * q), 2 * (x * zq + y * q)],
                  [2 * (x * y + zq * q), 1 - 2 * (x * x + zq * zq), 2 * (y * zq - x * q)],
                  [2 * (x * zq - y * q), 2 * (y * zq + x * q), 1 - 2 * (x * x + y * y)]])
    t = math.tan(35.0 * math.pi / 360)
    a = w / h
    eye = R.T @ np.array([0, 0, float(F32(distance))]) + ext / 2
    return (eye, z, z), (R.T @ np.array([-a * t, -t, -1.0]), R.T @ np.array([2 * a * t / w, 0, 0]),
                         R.T @ np.array([0, 2 * t / h, 0])), True


def _march(c, n, angles, w, h, u, v, xp):
    """Origin, direction, box interval, hit mask of the pixel centres (u, v); xp is numpy or torch."""
    o, d, clamp = _rays(c, n, angles, w, h)
    ext = _geometry(n)[0]
    vec = (lambda a: a) if xp is np else (lambda a: torch.tensor(a, dtype=torch.float64, device="cuda"))
    O = vec(o[0]) + u[:, None] * vec(o[1]) + v[:, None] * vec(o[2])
    D = vec(d[0]) + u[:, None] * vec(d[1]) + v[:, None] * vec(d[2])
    inf = float("inf")
    zero = D == 0
    safe = xp.where(zero, xp.ones_like(D), D)
    t0, t1 = -O / safe, (vec(ext) - O) / safe
    lo, hi = xp.minimum(t0, t1), xp.maximum(t0, t1)
    bad = (zero & ((O < 0) | (O > vec(ext)))).any(1)
    lo, hi = xp.where(zero, xp.full_like(lo, -inf), lo), xp.where(zero, xp.full_like(hi, inf), hi)
    tn, tf = (lo.max(1), hi.min(1)) if xp is np else (lo.amax(1), hi.amin(1))
    hit = (tn < tf) & ~bad
    if clamp:
        hit = hit & (tf > 0)
        tn = xp.maximum(tn, xp.zeros_like(tn))
    return O, D, tn, tf, hit


def _scale_vol(c, n):
    """scaleVol as the lit shaders receive it: the inverse scale."""
    g = _geometry(n)
    return g[2] if c["illum"] != "none" and c["kind"] != "animation" else g[1]


def _samples(c, n, angles):
    """Ray samples of one frame without early termination, from a coarse grid of pixels."""
    w, h, k = c["w"], c["h"], 40
    u, v = (np.arange(k) + 0.5) * w / k, (np.arange(k) + 0.5) * h / k
    u, v = np.tile(u, k), np.repeat(v, k)
    O, D, tn, tf, hit = _march(c, n, angles, w, h, u, v, np)
    sv = _scale_vol(c, n)
    step = c["spacing"] * (2 if c["low_res"] else 1)
    dr = D / np.linalg.norm(D, axis=1, keepdims=True) * sv
    with np.errstate(all="ignore"):
        p = (O + np.where(hit, tn, 0.0)[:, None] * D) * sv
        far = np.where(dr == 0, np.inf, (np.where(dr > 0, 1.0, 0.0) - p) / dr).min(1)
    return float(np.where(hit, np.floor(np.maximum(far, 0) / step) + 1, 0).mean() * w * h)


#: share of a ray's samples marched before it turns opaque, as counted on the seeded inputs
_SHARE = {"default": 1.0, "random": 0.3}


def _frames(c):
    """(extents, L_b, L_f, samples) of every frame of a pass (the batch's volumes at their mean)."""
    lb, lf = (15, 15) if c["low_res"] else (c["lb"], c["lf"])
    n = (c["nx"], c["ny"], c["nz"])
    if c["kind"] == "batch":
        n, lb, lf = (128, 128, 128), 37, 37
    frames = c["volumes"] * c["views"] if c["kind"] == "batch" else c["views"]
    one = _samples(c, n, (c["tilt"], c["turn"], c["distance"]))
    return n, lb, lf, one * frames * _SHARE[c["tf"]]


def _units(c):
    """Sample-steps of a pass, FP32 texels counted four times (an upper estimate of its cost)."""
    if c["kind"] in ("gradients", "animation"):
        return 0.0
    n, lb, lf, samples = _frames(c)
    if c["kind"] == "licvolume":
        samples = n[0] * n[1] * n[2]
    if c["technique"] == "volume":
        return samples
    return samples * (lb + lf) * (4 if c["storage"] == "f32" else 1) * (2 if c["integrator"] == "rk4" else 1) * (
        3 if c["kind"] == "fit" else 1)


_TEXEL = {"f32": 16, "f16": 8, "bf16": 8, "u8": 4}


def work(case):
    """Bytes: every input read once, every output written once.  Flops: a field evaluation is a
    three-channel trilinear (42) and its slope (9), a noise tap 14 (56 with gradients) plus its
    weight, an integration step 12 per slope."""
    c = dict(case)
    mvox = c["mx"] * c["my"] * c["mz"]
    if c["kind"] == "gradients":
        return {"bytes": mvox * 5.0, "flops": mvox * (27 * 6.0 + (54 * 3 if c["sobel"] else 9) + 20)}
    n, lb, lf, samples = _frames(c)
    vox = n[0] * n[1] * n[2] * (c["volumes"] if c["kind"] == "batch" else 1)
    lit = c["illum"] == "gradient"
    frames = c["volumes"] * c["views"] if c["kind"] == "batch" else c["views"]
    image = c["w"] * c["h"] * 16.0 * frames
    texels = vox * float(_TEXEL[c["storage"]])
    k = {"euler": 1, "heun": 2, "rk4": 4}[c["integrator"]]
    step = k * (51 + 12) + (58.0 * 1.15 if lit else 16.0)
    if c["kind"] == "animation":
        return {"bytes": vox * 12.0 + texels + image, "flops": vox * 20.0 + samples * 80}
    if c["technique"] == "volume":
        return {"bytes": texels + image, "flops": samples * 80}
    noise = mvox * (4.0 if lit else 1.0)
    if c["kind"] == "licvolume":
        return {"bytes": texels + noise + vox * 4.0 + image, "flops": vox * (lb + lf) * step + samples * 120}
    flops = samples * ((lb + lf) * step + 150)
    if c["kind"] == "fit":  # the adjoint forms the tap gradients from the same noise taps
        return {"bytes": texels + noise + 3 * image, "flops": flops * 2}
    return {"bytes": texels + noise + image, "flops": flops}


# --------------------------------------------------------------------------------------------
# exact values
# --------------------------------------------------------------------------------------------
def _encode(xyz, storage):
    """Encoded texels (direction 0.5 v/|v| + 0.5, magnitude |v|/max) at the storage's precision, in double."""
    v = xyz
    ln = torch.sqrt(v[..., 0] * v[..., 0] + v[..., 1] * v[..., 1] + v[..., 2] * v[..., 2])
    ln = torch.where(ln < 1e-5, torch.zeros_like(ln), ln)
    t = torch.empty(*v.shape[:3], 4, device=v.device)
    for i in range(3):
        t[..., i] = torch.where(ln == 0, torch.full_like(ln, 0.5), 0.5 * v[..., i] / ln + 0.5)
    top = ln.max()
    t[..., 3] = (ln / top).clamp(0, 1) if float(top) > 0 else 0.0
    if storage == "f16":
        t = t.half()
    elif storage == "bf16":
        t = t.bfloat16()
    elif storage == "u8":
        return (torch.round(t * 255).clamp(0, 255).double() / 255)
    return t.double()


def _central(noise):
    """Quantised noise gradients of the central-difference branch and the noise, RGBA bytes / 255."""
    v = noise.double()
    mz, my, mx = v.shape
    g = []
    for d, size in ((2, mx), (1, my), (0, mz)):
        lo, hi = torch.roll(v, 1, d), torch.roll(v, -1, d)
        q = (hi - lo) * 0.5
        first, last = [slice(None)] * 3, [slice(None)] * 3
        first[d], last[d] = slice(0, 1), slice(size - 1, size)
        q[tuple(first)] = (hi - v)[tuple(first)]
        q[tuple(last)] = (v - lo)[tuple(last)]
        g.append(q)
    w = {(i, j, k): math.exp(-(i * i + j * j + k * k) / 5.0) for i in range(3) for j in range(3) for k in range(3)}
    total = sum(w.values())
    ax = [torch.arange(s, device=v.device) for s in (mz, my, mx)]
    bd = torch.minimum(torch.minimum(torch.minimum(ax[0], mz - 1 - ax[0])[:, None, None],
                                     torch.minimum(ax[1], my - 1 - ax[1])[None, :, None]),
                       torch.minimum(ax[2], mx - 1 - ax[2])[None, None, :])
    out = torch.empty(mz, my, mx, 4, device=v.device, dtype=torch.float64)
    sums = []
    for q in g:
        acc = torch.zeros_like(v)
        for (i, j, k), t in w.items():
            acc += t / total * torch.roll(q, (k, j, i), (0, 1, 2))
        # next to the border the window shrinks to its far corner, on the border to nothing
        corner = w[2, 2, 2] / total * torch.roll(q, (1, 1, 1), (0, 1, 2))
        sums.append(torch.where(bd >= 2, acc, torch.where(bd == 1, corner, torch.zeros_like(acc))))
    ln = torch.sqrt(sums[0] ** 2 + sums[1] ** 2 + sums[2] ** 2)
    for i in range(3):
        u = torch.where(ln < 1e-5, torch.zeros_like(ln), sums[i] / ln.clamp(min=1e-30))
        out[..., i] = torch.floor((u + 1) / 2 * 255) / 255
    out[..., 3] = v / 255
    return out


def _taps(kind, lb, lf):
    """Tap weights and inverse area of a 256-texel filter table (LINEAR, zero border)."""
    t = (np.arange(256) + 0.5) / 256
    d = 2 * t - 1
    f = {"box": np.ones(256), "triangle": 1 - np.abs(d), "cos2": np.cos(np.pi * d / 2) ** 2, "gaussian": np.exp(-4.5 * d * d)}[kind]
    tab = np.floor(f * 255 + 0.5)

    def at(s):
        u = min(max(s, 0.0), 1.0) * 256 - 0.5
        i = math.floor(u)
        return sum(wt * tab[q] / 255 for q, wt in ((i, 1 - (u - i)), (i + 1, u - i)) if 0 <= q < 256)

    w = [at(0.5 - 0.5 * j / lb) for j in range(lb, 0, -1)] + [at(0.5)] + [at(0.5 + 0.5 * j / lf) for j in range(1, lf + 1)]
    return np.array(w), 0.5 if kind == "box" else 0.5 * 256 * 255 / tab.sum()


class _Exact:
    """The ray-cast of one volume in 64 bits."""

    def __init__(self, c, texels, noise, tf, lb, lf, kind):
        self.c = c
        nz, ny, nx = texels.shape[:3]
        self.n = (nx, ny, nz)
        self.field = texels.permute(3, 0, 1, 2).contiguous()[None]
        if noise is not None:
            q = noise if noise.dim() == 4 else noise[..., None]
            q = F.pad(q.permute(3, 0, 1, 2)[None], (1, 1, 1, 1, 1, 1), mode="circular")
            self.noise, self.m = q.contiguous(), torch.tensor(noise.shape[2::-1] if noise.dim() == 3 else
                                                              [noise.shape[2], noise.shape[1], noise.shape[0]],
                                                              dtype=torch.float64, device="cuda")
        self.lit = c["illum"] == "gradient"
        self.rgba = torch.tensor(tf[0], dtype=torch.float64, device="cuda")
        self.opac = torch.tensor(tf[1], dtype=torch.float64, device="cuda")
        self.lb, self.lf = lb, lf
        taps, area = _taps(kind, lb, lf)
        self.taps = torch.tensor(taps.astype(F32), dtype=torch.float64, device="cuda")
        low = c["low_res"]
        self.step = float(F32(c["spacing"])) * (2 if low else 1)
        self.h = (1.0 / 64 if low else float(F32(c["h_lic"]))) * float(F32(0.3))
        self.freq = c["freq"] * (float(F32(0.7)) if low else 1.0)
        self.corr = self.step * 128
        self.scale = area / (lb + lf) * 30.0

    def fetch(self, p, channels=4):
        q = (2 * p - 1).view(1, 1, 1, -1, 3)
        v = self.field if channels == 4 else self.field[:, :channels]
        return F.grid_sample(v, q, mode="bilinear", padding_mode="border", align_corners=False)[0, :, 0, 0].t()

    def noise_at(self, p, tex=None, m=None):
        tex, m = (self.noise, self.m) if tex is None else (tex, m)
        s = p if (self.lit or tex is not self.noise) else p * self.freq
        u = (s - torch.floor(s)) * m + 0.5  # index in the padded volume
        q = (2 * u / (m + 1) - 1).view(1, 1, 1, -1, 3)
        return F.grid_sample(tex, q, mode="bilinear", padding_mode="border", align_corners=True)[0, :, 0, 0].t()

    def advance(self, p, f, sign):
        h = self.h * sign
        slope = lambda t: (2 * t[:, :3] - 1) * h  # noqa: E731
        k1 = slope(f)
        kind = self.c["integrator"]
        if kind == "euler":
            p = p + k1
        elif kind == "heun":
            p = p + 0.5 * (k1 + slope(self.fetch(p + k1, 3)))
        else:
            k2 = slope(self.fetch(p + 0.5 * k1, 3))
            k3 = slope(self.fetch(p + 0.5 * k2, 3))
            k4 = slope(self.fetch(p + k3, 3))
            p = p + (k1 + 2 * k2 + 2 * k3 + k4) / 6
        return p, self.fetch(p, 3)

    def lic(self, pos, f, each=False):
        """sum over taps of weight * noise, or every tap's noise."""
        n0 = self.noise_at(pos)
        acc, taps = n0 * self.taps[self.lb], {self.lb: n0}
        for sign, count in ((-1, self.lb), (1, self.lf)):
            p, s = pos, f[:, :3]
            for i in range(1, count + 1):
                p, s = self.advance(p, s, sign)
                v = self.noise_at(p)
                if each:
                    taps[self.lb + sign * i] = v
                else:
                    acc = acc + v * self.taps[self.lb + sign * i]
        return torch.stack([taps[i] for i in range(self.lb + self.lf + 1)], 1) if each else acc

    @staticmethod
    def table(t, s):
        u = (s * 256 - 0.5).clamp(-1, 256)
        i = torch.floor(u)
        a = u - i
        i0, i1 = i.long().clamp(0, 255), (i.long() + 1).clamp(0, 255)
        a = a[:, None] if t.dim() == 2 else a
        return t[i0] * (1 - a) + t[i1] * a

    def alpha(self, I, tfa, opac=None):
        al = self.table(self.opac if opac is None else opac, 1.3 * I) * tfa
        return 1 - (1 - al).clamp(min=0) ** self.corr

    def shade(self, il, tf, dr, opac=None):
        """Colour and alpha of a sample; il: (gradient sums,) intensity."""
        I = il[:, -1]
        al = self.alpha(I, tf[:, 3], opac)
        if not self.lit:
            return tf[:, :3] * I[:, None], al
        unit = lambda v: v / v.norm(dim=1, keepdim=True).clamp(min=1e-30)  # noqa: E731
        L = unit(torch.tensor([[0.5, 0.5, 1.5]], dtype=torch.float64, device="cuda"))
        V, N = unit(-dr), unit(-il[:, :3])
        ln = (L * N).sum(1, keepdim=True)
        R = unit(N * 2 * ln - L)
        sp = (R * V).sum(1, keepdim=True).clamp(0, 1) ** 40 * I[:, None]
        return tf[:, :3] * I[:, None] * (ln.clamp(0, 1) + float(F32(0.3))) + sp, al

    def setup(self, angles, rows):
        c, w, h = self.c, self.c["w"], self.c["h"]
        v, u = torch.meshgrid(torch.arange(*rows, device="cuda", dtype=torch.float64) + 0.5,
                              torch.arange(w, device="cuda", dtype=torch.float64) + 0.5, indexing="ij")
        return _march(c, self.n, angles, w, h, u.reshape(-1), v.reshape(-1), torch)

    def image(self, angles, licvol=None):
        c, w, h = self.c, self.c["w"], self.c["h"]
        out = torch.zeros(h, w, 4, dtype=torch.float64, device="cuda")
        band = max(1, 131072 // w)
        for y in range(0, h, band):
            rows = (y, min(h, y + band))
            O, D, tn, tf, hit = self.setup(angles, rows)
            ids = torch.nonzero(hit)[:, 0]
            if ids.numel():
                f = self.slices if c["technique"] == "slicing" else self.rays
                out[rows[0]:rows[1]].view(-1, 4)[ids] = f(O[ids], D[ids], tn[ids], tf[ids], licvol, angles)
        return out

    def rays(self, O, D, tn, tf, licvol, angles):
        c = self.c
        sv = torch.tensor(_scale_vol(c, self.n), device="cuda")
        pos = (O + tn[:, None] * D) * sv
        dr = D / D.norm(dim=1, keepdim=True) * sv
        dest = torch.zeros(pos.shape[0], 4, dtype=torch.float64, device="cuda")
        live = torch.arange(pos.shape[0], device="cuda")
        dvr = c["technique"] == "volume" or licvol is not None
        while live.numel():
            many = max(1, min(32, 400000 // live.numel()))
            k = torch.arange(many, device="cuda", dtype=torch.float64)
            p = (pos[live][:, None] + dr[live][:, None] * (self.step * k)[None, :, None])
            flat, d = p.reshape(-1, 3), dr[live].repeat_interleave(many, 0)
            inside = ((flat >= 0) & (flat <= 1)).all(1).view(-1, many)
            inside[:, 0] = True  # the entry sample is always taken; later blocks start inside
            run = inside.cumprod(1).bool()
            at = torch.nonzero(run.reshape(-1))[:, 0]
            f = self.fetch(flat[at])
            if c["technique"] == "volume":
                col, al = f[:, :3], self.table(self.rgba, f[:, 3])[:, 3]
            else:
                t = self.table(self.rgba, f[:, 3] if c["tf_index"] == "magnitude" else f[:, 2])
                if licvol is not None:
                    il = self.noise_at(flat[at], licvol, torch.tensor([float(v) for v in self.n], dtype=torch.float64, device="cuda"))
                else:
                    il = self.lic(flat[at], f)
                    il = torch.cat([il[:, :-1], il[:, -1:] * self.scale], 1)
                col, al = self.shade(il, t, d[at])
            src = torch.zeros(flat.shape[0], 4, dtype=torch.float64, device="cuda")
            src[at] = torch.cat([col * al[:, None], al[:, None]], 1)
            src = src.view(-1, many, 4)
            D4, alive = dest[live], torch.ones(live.numel(), dtype=torch.bool, device="cuda")
            for j in range(many):
                take = alive & run[:, j]
                new = ((1 - D4[:, 3:]) * src[:, j] + D4).clamp(0, 1)
                D4 = torch.where(take[:, None], new, D4)
                stop = (D4[:, 3] if dvr else src[:, j, 3]) > float(F32(0.95))
                alive = take & ~stop
            dest[live] = D4
            nxt = pos[live] + dr[live] * (self.step * many)
            pos[live] = nxt
            live = live[alive & ((nxt >= 0) & (nxt <= 1)).all(1)]
        return dest

    def slices(self, O, D, tn, tf, licvol, angles):
        ext = _geometry(self.n)[0]
        tilt, turn, distance = angles
        if self.c["ortho"]:
            dv = np.array([0, 0, 1.0])
        else:
            x, y, z, q = _quat(tilt, turn)
            R2 = np.array([2 * (x * z - y * q), 2 * (y * z + x * q), 1 - 2 * (x * x + y * y)])
            dv = R2 / (-distance - R2 @ (ext / 2))
        V = dv / np.linalg.norm(dv)
        depth = 2 * np.abs(V * ext / 2).sum()
        count = int(F32(depth) / F32(self.step)) + 1
        Vt, C = torch.tensor(V, device="cuda"), torch.tensor(ext / 2, device="cuda")
        vd, voc = D @ Vt, (O - C) @ Vt
        sv = torch.tensor(_scale_vol(self.c, self.n), device="cuda")
        dr = D / D.norm(dim=1, keepdim=True) * sv
        dest = torch.zeros(O.shape[0], 4, dtype=torch.float64, device="cuda")
        for i in range(count):
            ti = (-0.5 * depth + (i + 0.5) * depth / count - voc) / vd
            at = torch.nonzero((ti >= tn) & (ti <= tf) & (dest[:, 3] < 0.95))[:, 0]
            if not at.numel():
                continue
            p = (O[at] + ti[at, None] * D[at]) * sv
            f = self.fetch(p)
            t = self.table(self.rgba, f[:, 3])
            keep = torch.nonzero(t[:, 3] > 0.05)[:, 0]
            if not keep.numel():
                continue
            at, p, f, t = at[keep], p[keep], f[keep], t[keep]
            il = self.lic(p, f)
            il = torch.cat([il[:, :-1], il[:, -1:] * self.scale], 1)
            col, al = self.shade(il, t, dr[at])
            old = dest[at]
            dest[at] = ((1 - old[:, 3:]) * torch.cat([col * al[:, None], al[:, None]], 1) + old).clamp(0, 1)
        return dest

    def fit(self, angles, target):
        """Image and its gradients of 1/2 |image - target|^2 in TF, opacity and taps (unlit)."""
        c, w, h = self.c, self.c["w"], self.c["h"]
        out = torch.zeros(h, w, 4, dtype=torch.float64, device="cuda")
        rgba, opac, taps = (t.clone().requires_grad_(True) for t in (self.rgba, self.opac, self.taps))
        band = max(1, 24576 // w)
        sv = torch.tensor(_scale_vol(c, self.n), device="cuda")
        for y in range(0, h, band):
            rows = (y, min(h, y + band))
            O, D, tn, tf, hit = self.setup(angles, rows)
            ids = torch.nonzero(hit)[:, 0]
            if not ids.numel():
                continue
            pos = (O[ids] + tn[ids, None] * D[ids]) * sv
            dr = D[ids] / D[ids].norm(dim=1, keepdim=True) * sv
            dest = torch.zeros(ids.numel(), 4, dtype=torch.float64, device="cuda")
            live = torch.ones(ids.numel(), dtype=torch.bool, device="cuda")
            while True:
                at = torch.nonzero(live)[:, 0]
                if not at.numel():
                    break
                with torch.no_grad():
                    f = self.fetch(pos[at])
                    nz = self.lic(pos[at], f, each=True)[:, :, 0]
                t = self.table(rgba, f[:, 3] if c["tf_index"] == "magnitude" else f[:, 2])
                col, al = self.shade(((nz @ taps) * self.scale)[:, None], t, None, opac)
                old = dest[at]
                new = ((1 - old[:, 3:]) * torch.cat([col * al[:, None], al[:, None]], 1) + old).clamp(0, 1)
                dest = dest.index_copy(0, at, new)
                pos = pos + dr * self.step
                live = live & ((pos >= 0) & (pos <= 1)).all(1)
                live[at[(al > float(F32(0.95))).detach()]] = False
            img = dest.detach()
            out[rows[0]:rows[1]].view(-1, 4)[ids] = img
            cot = img - target[rows[0]:rows[1]].reshape(-1, 4)[ids].double()
            (dest * cot).sum().backward()
        return out, rgba.grad.reshape(-1), opac.grad, taps.grad


#: sample-steps above which `exact` would take too long
_EXACT_STEPS = {"frame": 9e9, "batch": 3.2e10, "fit": 4e8, "licvolume": 9e9, "animation": math.inf}


def exact(case, seed):
    c = dict(case)
    if c["kind"] == "gradients":  # bytes: they stay equal
        return None
    n, lb, lf, samples = _frames(c)
    steps = (n[0] * n[1] * n[2] if c["kind"] == "licvolume" else samples) * (lb + lf)
    steps *= {"euler": 0.6, "heun": 1.0, "rk4": 1.9}[c["integrator"]] * (1.7 if c["illum"] == "gradient" else 1.0)
    if c["technique"] == "volume":
        steps = 0
    if c["illum"] in ("zoeckler", "mallo") and c["technique"] != "volume":  # table-lit models have no closed form here
        return None
    if steps > _EXACT_STEPS[c["kind"]] or (c["kind"] == "fit" and c["illum"] != "none"):
        return None
    d = _inputs(c, seed)
    noise = None
    if "noise" in d:
        noise = _central(d["noise"]) if c["illum"] == "gradient" else d["noise"].double() / 255
    if c["kind"] == "batch":
        out = []
        for i, xyz in enumerate(d["fields"]):
            e = _Exact(c, _encode(xyz, c["storage"]), noise, d["tf"], d["L"][i], d["L"][i], d["filters"][i])
            out += [e.image(_angles(c, i * c["views"] + k, d["turns"])) for k in range(c["views"])]
        return torch.stack(out)
    e = _Exact(c, _encode(d["field"], c["storage"]), noise, d["tf"], lb, lf, c["filter"])
    angles = [_angles(c, k, d["turns"]) for k in range(c["views"])]
    if c["kind"] == "fit":
        got = [e.fit(a, d["target"][k]) for k, a in enumerate(angles)]
        return {k: torch.stack([g[i] for g in got]) for i, k in enumerate(("image", "tf", "opacity", "taps"))}
    licvol = None
    if c["kind"] == "licvolume":
        nx, ny, nz = e.n
        sv = torch.tensor(_scale_vol(c, e.n), device="cuda")
        lv = torch.empty(nz, ny, nx, dtype=torch.float64, device="cuda")
        slab = max(1, 1000000 // (nx * ny))
        for z in range(0, nz, slab):
            g = torch.meshgrid(*((torch.arange(*r, device="cuda", dtype=torch.float64) + 0.5) / k
                                 for r, k in (((z, min(nz, z + slab)), nz), ((0, ny), ny), ((0, nx), nx))), indexing="ij")
            p = torch.stack([g[2], g[1], g[0]], -1).reshape(-1, 3) * sv
            lv[z:z + slab] = (e.lic(p, e.fetch(p))[:, 0] * e.scale).view(-1, ny, nx)
        licvol = F.pad(lv[None, None], (1, 1, 1, 1, 1, 1), mode="circular")
    return torch.stack([e.image(a, licvol) for a in angles])
