"""Workloads of the registration and filtering path, run through the torch API.

listed() gives the workloads that users of the library run day to day,
draw(rng) more of the same ranges; prepare(case, seed) makes the inputs on
the GPU, run(state) is one pass, work(case) the bytes and operations a pass
cannot do without, and exact(case, seed) the same outputs from a plain FP64
evaluation with torch.

Kinds of workload:
    register    batched affine / rigid registration to one volume
    normalise   T1 volume onto a template (affine and nonlinear pyramid)
    responses   7x7x7 complex quadrature filtering
    smooth      separable Gaussian smoothing of volumes
    smooth_mask normalised-convolution smoothing of an fMRI series
    objective   value and gradient of the differentiable objective
"""
import functools
import math
import os

import numpy as np
import torch

from broccoli_b200 import _lib as L
from broccoli_b200 import autograd as G
from broccoli_b200.api import Context

FILTER_DIR = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "tests", "golden", "filters")
PRECISIONS = {"fp32": L.PREC_FP32, "bf16x3": L.PREC_BF16X3, "tf32": L.PREC_TF32}
TYPES = {"rigid": L.RIGID, "affine": L.AFFINE}
DEVICE = "cuda"


def listed():
    return [
        # one registration of an EPI volume to another: a user at a prompt, or a
        # scanner that sends one volume at a time; latency
        dict(name="pair_affine_fp32", kind="register", w=64, h=64, d=33, batch=1, iterations=20, type="affine",
             precision="fp32", sigma=0.0, tolerance=0.0),
        # motion correction of a 200-volume fMRI run, the throughput workload
        dict(name="series_rigid_tf32", kind="register", w=64, h=64, d=33, batch=199, iterations=8, type="rigid",
             precision="tf32", sigma=1.0, tolerance=0.0),
        # the motion-correction tool as it runs by default: FP32, five iterations;
        # a matrix that no tile divides
        dict(name="series_rigid_fp32", kind="register", w=80, h=80, d=37, batch=59, iterations=5, type="rigid",
             precision="fp32", sigma=0.0, tolerance=0.0),
        # a short run whose volumes stop on their own, the loop ended on the device
        dict(name="series_early_exit_bf16x3", kind="register", w=64, h=64, d=33, batch=24, iterations=20,
             type="rigid", precision="bf16x3", sigma=1.0, tolerance=1e-3),
        # normalisation of one subject to a 1 mm template, mixed precision
        dict(name="t1_to_template_mixed", kind="normalise", w=256, h=256, d=170, tw=182, th=218, td=182,
             linear=10, nonlinear=10, scale=8, precision="tf32", fp64=True),
        # the smallest filtering: a coarse pyramid level
        dict(name="responses_small_fp32", kind="responses", w=18, h=20, d=14, batch=1, filters=3, precision="fp32"),
        # the six nonlinear filters at template size
        dict(name="responses_t1_tf32", kind="responses", w=182, h=218, d=182, batch=1, filters=6, precision="tf32"),
        # the three linear filters of a run, in the default precision
        dict(name="responses_series_fp32", kind="responses", w=64, h=64, d=33, batch=64, filters=3,
             precision="fp32"),
        # smoothing of a preprocessed run inside its brain mask, 6 mm
        dict(name="smooth_series", kind="smooth_mask", w=64, h=64, d=33, batch=200, fwhm=6.0),
        # Gaussian smoothing of template-size maps (a tensor field with its right-hand side)
        dict(name="smooth_t1", kind="smooth", w=182, h=218, d=182, batch=9, sigma=5.0),
        # one step of a gradient-based registration: loss and its gradient, affine
        dict(name="objective_affine", kind="objective", w=128, h=128, d=96, form="affine", sigma=2.0),
        # and by a displacement field
        dict(name="objective_field", kind="objective", w=128, h=128, d=96, form="field", sigma=2.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["register", "register", "normalise", "responses", "responses", "smooth", "smooth_mask",
                       "objective"])
    if kind == "register":
        w, h, d = rng.randint(40, 104), rng.randint(40, 104), rng.randint(18, 48)
        iterations = rng.randint(3, 20)
        most = max(1, int(199 * 64 * 64 * 33 * 8 / (w * h * d * iterations)))
        precision = rng.choice(["fp32", "tf32", "bf16x3"])
        if precision != "tf32":
            most = max(1, most // (6 if precision == "fp32" else 2))
        batch = _log_int(rng, 1, min(199, most))
        tolerance = 1e-3 if batch <= 24 and rng.random() < 0.5 else 0.0
        return dict(kind=kind, w=w, h=h, d=d, batch=batch, iterations=iterations,
                    type=rng.choice(["rigid", "affine"]), precision=precision, sigma=rng.choice([0.0, 1.0]),
                    tolerance=tolerance)
    if kind == "normalise":
        precision = rng.choice(["fp32", "tf32"])
        f = math.exp(rng.uniform(math.log(0.4), 0.0 if precision == "tf32" else math.log(0.8)))
        tw, th, td = (int(round(f * n)) + rng.randint(-3, 0) for n in (182, 218, 182))
        w, h, d = (int(round(n * rng.uniform(0.9, 1.25))) for n in (tw, th, td))
        return dict(kind=kind, w=w, h=h, d=d, tw=tw, th=th, td=td, linear=rng.randint(4, 10),
                    nonlinear=rng.randint(3, 6), scale=4 if min(tw, th, td) < 120 else 8, precision=precision,
                    fp64=precision == "tf32")
    if kind == "responses":
        voxels = _log_int(rng, 5000, 8000000)
        w, h, d, batch = _volume(rng, voxels)
        return dict(kind=kind, w=w, h=h, d=d, batch=batch, filters=rng.choice([3, 6]),
                    precision=rng.choice(["fp32", "tf32", "bf16x3"]))
    if kind == "smooth":
        w, h, d, batch = _volume(rng, _log_int(rng, 20000, 60000000))
        return dict(kind=kind, w=w, h=h, d=d, batch=batch, sigma=rng.choice([1.0, 2.0, 5.0]))
    if kind == "smooth_mask":
        w, h, d = rng.randint(40, 104), rng.randint(40, 104), rng.randint(18, 48)
        return dict(kind=kind, w=w, h=h, d=d, batch=_log_int(rng, 2, 250), fwhm=rng.choice([4.0, 6.0, 8.0]))
    w, h, d = rng.randint(32, 140), rng.randint(32, 140), rng.randint(24, 100)
    return dict(kind=kind, w=w, h=h, d=d, form=rng.choice(["affine", "field"]), sigma=rng.choice([1.0, 2.0]))


def _volume(rng, voxels):
    """Width, height, depth and batch of about `voxels` voxels in all: one
    volume, or a batch of volumes of EPI size."""
    if voxels > 300000 and rng.random() < 0.5:
        w, h, d = rng.randint(40, 104), rng.randint(40, 104), rng.randint(18, 48)
        return w, h, d, max(1, voxels // (w * h * d))
    voxels = min(voxels, 182 * 218 * 182)
    side = voxels ** (1.0 / 3.0)
    w, h = int(side * rng.uniform(0.8, 1.25)), int(side * rng.uniform(0.8, 1.25))
    return w, h, max(8, voxels // (w * h)), 1


# ---- inputs -----------------------------------------------------------------


@functools.lru_cache(None)
def _bank():
    """The shipped filter files: 343 float32 per part, x fastest."""
    def read(name, *shape):
        return np.fromfile(os.path.join(FILTER_DIR, name), np.float32).reshape(shape)
    def filters(n, which):
        return np.stack([np.stack([read("filter%d_%s_%s_registration.bin" % (k + 1, part, which), 7, 7, 7)
                                   for part in ("real", "imag")]) for k in range(n)])
    return {"linear": filters(3, "linear"), "nonlinear": filters(6, "nonlinear"),
            "projection_tensors": np.stack([read("projection_tensor%d.bin" % (k + 1), 6) for k in range(6)]),
            "directions": np.stack([read("filter_directions_%s.bin" % a, 6) for a in "xyz"])}


@functools.lru_cache(None)
def _context():
    return Context(torch.cuda.current_device())


def _gaussian_taps(sigma):
    u = np.arange(9, dtype=np.float64) - 4
    f = np.exp(-u * u / (2.0 * sigma * sigma)).astype(np.float32)
    return (f / f.sum(dtype=np.float32)).astype(np.float32)


def _fwhm_taps(fwhm, voxel):
    return [_gaussian_taps(fwhm / 2.354 / v) for v in voxel]


def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(int(seed) * 7919 + 13)


def _axes(shape, dtype):
    """z, y, x coordinate axes, broadcastable over (D, H, W)."""
    d, h, w = shape
    return (torch.arange(d, device=DEVICE, dtype=dtype)[:, None, None],
            torch.arange(h, device=DEVICE, dtype=dtype)[None, :, None],
            torch.arange(w, device=DEVICE, dtype=dtype)[None, None, :])


def _uniform(gen, lo, hi, *shape):
    return lo + (hi - lo) * torch.rand(*shape, generator=gen, device=DEVICE, dtype=torch.float64)


def _smooth_noise(shape, gen, sigma=2.0):
    n = torch.randn(shape, generator=gen, device=DEVICE, dtype=torch.float64)
    n = _smooth(n[None], [_gaussian_taps(sigma)] * 3)[0]
    return n / n.std()


def _rotation(angles):
    """(..., 3) angles about x, y, z -> (..., 3, 3)."""
    c, s = torch.cos(angles), torch.sin(angles)
    o, z = torch.ones_like(c[..., 0]), torch.zeros_like(c[..., 0])
    def m(*e):
        return torch.stack(e, -1).reshape(*angles.shape[:-1], 3, 3)
    rx = m(o, z, z, z, c[..., 0], -s[..., 0], z, s[..., 0], c[..., 0])
    ry = m(c[..., 1], z, s[..., 1], z, o, z, -s[..., 1], z, c[..., 1])
    rz = m(c[..., 2], -s[..., 2], z, s[..., 2], c[..., 2], z, z, z, o)
    return rz @ ry @ rx


def _epi(shape, gen):
    """An EPI-like volume: smooth noise and five bright ellipsoids."""
    d, h, w = shape
    z, y, x = _axes(shape, torch.float64)
    vol = _smooth_noise(shape, gen)
    for _ in range(5):
        c = _uniform(gen, 0.2, 0.8, 3) * torch.tensor([w, h, d], device=DEVICE)
        r = _rotation(_uniform(gen, 0.0, 6.28, 3))
        semi = _uniform(gen, 3.0, 12.0, 3)
        p = torch.stack(torch.broadcast_tensors(x - c[0], y - c[1], z - c[2]), -1) @ r / semi
        vol = vol + _uniform(gen, 200.0, 1000.0, 1) * ((p * p).sum(-1) <= 1.0)
    return vol


def _moved(vol, gen, n, translation, degrees, scale=0.0):
    """n copies of vol under rigid (or affine) motion, with Rician noise at SNR 50."""
    angles = _uniform(gen, -degrees, degrees, n, 3) * (math.pi / 180.0)
    a = _rotation(angles) * _uniform(gen, 1.0 - scale, 1.0 + scale, n, 1, 3)
    t = _uniform(gen, -translation, translation, n, 3)
    p = torch.cat([t, (a - torch.eye(3, device=DEVICE)).reshape(n, 9)], 1)
    noise = float(vol[vol > 100.0].mean()) / 50.0 if bool((vol > 100.0).any()) else 1.0
    out = torch.empty((n,) + tuple(vol.shape), device=DEVICE, dtype=torch.float32)
    for i in range(n):
        v = _warp_affine(vol[None], p[i:i + 1])[0]
        e = torch.randn((2,) + tuple(vol.shape), generator=gen, device=DEVICE, dtype=torch.float64) * noise
        out[i] = torch.sqrt((v + e[0]) ** 2 + e[1] ** 2)
    return out


def _head(shape, radii, gen):
    """A T1-like head: nested ellipsoidal tissue classes, inner structures, a
    bias field and noise; radii (x, y, z) in voxels."""
    d, h, w = shape
    z, y, x = _axes(shape, torch.float64)
    px, py, pz = (x - (w - 1) / 2.0) / radii[0], (y - (h - 1) / 2.0) / radii[1], (z - (d - 1) / 2.0) / radii[2]
    rho = torch.sqrt(px * px + py * py + pz * pz)
    vol = 300.0 * (rho <= 1.0) + 300.0 * (rho <= 0.85) + 300.0 * (rho <= 0.6)
    for k in range(6):
        c, r = _uniform(gen, -0.4, 0.4, 3), _uniform(gen, 0.08, 0.2, 3)
        inside = ((px - c[0]) / r[0]) ** 2 + ((py - c[1]) / r[1]) ** 2 + ((pz - c[2]) / r[2]) ** 2 <= 1.0
        vol = torch.where(inside & (rho <= 0.85), 300.0 + 300.0 * (k % 2), vol)
    b = _uniform(gen, -1.0, 1.0, 6)
    bias = b[0] * px + b[1] * py + b[2] * pz + b[3] * px * py + b[4] * py * pz + b[5] * px * px
    vol = vol * (1.0 + 0.2 * bias / bias.abs().max())
    return vol + 15.0 * torch.randn(shape, generator=gen, device=DEVICE, dtype=torch.float64)


def _smooth_field(shape, gen, largest):
    """A smooth displacement field (3, D, H, W) of at most `largest` voxels:
    noise on a coarse grid, enlarged trilinearly."""
    coarse = torch.randn((1, 3) + tuple(max(4, n // 16) for n in shape), generator=gen, device=DEVICE)
    f = torch.nn.functional.interpolate(coarse, size=shape, mode="trilinear", align_corners=True)[0].double()
    return f * (largest / torch.sqrt((f * f).sum(0)).max())


def _shape(case):
    return case["d"], case["h"], case["w"]


def _inputs(case, seed):
    """The tensors of a case, float32 on the GPU, from the seed alone."""
    gen = _generator(seed)
    kind, shape = case["kind"], _shape(case)
    if kind == "register":
        affine = case["type"] == "affine"
        v = _moved(_epi(shape, gen), gen, case["batch"] + 1, 2.0 if not affine else 1.5, 2.0, 0.02 if affine else 0.0)
        return {"ref": v[0].contiguous(), "moving": v[1:].contiguous()}
    if kind == "normalise":
        tshape = (case["td"], case["th"], case["tw"])
        radii = [0.40 * case["tw"], 0.42 * case["th"], 0.40 * case["td"]]
        tpl = _head(tshape, radii, gen)
        sub = _head(shape, radii, gen)
        sub = _warp_field(sub, _smooth_field(shape, gen, 6.0 * case["tw"] / 182.0))
        return {"subject": sub.float(), "template": tpl.float()}
    if kind == "responses":
        v = _epi(shape, gen)
        n = case["batch"]
        e = torch.randn((n,) + shape, generator=gen, device=DEVICE, dtype=torch.float32)
        return {"vol": (v.float() + 10.0 * e).contiguous()}
    if kind == "smooth":
        n = case["batch"]
        v = _smooth_noise(shape, gen).float()
        return {"vol": (v + torch.randn((n,) + shape, generator=gen, device=DEVICE)).contiguous()}
    if kind == "smooth_mask":
        n = case["batch"]
        v = _epi(shape, gen).float()
        vols = v + 10.0 * torch.randn((n,) + shape, generator=gen, device=DEVICE)
        smooth = _smooth(v[None].double(), _fwhm_taps(4.0, (3.0, 3.0, 3.5)))[0]
        mask = torch.where(smooth > 0.9 * smooth.mean(), 1.0, 0.001).float()
        return {"vols": vols.contiguous(), "mask": mask.contiguous()}
    ref = _head(shape, [0.40 * shape[2], 0.42 * shape[1], 0.40 * shape[0]], gen)
    field = _smooth_field(shape, gen, 2.0)
    moving = _warp_field(ref, field) + 5.0 * torch.randn(shape, generator=gen, device=DEVICE, dtype=torch.float64)
    if case["form"] == "field":
        x = (-0.5 * field).float().contiguous()
    else:
        a = _rotation(_uniform(gen, -1.0, 1.0, 3) * (math.pi / 180.0)) - torch.eye(3, device=DEVICE)
        x = torch.cat([_uniform(gen, -1.0, 1.0, 3), a.reshape(9)]).float()
    return {"ref": ref.float(), "moving": moving.float(), "x": x}


def prepare(case, seed):
    state = dict(case, ctx=_context(), bank=_bank(), **_inputs(case, seed))
    if case["kind"] == "objective":
        state["q_ref"] = G.reference_responses(state.pop("ref"), state["bank"]["linear"], case["sigma"])
        state["x"].requires_grad_(True)
    elif case["kind"] == "smooth_mask":
        state["taps"] = _fwhm_taps(case["fwhm"], (3.0, 3.0, 3.5))
    elif case["kind"] == "smooth":
        state["taps"] = [_gaussian_taps(case["sigma"])] * 3
    return state


def run(state):
    ctx, bank, kind = state["ctx"], state["bank"], state["kind"]
    if kind == "register":
        return ctx.register_linear(state["ref"], state["moving"], bank["linear"], state["iterations"],
                                   TYPES[state["type"]], tolerance=state["tolerance"],
                                   precision=PRECISIONS[state["precision"]], certainty_sigma=state["sigma"])
    if kind == "normalise":
        return ctx.register_two_volumes(state["subject"], (1.0, 1.0, 1.0), state["template"], (1.0, 1.0, 1.0), bank,
                                        state["linear"], state["nonlinear"], state["scale"],
                                        solve_fp64=state["fp64"], precision=PRECISIONS[state["precision"]])
    if kind == "responses":
        return ctx.filter3d(state["vol"], bank["linear" if state["filters"] == 3 else "nonlinear"],
                            precision=PRECISIONS[state["precision"]])
    if kind == "smooth":
        return ctx.smooth3d(state["vol"], *state["taps"])
    if kind == "smooth_mask":
        return ctx.smooth_normalized(state["vols"], state["mask"], *state["taps"])
    x = state["x"]
    loss = G.registration_objective(state["moving"], state["q_ref"], bank["linear"], state["sigma"],
                                    **({"params": x} if state["form"] == "affine" else {"field": x}))
    grad, = torch.autograd.grad(loss, x)
    return {"loss": loss.detach(), "grad": grad}


def work(case):
    v = float(case["w"] * case["h"] * case["d"])
    b = float(case.get("batch", 1))
    kind = case["kind"]
    if kind == "register":
        # volumes in and aligned volumes out; per iteration three complex
        # filters of 343 taps and the normal equations and warp
        return {"bytes": 4 * v * (2 * b + 1), "flops": v * b * case["iterations"] * (3 * 1372 + 3 * 120 + 40)}
    if kind == "normalise":
        t = float(case["tw"] * case["th"] * case["td"])
        scales = [2 ** k for k in range(int(math.log2(case["scale"])) + 1)]
        lin = sum((math.ceil(case["linear"] / 5) if s == 1 else case["linear"]) / s ** 3 for s in scales)
        non = sum((math.ceil(case["nonlinear"] / 2) if s == 1 else case["nonlinear"]) / s ** 3 for s in scales)
        return {"bytes": 4 * (v + 7 * t), "flops": t * (lin * (3 * 1372 + 400) + non * (6 * 1372 + 18 * 54 + 700))}
    if kind == "responses":
        return {"bytes": 4 * v * b * (1 + 2 * case["filters"]), "flops": v * b * case["filters"] * 1372}
    if kind in ("smooth", "smooth_mask"):
        return {"bytes": 8 * v * b, "flops": 54 * v * b}
    return {"bytes": 4 * v * (1 + 6 + (3 + 3 if case["form"] == "field" else 0)), "flops": v * (2 * 3 * 1372 + 200)}


# ---- the same outputs in FP64 -----------------------------------------------


def _filter(vol, filters):
    """(B, D, H, W) float64 -> (B, nfilt, D, H, W) complex128, zero padding."""
    shape = vol.shape[-3:]
    full = [n + 6 for n in shape]
    f = torch.from_numpy(np.ascontiguousarray(filters)).to(DEVICE).double()
    spectrum = torch.fft.rfftn(vol, s=full, dim=(-3, -2, -1))
    out = []
    for k in range(f.shape[0]):
        parts = [torch.fft.irfftn(spectrum * torch.fft.rfftn(f[k, c], s=full), s=full, dim=(-3, -2, -1))
                 [..., 3:3 + shape[0], 3:3 + shape[1], 3:3 + shape[2]] for c in (0, 1)]
        out.append(torch.complex(*parts))
    return torch.stack(out, 1)


def _smooth(vol, taps):
    """(B, D, H, W) smoothed by 9 taps along x, y, z (symmetric), zero padding."""
    for axis, t in zip((3, 2, 1), taps):
        pad = [0] * 6
        pad[2 * (3 - axis)] = pad[2 * (3 - axis) + 1] = 4
        p = torch.nn.functional.pad(vol, pad)
        n = vol.shape[axis]
        vol = sum(float(t[i]) * p.narrow(axis, i, n) for i in range(9))
    return vol


def _sample(vol, x, y, z):
    """Trilinear samples of (B, D, H, W) at (B, ...) coordinates, clamped to the edges."""
    b, d, h, w = vol.shape
    flat = vol.reshape(b, -1)
    lo = [torch.floor(c.detach()) for c in (x, y, z)]
    fx, fy, fz = x - lo[0], y - lo[1], z - lo[2]
    out = 0.0
    for k in range(8):
        ix, iy, iz = ((lo[a] + ((k >> a) & 1)).clamp(0, n - 1).long() for a, n in ((0, w), (1, h), (2, d)))
        wt = 1.0
        for a, f in enumerate((fx, fy, fz)):
            wt = wt * (f if (k >> a) & 1 else 1.0 - f)
        out = out + wt * torch.gather(flat, 1, (ix + w * (iy + h * iz)).reshape(b, -1)).reshape(x.shape)
    return out


def _affine_displacement(p, shape):
    """(B, 12) -> displacements x, y, z of (B, D, H, W) voxels."""
    d, h, w = shape
    z, y, x = _axes(shape, torch.float64)
    x, y, z = x - (w - 1) / 2.0, y - (h - 1) / 2.0, z - (d - 1) / 2.0
    q = p[:, :, None, None, None]
    return [q[:, a] + q[:, 3 + 3 * a] * x + q[:, 4 + 3 * a] * y + q[:, 5 + 3 * a] * z for a in range(3)]


def _warp(vol, displacement):
    z, y, x = _axes(vol.shape[-3:], torch.float64)
    return _sample(vol, x + displacement[0], y + displacement[1], z + displacement[2])


def _warp_affine(vol, p):
    return _warp(vol, _affine_displacement(p, vol.shape[-3:]))


def _warp_field(vol, field):
    return _warp(vol[None], [f[None] for f in field])[0]


def _resample(vol, shape):
    """(B, D, H, W) on another grid, sample spacing (N - 1) / (N' - 1)."""
    z, y, x = _axes(shape, torch.float64)
    s = [(a - 1) / (b - 1) for a, b in zip(vol.shape[-3:], shape)]
    one = torch.ones((vol.shape[0],) + tuple(shape), device=DEVICE, dtype=torch.float64)
    return _sample(vol, one * x * s[2], one * y * s[1], one * z * s[0])


def _matrix(p):
    m = torch.eye(4, device=DEVICE, dtype=torch.float64).repeat(p.shape[0], 1, 1)
    m[:, :3, :3] += p[:, 3:].reshape(-1, 3, 3)
    m[:, :3, 3] = p[:, :3]
    return m


def _parameters(m):
    eye = torch.eye(3, device=DEVICE, dtype=torch.float64)
    return torch.cat([m[:, :3, 3], (m[:, :3, :3] - eye).reshape(-1, 9)], 1)


def _neighbours(q, axis):
    """Sum of q(x+1) q*(x) + q(x) q*(x-1) along an axis of the interior."""
    def part(step):
        s = [slice(3, -3)] * 3
        s[axis] = slice(3 + step, q.shape[axis - 3] - 3 + step)
        return q[(...,) + tuple(s)]
    return part(1) * part(0).conj() + part(0) * part(-1).conj()


def _normal_equations(q1, q2, sigma):
    """One affine update (B, 12) from responses (3, ...) and (B, 3, ...)."""
    d, h, w = q2.shape[-3:]
    z, y, x = _axes((d, h, w), torch.float64)
    inner = (slice(3, -3),) * 3
    one = torch.ones((d, h, w), device=DEVICE, dtype=torch.float64)
    basis = torch.stack([one, one * (x - (w - 1) / 2.0), one * (y - (h - 1) / 2.0), one * (z - (d - 1) / 2.0)])
    basis = basis[(slice(None),) + inner].reshape(4, -1)
    p = torch.zeros((q2.shape[0], 12), device=DEVICE, dtype=torch.float64)
    for k in range(3):
        cross = q1[k] * q2[:, k].conj()
        cert = 0.5 * (cross.abs() + cross.real)
        if sigma > 0.0:
            e = math.exp(-1.0 / (2.0 * sigma * sigma))
            t = [0.0] * 3 + [e / (1 + 2 * e), 1 / (1 + 2 * e), e / (1 + 2 * e)] + [0.0] * 3
            cert = _smooth(cert, [t, t, t])
        grad = torch.angle(_neighbours(q1[k], 2 - k) + _neighbours(q2[:, k], 2 - k))
        cert, diff = cert[(...,) + inner], torch.angle(cross)[(...,) + inner]
        weight = (cert * grad * grad).reshape(q2.shape[0], -1)
        right = (cert * grad * diff).reshape(q2.shape[0], -1)
        a = torch.einsum("iv,bv,jv->bij", basis, weight, basis) if q2.shape[0] == 1 else torch.stack(
            [(basis * wv) @ basis.T for wv in weight])
        u = torch.linalg.solve(a, right @ basis.T)
        p[:, k] = u[:, 0]
        p[:, 3 + 3 * k:6 + 3 * k] = u[:, 1:]
    return p


def _rotations(p):
    m = (p[:, 3:].reshape(-1, 3, 3) + torch.eye(3, device=DEVICE, dtype=torch.float64))
    a1 = -torch.atan2(m[:, 1, 2], m[:, 2, 2])
    a2 = -torch.atan2(-m[:, 0, 2], torch.sqrt(m[:, 0, 0] ** 2 + m[:, 0, 1] ** 2))
    s, c = torch.sin(a1), torch.cos(a1)
    a3 = -torch.atan2(s * m[:, 2, 0] - c * m[:, 1, 0], c * m[:, 1, 1] - s * m[:, 2, 1])
    return torch.stack([a1, a2, a3], 1) * (180.0 / math.pi)


def _register(ref, moving, filters, iterations, rigid, sigma=0.0, tolerance=0.0):
    """Parameters, aligned volumes and iterations of moving (B, D, H, W) onto ref."""
    q1 = _filter(ref[None], filters)[0]
    b, shape = moving.shape[0], moving.shape[-3:]
    half = [(n - 1) / 2.0 for n in reversed(shape)]
    corners = torch.tensor([[half[a] * (1 if (c >> a) & 1 else -1) for a in range(3)] for c in range(8)],
                           device=DEVICE, dtype=torch.float64)
    p = torch.zeros((b, 12), device=DEVICE, dtype=torch.float64)
    ran = torch.zeros(b, dtype=torch.int32, device=DEVICE)
    aligned = moving.clone()
    per = max(1, int(4e6 // ref.numel()))
    for i in range(0, b, per):
        active = list(range(i, min(b, i + per)))
        for it in range(iterations):
            if not active:
                break
            u = _normal_equations(q1, _filter(aligned[active], filters), sigma)
            if rigid:
                left, _, right = torch.linalg.svd(u[:, 3:].reshape(-1, 3, 3) +
                                                  torch.eye(3, device=DEVICE, dtype=torch.float64))
                u = torch.cat([u[:, :3], (left @ right - torch.eye(3, device=DEVICE)).reshape(-1, 9)], 1)
            p[active] = _parameters(_matrix(u) @ _matrix(p[active]))
            ran[active] = it + 1
            aligned[active] = _warp_affine(moving[active], p[active])
            if tolerance > 0.0:
                move = corners @ u[:, 3:].reshape(-1, 3, 3).transpose(1, 2) + u[:, None, :3]
                size = move.square().sum(-1).sqrt().max(1).values
                active = [n for n, s in zip(active, size.tolist()) if not s < tolerance]
    return p, aligned, ran


def _round(v):
    return int(math.floor(v + 0.5))


def _scaled(shape, scale):
    return tuple(_round(n / scale) for n in shape)


def _register_scales(ref, moving, filters, iterations, coarsest):
    """Affine pyramid registration of one volume: parameters and aligned volume."""
    total = torch.zeros((1, 12), device=DEVICE, dtype=torch.float64)
    scale = coarsest
    while scale >= 1:
        shape = _scaled(ref.shape, scale)
        r, m = _resample(ref[None], shape)[0], _resample(moving[None], shape)
        if scale != coarsest:
            m = _warp_affine(m, total)
        u, _, _ = _register(r, m, filters, math.ceil(iterations / 5) if scale == 1 else iterations, False)
        f = 1.0 if scale == 1 else 2.0
        lengthen = torch.tensor([f] * 3 + [1.0] * 9, device=DEVICE, dtype=torch.float64)
        total = _parameters(_matrix(u * lengthen) @ _matrix(total * lengthen))
        scale //= 2
    return total, _warp_affine(moving[None], total)[0]


def _nonlinear_update(q1, q2, bank):
    """Smoothed displacement update (3, D, H, W) from responses (6, D, H, W)."""
    taps = [_gaussian_taps(5.0)] * 3
    m = torch.from_numpy(bank["projection_tensors"]).to(DEVICE).double()
    n = torch.from_numpy(bank["directions"]).to(DEVICE).double()
    t = _smooth(torch.einsum("k...,kc->c...", q2.abs(), m), taps)
    norm = torch.sqrt(t[0] ** 2 + 2 * t[1] ** 2 + 2 * t[2] ** 2 + t[3] ** 2 + 2 * t[4] ** 2 + t[5] ** 2)
    t = t / norm.max()
    full = [[t[0], t[1], t[2]], [t[1], t[3], t[4]], [t[2], t[4], t[5]]]
    tt = [[sum(full[i][k] * full[k][j] for k in range(3)) for j in range(3)] for i in range(3)]
    upper = [(0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2)]
    ah = [norm] + [torch.zeros_like(norm) for _ in range(8)]
    for k in range(6):
        cross = q1[k] * q2[k].conj()
        size = cross.abs()
        cert = torch.where(size > 0, 0.5 * (size + cross.real) / torch.sqrt(size.clamp_min(1e-300)), 0.0)
        move = cert * torch.angle(cross)
        for c, (i, j) in enumerate(upper):
            ah[c] = ah[c] + cert * tt[i][j]
        for i in range(3):
            ah[6 + i] = ah[6 + i] + move * sum(n[a, k] * tt[i][a] for a in range(3))
    a11, a12, a13, a22, a23, a33, h1, h2, h3 = _smooth(torch.stack(ah), taps)
    c11, c12, c13 = a22 * a33 - a23 * a23, a13 * a23 - a12 * a33, a12 * a23 - a13 * a22
    c22, c23, c33 = a11 * a33 - a13 * a13, a12 * a13 - a11 * a23, a11 * a22 - a12 * a12
    r = 1.0 / (a11 * c11 + a12 * c12 + a13 * c13 + 1e-16)
    step = torch.stack([r * (c11 * h1 + c12 * h2 + c13 * h3), r * (c12 * h1 + c22 * h2 + c23 * h3),
                        r * (c13 * h1 + c23 * h2 + c33 * h3)])
    return _smooth(step, taps)


def _register_nonlinear(ref, moving, bank, iterations, coarsest):
    """Displacement field (3, D, H, W) of moving onto ref, coarse to fine."""
    total, scale = None, coarsest
    while scale >= 1:
        shape = _scaled(ref.shape, scale)
        r, m = _resample(ref[None], shape)[0], _resample(moving[None], shape)[0]
        if total is None:
            total = torch.zeros((3,) + shape, device=DEVICE, dtype=torch.float64)
            start = m
        else:
            total = 2.0 * _resample(total, shape)
            start = _warp_field(m, total)
        q1 = _filter(r[None], bank["nonlinear"])[0]
        field, aligned = torch.zeros_like(total), start
        for _ in range(math.ceil(iterations / 2) if scale == 1 else iterations):
            q2 = _filter(aligned[None], bank["nonlinear"])[0]
            field = field + _nonlinear_update(q1, q2, bank)
            aligned = _warp_field(start, field)
        total = total + field
        scale //= 2
    return total


def _centre(vol):
    z, y, x = _axes(vol.shape, torch.float64)
    return [float((vol * c).sum() / vol.sum()) for c in (x, y, z)]


def _onto_grid(vol, shape):
    """Centred in or cropped to another grid of the same voxel size."""
    out = torch.zeros(shape, device=DEVICE, dtype=torch.float64)
    src, dst = [], []
    for a, b in zip(vol.shape, shape):
        half = (abs(a - b) + 1) // 2
        n = min(b, a - half) if a > b else min(a, b - half)
        src.append(slice(half, half + n) if a > b else slice(0, n))
        dst.append(slice(0, n) if a > b else slice(half, half + n))
    out[tuple(dst)] = vol[tuple(src)]
    return out


def _normalise(case, sub, tpl, bank):
    grid = _onto_grid(sub, tpl.shape)
    match = torch.zeros((1, 12), device=DEVICE, dtype=torch.float64)
    for a, (s, t) in enumerate(zip(_centre(grid), _centre(tpl))):
        match[0, a] = -_round(t - s)
    inter = _warp_affine(grid[None], match)[0]
    p, lin = _register_scales(tpl, inter, bank["linear"], case["linear"], case["scale"])
    p = _parameters(_matrix(match) @ _matrix(p))
    field = _register_nonlinear(tpl, lin, bank, case["nonlinear"], case["scale"])
    field = field + torch.cat(_affine_displacement(p, tpl.shape))
    return {"params": p[0], "interpolated": inter, "aligned_linear": lin, "aligned_nonlinear": _warp_field(grid, field),
            "field": field}


def exact(case, seed):
    bank, x = _bank(), _inputs(case, seed)
    x = {k: v.double() for k, v in x.items()}
    kind = case["kind"]
    if kind == "register":
        rigid = case["type"] == "rigid"
        p, aligned, ran = _register(x["ref"], x["moving"], bank["linear"], case["iterations"], rigid, case["sigma"],
                                    case["tolerance"])
        return {"params": p, "aligned": aligned, "rotations": _rotations(p) if rigid else torch.zeros_like(p[:, :3]),
                "iterations": ran}
    if kind == "normalise":
        return _normalise(case, x["subject"], x["template"], bank)
    if kind == "responses":
        f = bank["linear" if case["filters"] == 3 else "nonlinear"]
        return torch.cat([_filter(v[None], f) for v in x["vol"]])
    if kind == "smooth":
        return torch.cat([_smooth(v[None], [_gaussian_taps(case["sigma"])] * 3) for v in x["vol"]])
    if kind == "smooth_mask":
        taps = _fwhm_taps(case["fwhm"], (3.0, 3.0, 3.5))
        weight = _smooth(x["mask"][None], taps)
        return torch.cat([_smooth((v * x["mask"])[None], taps) / weight * x["mask"] for v in x["vols"]])
    taps = [_gaussian_taps(case["sigma"])] * 3
    q_ref = _filter(_smooth(x["ref"][None], taps), bank["linear"])
    y = x["x"].requires_grad_(True)
    moving = _smooth(x["moving"][None], taps)
    warped = _warp_affine(moving, y[None]) if case["form"] == "affine" else _warp(moving, [f[None] for f in y])
    loss = (_filter(warped, bank["linear"]) - q_ref).abs().square().sum()
    grad, = torch.autograd.grad(loss, y)
    return {"loss": loss.detach(), "grad": grad}
