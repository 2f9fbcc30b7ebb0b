"""Performance cases of the projection framework: the calls its users make, at the sizes they make them.

A case is a dict of plain values.  ``listed()`` gives the fixed ones, ``draw(rng)`` one more of the same
ranges, ``prepare(case, seed)`` builds what a program holds before the call (device inputs from the seed,
the projector or optimizer it keeps), ``run(state)`` makes one pass through the public API and returns its
outputs, ``work(case)`` is the traffic and arithmetic the operation itself needs, and ``exact(case, seed)``
the same outputs in float64 from the definitions, without this package's code.
"""
import math

import numpy as np
import torch

from vamtoolbox_b200 import autograd, geometry, medium, optimize, projectorconstructor
from vamtoolbox_b200.batch import ProjectionBatch
from vamtoolbox_b200.optimizer.BCLP import BCLPNorm

PIXEL_CM = 0.002  # 20 micron voxels, the toolbox's default sampling rate


def listed():
    return [
        # one 2-D slice, both directions: the smallest call (an interactive preview, a layer at a time)
        {"name": "slice_small", "kind": "pair", "n": 128, "nz": 1, "angles": 180, "absorption": "none"},
        # a full-resolution 2-D slice
        {"name": "slice_large", "kind": "pair", "n": 512, "nz": 1, "angles": 720, "absorption": "none"},
        # the forward projection of a large part
        {"name": "forward_large", "kind": "forward", "n": 512, "nz": 128, "angles": 720, "absorption": "none"},
        # the backprojection of the usual part: 256^3 in an absorbing resin, one angle per degree
        {"name": "backward_256", "kind": "backward", "n": 256, "nz": 256, "angles": 360, "absorption": "mask"},
        # a part as a voxeliser gives it: no size a multiple of anything
        {"name": "ragged_pair", "kind": "pair", "n": 201, "nz": 117, "angles": 240, "absorption": "none"},
        # projector inside a differentiable loss: forward and its exact transpose
        {"name": "gradient_160", "kind": "gradient", "n": 160, "nz": 96, "angles": 180, "absorption": "none"},
        # one iteration of the device engine on the usual part: what every BCLP run spends its time on
        {"name": "bclp_step_256", "kind": "step", "n": 256, "nz": 256, "angles": 360, "absorption": "mask"},
        # a whole optimisation of a small part, numpy in, numpy out
        {"name": "bclp_call_small", "kind": "call", "n": 64, "nz": 40, "angles": 90, "absorption": "none",
         "iterations": 10},
        # graded-index medium, paths kept for a run of iterations: integrate and deposit
        {"name": "ray_cached_96", "kind": "ray", "n": 96, "nz": 96, "angles": 120, "cached": True},
        # the same without kept paths: a single forward and backward
        {"name": "ray_traced_64", "kind": "ray", "n": 64, "nz": 48, "angles": 90, "cached": False},
        # laminography: inclined rays, both directions
        {"name": "inclined_128", "kind": "inclined", "n": 128, "nz": 96, "angles": 120, "incline": 15.0},
        # several targets of uneven size through one work queue, both directions
        {"name": "batch_uneven", "kind": "batch", "n": 128, "nz": 128, "angles": 180, "targets": 6},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["forward", "backward", "pair", "pair", "gradient", "step", "call", "ray", "inclined", "batch"])
    absorption = rng.choice(["none", "mask", "mask", "ray"]) if kind in ("forward", "backward", "pair") else rng.choice(["none", "mask"])
    if kind == "ray":
        return {"kind": "ray", "n": log_int(24, 96), "nz": log_int(8, 96), "angles": log_int(16, 120),
                "cached": rng.random() < 0.5}
    if kind == "inclined":
        return {"kind": "inclined", "n": log_int(32, 160), "nz": log_int(16, 96), "angles": log_int(30, 160),
                "incline": rng.choice([-30.0, 10.0, 15.0, 45.0])}
    if kind == "call":
        return {"kind": "call", "n": log_int(32, 96), "nz": log_int(1, 64), "angles": log_int(30, 180),
                "absorption": absorption, "iterations": rng.randint(5, 20)}
    if kind == "batch":
        return {"kind": "batch", "n": log_int(48, 128), "nz": log_int(32, 128), "angles": log_int(60, 180),
                "targets": rng.randint(3, 8)}
    if kind == "pair" and rng.random() < 0.35:
        return {"kind": "pair", "n": log_int(64, 600), "nz": 1, "angles": log_int(60, 800), "absorption": absorption}
    # volumes: half of the slice counts a multiple of four, half any; the product of the sizes at most that of
    # the largest listed case (a pass in both directions at most half of it)
    most = 2.4e10 if kind in ("forward", "backward") else 0.6e10
    while True:
        n, nz, na = log_int(48, 512), log_int(8, 320), log_int(45, 720)
        if rng.random() < 0.5:
            nz = max(4, nz - nz % 4)
        if n * n * nz * na <= most:
            return {"kind": kind, "n": n, "nz": nz, "angles": na, "absorption": absorption}


# ---------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------
def _angles(case):
    return np.linspace(0, 360, case["angles"], endpoint=False)


def _blobs(seed):
    """Random ellipsoids of a part, in units of the vial radius (centre x, y; height; radius; half height)."""
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(int(rng.integers(5, 9))):
        a = rng.uniform(0.1, 0.45)
        r, phi = rng.uniform(0, 0.9 - a), rng.uniform(0, 2 * np.pi)
        out.append((r * np.cos(phi), r * np.sin(phi), rng.uniform(-0.5, 0.5), a, rng.uniform(0.3, 1.0)))
    return out


def _z(nz):
    return (torch.arange(nz, device="cuda", dtype=torch.float64) - (nz - 1) / 2) / max(nz / 2, 1.0)


def _target(n, nz, seed):
    """Binary part: the union of the ellipsoids, float32 [n, n, nz] on the device."""
    c = (torch.arange(n, device="cuda", dtype=torch.float64) - (n - 1) / 2) / (n / 2)
    z = _z(nz)
    vol = torch.zeros((n, n, nz), dtype=torch.bool, device="cuda")
    for cx, cy, cz, a, h in _blobs(seed):
        rho = ((c[None, :] - cx) ** 2 + (c[:, None] - cy) ** 2) / a ** 2
        vol |= rho[:, :, None] <= (1 - ((z - cz) / h) ** 2)[None, None, :]
    return vol.to(torch.float32)


def _volume(n, nz, seed):
    """What a forward projection gets inside an optimizer: a signed residual on the part and a faint one
    around it, zero outside the vial."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    c = (torch.arange(n, device="cuda", dtype=torch.float32) - (n - 1) / 2) / (n / 2)
    vial = ((c[None, :] ** 2 + c[:, None] ** 2) <= 0.94).to(torch.float32)[:, :, None]
    noise = torch.randn((n, n, nz), device="cuda", generator=g)
    t = _target(n, nz, seed)
    return (vial * (t * (0.6 + 0.3 * noise) + (1 - t) * 0.05 * noise)).contiguous()


def _sinogram(n, angles, nz, seed):
    """Non-negative projections of the part with a large dark share: the ellipsoids' chord lengths less a
    constant, clipped at zero, with a little texture."""
    th = torch.as_tensor(np.deg2rad(angles), device="cuda")
    t = (torch.arange(n, device="cuda", dtype=torch.float64) - (n - 1) / 2) / (n / 2)
    z = _z(nz)
    b = torch.zeros((n, len(angles), nz), dtype=torch.float32, device="cuda")
    for cx, cy, cz, a, h in _blobs(seed):
        tc = cx * torch.cos(th) - cy * torch.sin(th)
        r2 = a * a * (1 - ((z - cz) / h) ** 2)
        chord = (r2[None, None, :] - ((t[:, None] - tc[None, :]) ** 2)[:, :, None]).clamp_(min=0).sqrt_()
        b += chord.to(torch.float32)
        del chord
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    b *= 1 + 0.1 * torch.rand(b.shape, device="cuda", generator=g)
    return (b - 0.15).clamp_(min=0).contiguous()


def _proj_geo(case, angles=None):
    n, mode = case["n"], case.get("absorption", "none")
    kw = {}
    if mode != "none":  # e^-1 across the vial
        R = n / 2 * PIXEL_CM
        kw = {"projector_pixel_size": PIXEL_CM, "absorption_coeff": 1.0 / (2 * R), "container_radius": R}
    return geometry.ProjectionGeometry(_angles(case) if angles is None else angles, "parallel", CUDA=True, **kw)


def _projector(case):
    tg = geometry.Volume(np.zeros((case["n"], case["n"], case["nz"]), dtype=np.float32), vol_type="target")
    mode = case.get("absorption", "none")
    kw = {"absorption": "ray"} if mode == "ray" else {}
    return projectorconstructor.projectorconstructor(tg, _proj_geo(case), **kw)


def _batch_sizes(case):
    """Sizes of a batch's targets: slices and volumes of falling size, every third one a slice."""
    out = []
    for k in range(case["targets"]):
        f = 1.0 - 0.1 * k
        n, na = max(32, int(case["n"] * f)), case["angles"] * (2 if k % 2 else 1)
        out.append({"n": 2 * n if k % 3 == 2 else n, "nz": 1 if k % 3 == 2 else max(8, int(case["nz"] * f) // 4 * 4),
                    "angles": na, "absorption": "mask" if k % 2 else "none"})
    return out


def _smooth_noise(shape, sigma, seed):
    """Gaussian-filtered noise of unit largest magnitude, float64 on the device."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    f = torch.fft.fftn(torch.randn(shape, device="cuda", dtype=torch.float64, generator=g))
    for d, m in enumerate(shape):
        k = torch.fft.fftfreq(m, device="cuda", dtype=torch.float64)
        f = f * torch.exp(-2 * (np.pi * sigma * k) ** 2).reshape([-1 if e == d else 1 for e in range(3)])
    p = torch.fft.ifftn(f).real
    return p / p.abs().max()


def _ray_fields(case, seed):
    """Coordinates, refractive index 1.50 + 0.02 (r / R)^2 with a smooth disturbance, and an attenuation of
    e^-1 across the grid with smooth variation."""
    n, nz = case["n"], case["nz"]
    tg = geometry.Volume(np.zeros((n, n, nz), dtype=np.float32), vol_type="target")
    cv = tg.constructCoordVec()
    x = torch.as_tensor(cv[0], device="cuda")
    r2 = (x[:, None] ** 2 + x[None, :] ** 2) / x.max() ** 2
    nx = 1.50 + 0.02 * r2[:, :, None] + 0.005 * _smooth_noise((n, n, nz), 6.0, seed + 2)
    ax = (1.0 + 0.3 * _smooth_noise((n, n, nz), 6.0, seed + 3)) / (n * (cv[0][1] - cv[0][0]))
    return tg, cv, nx, ax


def _ray_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed + 4)
    f = _volume(case["n"], case["nz"], seed).abs_()
    e = torch.rand(case["n"] * case["angles"] * case["nz"], device="cuda", generator=g)
    return f, (e - 0.4).clamp_(min=0)


def _bclp_options(case, **kw):
    return optimize.Options(method="BCLP", p=2, q=1, eps=0.1, filter="ram-lak", **kw)


# ---------------------------------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------------------------------
def prepare(case, seed):
    kind, n, nz = case["kind"], case["n"], case["nz"]
    s = {"kind": kind}
    if kind in ("forward", "backward", "pair", "gradient"):
        s["P"] = _projector(case)
        if kind != "backward":
            s["x"] = _volume(n, nz, seed)
        if kind != "forward":
            s["b"] = _sinogram(n, _angles(case), nz, seed)
    elif kind == "step":
        # the device engine from a given first sinogram; the graph replays one iteration
        tg = geometry.Volume(_target(n, nz, seed).cpu().numpy(), vol_type="target")
        g0 = _sinogram(n, _angles(case), nz, seed).mul_(3.0 / case["angles"]).cpu().numpy()
        solver = BCLPNorm(tg, _proj_geo(case), _bclp_options(case, n_iter=8, learning_rate=1e-5, g0=g0))
        s["solver"], s["it"] = solver, solver.device_iteration()
        s["graph"] = s["it"].capture()
    elif kind == "call":
        s["tg"] = geometry.TargetGeometry(target=_target(n, nz, seed).double().cpu().numpy())
        s["pg"] = _proj_geo(case)
        s["options"] = _bclp_options(case, n_iter=case["iterations"], learning_rate=1e-4)
    elif kind == "ray":
        tg, cv, nx, ax = _ray_fields(case, seed)
        im = medium.IndexModel(cv, type="interpolation", form="freeform", n_x=nx)
        am = medium.AttenuationModel(cv, type="interpolation", form="freeform", alpha_x=ax)
        pg = geometry.ProjectionGeometry(_angles(case), "ray_trace", CUDA=True, index_model=im, attenuation_model=am,
                                         absorption_model=am, ray_trace_method="eikonal",
                                         eikonal_parametrization="physical_path_length",
                                         ray_trace_ode_solver="forward_symplectic_euler",
                                         ray_trace_ray_config="parallel", inclination_angle=0.0, ray_density=1)
        s["P"] = projectorconstructor.projectorconstructor(tg, pg, output_torch_tensor=True)
        if case["cached"]:
            s["P"].plan.prepare_trajectories()
        s["x"], s["b"] = _ray_inputs(case, seed)
    elif kind == "inclined":
        tg = geometry.Volume(np.zeros((n, n, nz), dtype=np.float32), vol_type="target")
        pg = geometry.ProjectionGeometry(_angles(case), "parallel", CUDA=True, inclination_angle=case["incline"])
        s["P"] = projectorconstructor.projectorconstructor(tg, pg)
        s["x"], s["b"] = _volume(n, nz, seed), _sinogram(n, _angles(case), nz, seed)
    elif kind == "batch":
        s["queue"], s["keep"], s["fwd"], s["bwd"] = ProjectionBatch(), [], [], []
        for k, c in enumerate(_batch_sizes(case)):
            P = _projector(c)
            x, b = _volume(c["n"], c["nz"], seed + 10 * k), _sinogram(c["n"], _angles(c), c["nz"], seed + 10 * k)
            s["keep"].append(P)
            s["fwd"].append((P.plan, "forward", x, torch.empty_like(b)))
            s["bwd"].append((P.plan, "backward", b, torch.empty_like(x)))
    return s


def run(s):
    kind = s["kind"]
    if kind == "forward":
        return s["P"].forward(s["x"])
    if kind == "backward":
        return s["P"].backward(s["b"])
    if kind in ("pair", "inclined"):
        return [s["P"].forward(s["x"]), s["P"].backward(s["b"])]
    if kind == "gradient":  # the least-squares loss 1/2 |A x - b|^2 and its gradient
        x = s["x"].requires_grad_(True)
        y = autograd.parallel_forward(x, s["P"].plan)
        (gx,) = torch.autograd.grad(y, x, y.detach() - s["b"])
        return [y.detach(), gx]
    if kind == "step":
        s["graph"].replay()
        it = s["it"]
        return [it.g, it.grad, it.dose, it.mapped, it.stats]
    if kind == "call":
        # the engine computes in float32 and hands out float64 arrays; what is kept is the float32 part
        sino, recon, loss = optimize.optimize(s["tg"], s["pg"], s["options"])
        return [np.asarray(v, dtype=np.float32) for v in (sino.array, recon.array, loss)]
    if kind == "ray":
        return [s["P"].forward(s["x"]), s["P"].backward(s["b"])]
    s["queue"].submit(s["fwd"])
    s["queue"].submit(s["bwd"])
    return [w[3] for w in s["fwd"]] + [w[3] for w in s["bwd"]]


# ---------------------------------------------------------------------------------------------------
# the work an operation cannot do without
# ---------------------------------------------------------------------------------------------------
def work(case):
    n, nz, na, kind = case["n"], case["nz"], case["angles"], case["kind"]
    if kind == "batch":
        parts = [work({**c, "kind": "pair"}) for c in _batch_sizes(case)]
        return {"bytes": sum(p["bytes"] for p in parts), "flops": sum(p["flops"] for p in parts)}
    vol, sino = 4.0 * n * n * nz, 4.0 * n * na * nz
    fwd = 8.0 * n * n * nz * na            # four taps a sample
    bwd = 4.0 * (math.pi / 4) * n * n * nz * na  # two taps a pixel of the disk
    if kind == "forward":
        return {"bytes": vol + sino, "flops": fwd}
    if kind == "backward":
        return {"bytes": vol + sino, "flops": bwd}
    if kind == "pair":
        return {"bytes": 2 * (vol + sino), "flops": fwd + bwd}
    if kind == "gradient":
        return {"bytes": 2 * (vol + sino) + sino, "flops": 2 * fwd}
    if kind in ("step", "call"):
        k = case.get("iterations", 1)
        # g read and written, the target read, dose, mapped dose and gradient written
        return {"bytes": k * (3 * sino + 3 * vol), "flops": k * (fwd + bwd)}
    if kind == "ray":
        # about 2 n half-voxel steps through the grid a ray; a sample of the medium (unless kept) and of the field
        steps = 2.0 * n * n * na * nz
        return {"bytes": 2 * (vol + sino), "flops": 2 * steps * (16 if case["cached"] else 100)}
    return {"bytes": 2 * (vol + sino), "flops": 16.0 * n * n * nz * na}  # inclined: four taps each way


# ---------------------------------------------------------------------------------------------------
# float64 references, from the definitions
# ---------------------------------------------------------------------------------------------------
def _disk(n):
    """The inscribed circle's pixels (numpy's linspace decides the ones on its edge), 1.0 inside."""
    lin = np.linspace(-1, 1, n)
    return torch.as_tensor((lin[:, None] ** 2 + lin[None, :] ** 2 <= 1).astype(np.float64), device="cuda")


def _f64_setup(case):
    n = case["n"]
    C = n // 2
    circle = _disk(n)
    mask = None
    if case.get("absorption") == "mask":
        r = n / 2 * PIXEL_CM
        p = torch.as_tensor(np.linspace(-r, r, n), device="cuda")
        depth = r - torch.sqrt(p[:, None] ** 2 + p[None, :] ** 2)
        mask = torch.where(depth < 0, torch.zeros_like(depth), torch.exp(-depth / (2 * r)))
    ray = (1.0 / n, n / 2) if case.get("absorption") == "ray" else None  # attenuation a pixel, radius in pixels
    return n, C, circle, mask, ray


def _lattice(n, C, deg):
    """Sample coordinates of one angle, [k, j]: the rotated image's pixels in the image."""
    r = deg * (math.pi / 180.0)
    c, s = math.cos(r), math.sin(r)
    k = torch.arange(n, device="cuda", dtype=torch.float64)[:, None]
    j = torch.arange(n, device="cuda", dtype=torch.float64)[None, :]
    return c * k - s * j - C * (c - s - 1), s * k + c * j - C * (c + s - 1)


def _taps(row, col, n):
    r0, c0 = torch.floor(row), torch.floor(col)
    for a in (0, 1):
        for b in (0, 1):
            r, c = r0 + a, c0 + b
            w = (1 - (row - r).abs()) * (1 - (col - c).abs())
            ok = (r >= 0) & (r < n) & (c >= 0) & (c < n)
            yield (w * ok).reshape(-1, 1), (r.clamp(0, n - 1) * n + c.clamp(0, n - 1)).long().reshape(-1)


def _ray_weight(n, C, ray):
    """Per-sample factor exp(-a (s - s_entry)) of [k, j], zero for rays outside the container."""
    al, R = ray
    t = torch.arange(n, device="cuda", dtype=torch.float64)[None, :] - C
    s = torch.arange(n, device="cuda", dtype=torch.float64)[:, None] - C
    depth = (s + torch.sqrt((R * R - t * t).clamp(min=0))).clamp(min=0)
    return (torch.exp(-al * depth) * (t.abs() <= R)).reshape(-1, 1)


def _forward64(x, case):
    n, C, _, mask, ray = _f64_setup(case)
    nz = x.shape[2]
    x = x.double() if mask is None else x.double() * mask[:, :, None]
    flat, out = x.reshape(n * n, nz), torch.empty((n, case["angles"], nz), dtype=torch.float64, device="cuda")
    for a, deg in enumerate(_angles(case)):
        row, col = _lattice(n, C, deg)
        acc = sum(w * flat[i] for w, i in _taps(row, col, n))
        if ray:
            acc = acc * _ray_weight(n, C, ray)
        out[:, a] = acc.reshape(n, n, nz).sum(0)
    return out


def _adjoint64(b, case):
    n, C, _, mask, _ = _f64_setup(case)
    nz = b.shape[2]
    flat = torch.zeros((n * n, nz), dtype=torch.float64, device="cuda")
    for a, deg in enumerate(_angles(case)):
        row, col = _lattice(n, C, deg)
        v = b[:, a].double()[None].expand(n, n, nz).reshape(n * n, nz)
        for w, i in _taps(row, col, n):
            flat.index_add_(0, i, w * v)
    x = flat.reshape(n, n, nz)
    return x if mask is None else x * mask[:, :, None]


def _backward64(b, case):
    n, C, circle, mask, ray = _f64_setup(case)
    X = torch.arange(n, device="cuda", dtype=torch.float64)[None, :] - C
    Y = torch.arange(n, device="cuda", dtype=torch.float64)[:, None] - C
    x = torch.zeros((n * n, b.shape[2]), dtype=torch.float64, device="cuda")
    for a, deg in enumerate(_angles(case)):
        r = deg * (math.pi / 180.0)
        t = (X * math.cos(r) - Y * math.sin(r)).reshape(-1)
        f = torch.floor(t)
        j0 = (f.long() + C).clamp(0, n - 1)
        w = t - f
        ok = ((t >= -C) & (t <= n - 1 - C)).double()
        if ray:
            al, R = ray
            s = (X * math.sin(r) + Y * math.cos(r)).reshape(-1)
            depth = (s + torch.sqrt((R * R - t * t).clamp(min=0))).clamp(min=0)
            ok = ok * torch.exp(-al * depth) * (t.abs() <= R)
        rows = b[:, a].double()
        x += (ok * (1 - w))[:, None] * rows[j0] + (ok * w)[:, None] * rows[(j0 + 1).clamp(max=n - 1)]
    x = x.reshape(n, n, -1) * circle[:, :, None]
    return x if mask is None else x * mask[:, :, None]


def _interp64(x, xp, fp):
    xp, fp = torch.as_tensor(xp, device="cuda"), torch.as_tensor(fp, device="cuda")
    j = (torch.searchsorted(xp, x.contiguous(), right=True) - 1).clamp(0, len(xp) - 2)
    y = fp[j] + (fp[j + 1] - fp[j]) / (xp[j + 1] - xp[j]) * (x - xp[j])
    return torch.where(x <= xp[0], fp[0], torch.where(x >= xp[-1], fp[-1], y))


def _response_tables():
    """The default response: a logistic curve of midpoint 0.5 and slope 25, sampled at 512 doses."""
    f = np.linspace(0, 1, 512)
    m = 1 / (1 + np.exp(-25 * (f - 0.5)))
    return f, m, 25 * m * m * np.exp(-25 * (f - 0.5))


def _bclp64(g, target, case, lr):
    """One iteration from g: the new sinogram, its gradient before the loss factor, dose, mapped dose, sums."""
    f, m, dm = _response_tables()
    dose = _backward64(g, case)
    mapped = _interp64(dose, f, m)
    e = mapped - target
    band = e.abs() - 0.1
    v = (band > 0).double()
    fwd = _forward64(v * band.abs() * torch.sign(e) * _interp64(dose, f, dm), case)
    stats = torch.stack([(v * band ** 2).sum(), v.sum(), (e != 0).double().sum(), (v * band.abs()).sum(), e.abs().sum(),
                         (v * band ** 2).sum(), (e ** 2).sum(), (v * band.abs()).max(), e.abs().max()])
    loss = stats[0].sqrt()
    scale = 1 / loss if float(loss) != 0.0 else 1.0
    return (g - lr * scale * fwd).clamp(min=0), fwd, dose, mapped, stats


def _first_sinogram64(target, case):
    """The default start: the inverse response of the target, projected, ramp-filtered along the detector
    (the band-limited ramp's samples, zero-padded to a power of two), scaled and clipped at zero."""
    f, m, _ = _response_tables()
    b = _forward64(_interp64(target, m, f), case)
    n = b.shape[0]
    size = max(64, 2 ** math.ceil(math.log2(2 * n)))
    h = np.zeros(size)
    h[0] = 0.25
    odd = np.arange(1, size, 2)
    h[odd] = -1.0 / (np.pi * np.minimum(odd, size - odd)) ** 2
    H = torch.as_tensor(2 * np.real(np.fft.fft(h)), device="cuda")[:, None, None]
    y = torch.fft.ifft(torch.fft.fft(b, n=size, dim=0) * H, dim=0).real[:n]
    return (y * (math.pi / (2 * case["angles"]))).clamp(min=0)


def _ray64(case, seed):
    """Symplectic Euler through the sampled medium in float64: line integrals of f and the deposited dose."""
    n, nz, na = case["n"], case["nz"], case["angles"]
    _, cv, nx, ax = _ray_fields(case, seed)
    f, e0 = _ray_inputs(case, seed)
    vox = [float(c[1] - c[0]) for c in cv]
    grad = torch.zeros((n, n, nz, 3), dtype=torch.float64, device="cuda")
    grad[1:-1, :, :, 0] = (nx[2:] - nx[:-2]) / (2 * vox[0])
    grad[:, 1:-1, :, 1] = (nx[:, 2:] - nx[:, :-2]) / (2 * vox[1])
    grad[:, :, 1:-1, 2] = (nx[:, :, 2:] - nx[:, :, :-2]) / (2 * vox[2])
    tex = torch.cat([nx[..., None], grad], dim=3).reshape(-1, 4)
    att = ax.reshape(-1)
    dims = (n, n, nz)
    half = [float(c[-1] - c[0]) / 2 for c in cv]
    # starting states in float32, as the tracer takes them
    t32 = lambda a: torch.as_tensor(np.asarray(a), dtype=torch.float32)
    G0, G1, G2 = (v.ravel() for v in torch.meshgrid(t32(cv[0]), t32(_angles(case) * np.pi / 180.0), t32(cv[2]),
                                                    indexing="ij"))
    off = float(np.sqrt(cv[0][-1] ** 2 + cv[2][-1] ** 2))
    x0 = torch.stack([off * torch.cos(G1) - G0 * torch.sin(G1), off * torch.sin(G1) + G0 * torch.cos(G1), G2], 1)
    x = x0.cuda().double()
    v = torch.stack([-torch.cos(G1), -torch.sin(G1), torch.zeros_like(G1)], 1).cuda().double()

    def corners(u, border):
        """(flat index, weight) of the eight corners of grid coordinates u; outside: clamped, or weight zero."""
        if border:
            u = torch.stack([u[:, d].clamp(0, dims[d] - 1) for d in range(3)], 1)
        lo = torch.floor(u)
        for c in range(8):
            i, w = [], 1.0
            for d in range(3):
                p = lo[:, d] + ((c >> d) & 1)
                w = w * (1 - (u[:, d] - p).abs()) * ((p >= 0) & (p < dims[d]))
                i.append(p.clamp(0, dims[d] - 1).long())
            yield (i[0] * n + i[1]) * nz + i[2], w

    h = vox[0] / 2
    att_sum = torch.zeros(x.shape[0], dtype=torch.float64, device="cuda")
    integral = torch.zeros_like(att_sum)
    dose = torch.zeros(n * n * nz, dtype=torch.float64, device="cuda")
    fa = f.double().reshape(-1) * att
    scale = torch.tensor([1 / p for p in vox], dtype=torch.float64, device="cuda")
    shift = torch.tensor(half, dtype=torch.float64, device="cuda")
    for _ in range(3 * n):
        u = (x + shift) * scale
        t = sum(w[:, None] * tex[i] for i, w in corners(u, True))
        alpha = sum(w * att[i] for i, w in corners(u, False))
        v = v + t[:, 1:] * h
        dx = v / t[:, :1] * h
        x = x + dx
        att_sum = att_sum + alpha * dx.norm(dim=1)
        E = torch.exp(-att_sum)
        for i, w in corners((x + shift) * scale, False):
            wE = w * E * 0.5
            integral += fa[i] * wE
            dose.index_add_(0, i, wE * e0.double())
    return [integral, (dose * att).reshape(n, n, nz)]


def _bilinear64(plane, f0, f1):
    n0, n1 = plane.shape
    g0, g1 = torch.floor(f0), torch.floor(f1)
    out = 0.0
    for a in (0, 1):
        for b in (0, 1):
            p, q = g0 + a, g1 + b
            w = (1 - (f0 - p).abs()) * (1 - (f1 - q).abs()) * ((p >= 0) & (p < n0) & (q >= 0) & (q < n1))
            out = out + w * plane[p.clamp(0, n0 - 1).long(), q.clamp(0, n1 - 1).long()]
    return out


def _inclined64(case, seed):
    """Joseph's forward (bilinear on the planes across a ray's largest component) and the voxel-driven
    backprojection of rays inclined out of the slice plane; the volume clipped to the inscribed circle."""
    n, nz, angles = case["n"], case["nz"], _angles(case)
    x, b = _volume(n, nz, seed).double(), _sinogram(n, angles, nz, seed).double()
    circle = _disk(n)[:, :, None]
    x = x * circle
    cen = np.array([0.5 - n / 2, 0.5 - n / 2, 0.5 - nz / 2])
    inc = math.radians(case["incline"])
    ar = lambda m: torch.arange(m, device="cuda", dtype=torch.float64)
    sino, vol = torch.empty_like(b), torch.zeros_like(x)
    cc, rr = ar(n)[:, None] - n / 2 + 0.5, ar(nz)[None, :] - nz / 2 + 0.5
    vi, vj, vk = ar(n)[:, None, None] + cen[0], ar(n)[None, :, None] + cen[1], ar(nz)[None, None, :] + cen[2]
    for a, th in enumerate(np.deg2rad(angles)):
        s, c = math.sin(th), math.cos(th)
        ray = np.array([s, -c, math.sin(inc)])
        u = np.array([c, s, 0.0])
        w = np.array([s * math.cos(inc), -c * math.cos(inc), math.cos(inc)])
        p = np.abs(ray)
        d = 0 if p[0] >= p[1] and p[0] >= p[2] else (1 if p[1] >= p[2] else 2)
        rest = [e for e in range(3) if e != d]
        P = [cc * u[e] + rr * w[e] for e in range(3)]
        acc = 0.0
        for k in range(x.shape[d]):
            t = (cen[d] + k - P[d]) / ray[d]
            acc = acc + _bilinear64(x.select(d, k), *[P[e] + t * ray[e] - cen[e] for e in rest])
        sino[:, a] = acc * float(np.linalg.norm(ray) / p[d])
        M = np.linalg.inv(np.stack([u, w, ray], axis=1))
        fu = M[0, 0] * vi + M[0, 1] * vj + M[0, 2] * vk + n / 2 - 0.5
        fv = M[1, 0] * vi + M[1, 1] * vj + M[1, 2] * vk + nz / 2 - 0.5
        vol += _bilinear64(b[:, a], fu.expand_as(vol), fv.expand_as(vol))
    return [sino, vol * circle]


def exact(case, seed):
    kind, n, nz = case["kind"], case["n"], case["nz"]
    if kind == "forward":
        return _forward64(_volume(n, nz, seed), case)
    if kind == "backward":
        return _backward64(_sinogram(n, _angles(case), nz, seed), case)
    if kind == "pair":
        return [_forward64(_volume(n, nz, seed), case), _backward64(_sinogram(n, _angles(case), nz, seed), case)]
    if kind == "gradient":
        y = _forward64(_volume(n, nz, seed), case)
        return [y, _adjoint64(y - _sinogram(n, _angles(case), nz, seed), case)]
    if kind == "step":
        g = _sinogram(n, _angles(case), nz, seed).mul_(3.0 / case["angles"]).double()
        return list(_bclp64(g, _target(n, nz, seed).double(), case, 1e-5))
    if kind == "call":
        t = _target(n, nz, seed).double() * _disk(n)[:, :, None]
        g, loss = _first_sinogram64(t, case), []
        for _ in range(case["iterations"]):
            g, _, _, _, stats = _bclp64(g, t, case, 1e-4)
            loss.append(stats[0].sqrt())
        _, _, dose, _, stats = _bclp64(g, t, case, 1e-4)
        return [g, dose, torch.stack(loss + [stats[0].sqrt()])]
    if kind == "ray":
        return _ray64(case, seed)
    if kind == "inclined":
        return _inclined64(case, seed)
    fwd, bwd = [], []
    for k, c in enumerate(_batch_sizes(case)):
        fwd.append(_forward64(_volume(c["n"], c["nz"], seed + 10 * k), c))
        bwd.append(_backward64(_sinogram(c["n"], _angles(c), c["nz"], seed + 10 * k), c))
    return fwd + bwd
