"""The work that users of this framework have it do, as cases that can be timed and checked.

Each case is one call (or one training-style forward and backward) through the public entry points, with
the plan, background and inputs a program has in hand before it:

  unwrap        phase frames, capi.unwrap_noalloc (a camera loop: one or a few frames, latency)
  unwrap_batch  phase images of uneven sides packed in one buffer, capi.UnwrapBatch
  tv            total-variation proximal step of a volume, capi.tv_prox_workspace (the regulariser by itself)
  pipeline      off-axis holograms on the device to a refractive-index volume, capi.Pipeline.process_device
                or, for a batch of requests of one geometry, process_device_graph
  numpy         the same through the reference-compatible numpy API, qoraholo_b200.Pipeline.run
  bpm           multi-slice beam propagation, BpmModel forward and backward (a gradient step)

`listed` are the sizes of the repository's benchmark and tests and generic ones beside them (sides that are
not powers of two, odd multiples, more views, fewer slices); `draw` gives more of the same ranges.
"""

from __future__ import annotations

import math
import random

import numpy as np
import torch

WAVELENGTH, N_MEDIUM, NA = 0.532, 1.337, 1.2
FIELD_PIXEL = 0.11  # micrometres per field (and volume) pixel of the pipelines
BPM_PIXEL = 0.2
NA_ILLUMINATION = 0.9
NOISE = 0.02
TV_WEIGHT = 1e-2

DEV = "cuda"
F64, C128 = torch.float64, torch.complex128


# ---- the cases ------------------------------------------------------------------------------------


def _pipeline(name, count, holo, m, nz, solver, iterations, inner=0, batch=1, kind="pipeline"):
    return {"name": name, "kind": kind, "count": count, "holo": holo, "m": m, "nz": nz, "solver": solver,
            "iterations": iterations, "inner": inner, "batch": batch}


def listed():
    return [
        # One frame of a phase camera: five small launches, nothing to fill the GPU with.
        {"name": "unwrap_frame_120x160", "kind": "unwrap", "count": 1, "ny": 120, "nx": 160},
        # A folder of phase images of all sizes in one call (quantitative phase imaging in bulk).
        {"name": "unwrap_batch_200", "kind": "unwrap_batch", "count": 200, "low": 96, "high": 640, "mix": 5},
        # TV denoising of a volume whose rows are longer than 256 voxels.
        {"name": "tv_160x300x320", "kind": "tv", "nz": 160, "ny": 300, "nx": 320, "inner": 10},
        # A preview while the sample is being focused: small volume, few iterations, latency.
        _pipeline("preview_gp_64", 49, 128, 64, 64, "gp", 10),
        # Many small requests of one instrument, reconstructed together and replayed as a graph.
        _pipeline("batch8_gp_96", 25, 192, 96, 96, "gp", 10, batch=8),
        # The default of `reconstruct`: direct inversion, no iterations, complex spectra.
        _pipeline("direct_200", 49, 400, 200, 200, "direct", 0),
        # The largest volume of the served mix: 97 megapixel-size holograms, half-spectrum iterations.
        _pipeline("gp_384", 97, 1024, 384, 384, "gp", 20),
        # The headline reconstruction: 49 holograms of 512^2 into 256^3 with FISTA-TV 20 x 10.
        _pipeline("tv_256", 49, 512, 256, 256, "tv", 20, 10),
        # The same solver on a camera crop that is no power of two, fewer planes than rows.
        _pipeline("tv_180x150", 31, 360, 180, 150, "tv", 10, 10),
        # A drop-in user's call: numpy holograms in, numpy volume out.
        _pipeline("numpy_gp_128", 49, 256, 128, 128, "gp", 20, kind="numpy"),
        # Gradient of the beam-propagation misfit, the benchmark's size.
        {"name": "bpm_256x128", "kind": "bpm", "n": 256, "nz": 128, "count": 49, "every": 16},
        # And a smaller one whose side is no power of two.
        {"name": "bpm_160x60", "kind": "bpm", "n": 160, "nz": 60, "count": 24, "every": 8},
    ]


def _log_even(rng, low, high):
    return max(low, min(high, 2 * round(math.exp(rng.uniform(math.log(low), math.log(high))) / 2)))


def _smooth_even(rng, low, high):
    """An even side whose largest prime factor is at most 13, as reconstruction grids are chosen."""
    while True:
        n = m = _log_even(rng, low, high)
        for p in (2, 3, 5, 7, 11, 13):
            while m % p == 0:
                m //= p
        if m == 1:
            return n


def draw(rng: random.Random):
    kind = rng.choice(["unwrap", "unwrap_batch", "tv", "gp", "gp", "tvpipe", "tvpipe", "direct", "c2c", "numpy", "bpm"])
    if kind == "unwrap":
        return {"kind": "unwrap", "count": rng.randint(1, 8), "ny": _log_even(rng, 64, 700), "nx": _log_even(rng, 64, 700)}
    if kind == "unwrap_batch":
        low = rng.choice([64, 96, 128, 200])
        return {"kind": "unwrap_batch", "count": rng.randint(10, 200), "low": low, "high": rng.choice([300, 512, 640]),
                "mix": rng.randint(0, 10 ** 6)}
    if kind == "tv":
        nx = rng.randint(40, 330)
        return {"kind": "tv", "nz": rng.randint(20, 200), "ny": rng.randint(40, 300), "nx": nx if nx <= 256 else 4 * (nx // 4),
                "inner": rng.randint(3, 10)}
    if kind == "bpm":
        return {"kind": "bpm", "n": _smooth_even(rng, 64, 256), "nz": rng.randint(16, 100), "count": rng.randint(5, 40),
                "every": rng.choice([8, 16])}
    top = {"gp": 360, "tvpipe": 300, "direct": 300, "c2c": 200, "numpy": 200}[kind]
    m = _smooth_even(rng, 48, top)
    while kind == "tvpipe" and m > 256 and m % 4:  # longer TV rows come in multiples of 4
        m = _smooth_even(rng, 48, top)
    nz = m if rng.random() < 0.5 else _smooth_even(rng, max(24, m // 2), m)
    solver = {"gp": "gp", "tvpipe": "tv", "direct": "direct", "c2c": "c2c", "numpy": "gp"}[kind]
    case = {"kind": "numpy" if kind == "numpy" else "pipeline", "count": rng.randint(15, 70),
            "holo": 2 * round(m * rng.uniform(1.7, 2.4) / 2), "m": m, "nz": nz, "solver": solver,
            "iterations": 0 if kind == "direct" else rng.randint(4, 12), "inner": rng.randint(4, 10) if solver == "tv" else 0,
            "batch": rng.choice([1, 1, 4]) if kind in ("gp", "tvpipe") and m <= 96 else 1}
    return case


def _sides(case):
    """The images of an uneven batch: sides over the logarithm of [low, high] in steps of 8 (as camera
    regions come), a third of them square."""
    rng = random.Random(case["mix"])
    side = lambda: 8 * round(math.exp(rng.uniform(math.log(case["low"]), math.log(case["high"]))) / 8)  # noqa: E731
    out = []
    for _ in range(case["count"]):
        ny = side()
        out.append((ny, ny if rng.random() < 1 / 3 else side()))
    return out


# ---- inputs ---------------------------------------------------------------------------------------


def _circular_scan(count):
    """One view on axis, the others evenly on the illumination cone; (count, 2) of (fy, fx), float32."""
    out = np.zeros((count, 2), np.float32)
    f = NA_ILLUMINATION / WAVELENGTH
    for i in range(1, count):
        phi = 2.0 * math.pi * (i - 1) / (count - 1)
        out[i] = (f * math.sin(phi), f * math.cos(phi))
    return out


def _phase_maps(shapes, seed):
    """Wrapped phase of smooth random surfaces (Gaussians and a tilt, 10 to 60 rad) with 0.1 rad of noise."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    rng = np.random.default_rng(seed)
    out = []
    for ny, nx in shapes:
        y = torch.arange(ny, device=DEV, dtype=torch.float32)[:, None] / ny
        x = torch.arange(nx, device=DEV, dtype=torch.float32)[None, :] / nx
        surf = float(rng.uniform(-1, 1)) * y + float(rng.uniform(-1, 1)) * x
        for _ in range(int(rng.integers(3, 7))):
            cy, cx, sy, sx = rng.uniform(0, 1), rng.uniform(0, 1), rng.uniform(0.05, 0.3), rng.uniform(0.05, 0.3)
            surf = surf + float(rng.uniform(-1, 1)) * torch.exp(-((y - cy) / sy) ** 2 - ((x - cx) / sx) ** 2)
        surf = (surf - surf.min()) / (surf.max() - surf.min()).clamp_min(1e-9) * float(rng.uniform(10, 60))
        surf = surf + 0.1 * torch.randn((ny, nx), device=DEV, generator=g)
        out.append(torch.remainder(surf + math.pi, 2 * math.pi) - math.pi)
    return out


def _cell(rng, scale):
    """A cell of ellipsoids, (centre zyx, semi-axes zyx, index step over what surrounds it): a body, a
    nucleus and a vesicle, for a field of view `scale` times that of 256 pixels."""
    dn = rng.uniform(0.015, 0.03)
    dy, dx = rng.uniform(-2.0, 2.0, 2)
    s = scale
    return [((0.0, dy * s, dx * s), (4.0 * s, 5.0 * s, 6.0 * s), N_MEDIUM, N_MEDIUM + dn),
            ((0.0, dy * s, (dx - 1.5) * s), (3.0 * s,) * 3, N_MEDIUM + dn, N_MEDIUM + dn + 0.015),
            ((0.0, (dy + 1.5) * s, (dx + 3.0) * s), (1.0 * s,) * 3, N_MEDIUM + dn, N_MEDIUM + dn + 0.03)]


def _rytov_ratio(shapes, fy_i, fx_i, n, pixel):
    """Field ratio (n, n) at z = 0 of an illumination: the first Born spectrum of the ellipsoids on its
    Ewald cap, taken as a Rytov phase."""
    k0 = 2 * math.pi / WAVELENGTH
    fm2, fna2 = (N_MEDIUM / WAVELENGTH) ** 2, (NA / WAVELENGTH) ** 2
    sb = torch.fft.fftfreq(n, d=1.0 / n, dtype=F64, device=DEV) / (n * pixel)
    my, mx = sb[:, None], sb[None, :]
    ar = torch.arange(n, device=DEV)
    par = 1.0 - 2.0 * ((ar[:, None] + ar[None, :]) % 2)
    fiz = math.sqrt(fm2 - fy_i * fy_i - fx_i * fx_i)
    rho2 = (my + fy_i) ** 2 + (mx + fx_i) ** 2
    ok = (rho2 <= fna2) & (rho2 < fm2)
    nuz = torch.sqrt(torch.where(ok, fm2 - rho2, torch.ones_like(rho2)))
    qz = nuz - fiz
    o = 0.0
    for c, a, n0, n1 in shapes:
        step = k0 * k0 * (n1 * n1 - n0 * n0) * 4.0 / 3.0 * math.pi * a[0] * a[1] * a[2]
        arg = 2 * math.pi * torch.sqrt((a[0] * qz) ** 2 + (a[1] * my) ** 2 + (a[2] * mx) ** 2)
        safe = arg.clamp_min(1e-3)
        ball = torch.where(arg < 1e-3, 1.0 - arg * arg / 10.0, 3.0 * (torch.sin(safe) - safe * torch.cos(safe)) / safe ** 3)
        o = o + step * ball * torch.exp(-2j * math.pi * (qz * c[0] + my * c[1] + mx * c[2]))
    u = 1j / (4 * math.pi * nuz) * o * par / (pixel * pixel)
    return torch.exp(torch.fft.ifft2(torch.where(ok, u, torch.zeros_like(u))))


def _carrier(case):
    return round(0.55 * case["m"])


def _radius(case):
    return min(case["m"] / 2.0, math.ceil(NA / WAVELENGTH * case["m"] * FIELD_PIXEL) + 1.0)


def _holograms(case, seed, sample):
    """(count, N, N) float32 off-axis holograms on the GPU, of the sample or (sample None) the background."""
    n, count = case["holo"], case["count"]
    pixel = FIELD_PIXEL * case["m"] / n
    c = _carrier(case) / (n * pixel)
    r = (torch.arange(n, device=DEV, dtype=F64) - n // 2) * pixel
    ref = torch.exp(-2j * math.pi * c * (r[:, None] + r[None, :]))
    g = torch.Generator(device=DEV).manual_seed(seed)
    out = torch.empty((count, n, n), dtype=torch.float32, device=DEV)
    for a, (fy, fx) in enumerate(_circular_scan(count).astype(np.float64)):
        u = torch.exp(2j * math.pi * (fy * r[:, None] + fx * r[None, :]))
        if sample is not None:
            u = u * _rytov_ratio(sample, fy, fx, n, pixel)
        out[a] = (ref + u).abs().square().float() + NOISE * torch.randn((n, n), device=DEV, generator=g)
    return out


def _stacks(case, seed):
    """Sample holograms (batch * count, N, N) and background holograms (count, N, N), on the GPU."""
    rng = np.random.default_rng(seed)
    holo = [_holograms(case, 1000 * seed + b, _cell(rng, case["m"] / 256.0)) for b in range(case["batch"])]
    return torch.cat(holo) if len(holo) > 1 else holo[0], _holograms(case, 1000 * seed + 999, None)


def _bpm_inputs(case, seed):
    """Contrast of the current estimate (nz, n, n) and the measured fields (count, n, n) of the truth."""
    n, nz = case["n"], case["nz"]
    rng = np.random.default_rng(seed)
    z = ((torch.arange(nz, device=DEV) - nz // 2) * BPM_PIXEL)[:, None, None]
    y = ((torch.arange(n, device=DEV) - n // 2) * BPM_PIXEL)[None, :, None]
    x = ((torch.arange(n, device=DEV) - n // 2) * BPM_PIXEL)[None, None, :]
    truth = torch.zeros((nz, n, n), device=DEV)
    half_z, half_x = 0.5 * nz * BPM_PIXEL, 0.5 * n * BPM_PIXEL
    for _ in range(20):
        c = rng.uniform(-0.4, 0.4, 3) * np.array([half_z, 2 * half_x, 2 * half_x]) * 0.8
        inside = (z - c[0]) ** 2 + (y - c[1]) ** 2 + (x - c[2]) ** 2 <= float(rng.uniform(0.04, 0.12) * 2 * half_x) ** 2
        truth = torch.where(inside, torch.full_like(truth, float(rng.uniform(0.005, 0.05))), truth)
    start = 0.6 * truth + 0.002 * torch.rand(truth.shape, device=DEV, generator=torch.Generator(device=DEV).manual_seed(seed))
    return start, _bpm_forward(truth, case, torch.complex64).contiguous()


def _geometry(pixel):
    return (WAVELENGTH, N_MEDIUM, NA, pixel)


def _solver(case):
    s = case["solver"]
    o = {"nz": case["nz"], "iterations": case["iterations"], "solver": "tv" if s == "tv" else "gp",
         "gp_transform": "c2c" if s == "c2c" else "r2c"}
    if s == "tv":
        o.update(tv_weight=TV_WEIGHT, tv_inner=case["inner"])
    return o


def _stream():
    return torch.cuda.current_stream().cuda_stream


def prepare(case, seed):
    from qoraholo_b200 import capi

    kind = case["kind"]
    if kind == "unwrap":
        wrapped = torch.stack(_phase_maps([(case["ny"], case["nx"])] * case["count"], seed))
        return {"kind": kind, "case": case, "in": wrapped, "out": torch.empty_like(wrapped)}
    if kind == "unwrap_batch":
        shapes = _sides(case)
        packed = torch.cat([m.reshape(-1) for m in _phase_maps(shapes, seed)])
        return {"kind": kind, "plan": capi.UnwrapBatch(shapes), "in": packed, "out": torch.empty_like(packed)}
    if kind == "tv":
        b = _tv_input(case, seed)
        work = torch.empty((12,) + tuple(b.shape), dtype=torch.float32, device=DEV)
        return {"kind": kind, "case": case, "b": b, "x": torch.empty_like(b), "work": work}
    if kind == "bpm":
        from qoraholo_b200.autograd import BpmModel

        start, data = _bpm_inputs(case, seed)
        model = BpmModel(case["nz"], case["n"], _circular_scan(case["count"]), _geometry(BPM_PIXEL),
                         checkpoint_every=case["every"])
        return {"kind": kind, "model": model, "data": data, "ri": (N_MEDIUM + start).requires_grad_(True)}
    holo, background = _stacks(case, seed)
    center = (_carrier(case), _carrier(case))
    il = _circular_scan(case["count"])
    if kind == "numpy":
        import qoraholo_b200 as qh

        g = qh.Geometry(wavelength=WAVELENGTH, n_medium=N_MEDIUM, na=NA, pixel=FIELD_PIXEL)
        plan = qh.Pipeline(case["count"], case["holo"], center, il, g, radius=_radius(case), output_size=case["m"],
                           **_solver(case))
        plan.set_background(background.cpu().numpy())
        return {"kind": kind, "plan": plan, "in": holo.cpu().numpy()}
    plan = capi.Pipeline(case["count"], case["holo"], center, il, _geometry(FIELD_PIXEL), radius=_radius(case),
                         output_size=case["m"], batch=case["batch"], **_solver(case))
    plan.set_background(background.cpu().numpy())
    return {"kind": kind, "plan": plan, "in": holo, "batch": case["batch"],
            "out": torch.empty(plan.shape, dtype=torch.float32, device=DEV)}


def _tv_input(case, seed):
    """A piecewise constant volume with noise, in the units of a scattering potential."""
    rng = np.random.default_rng(seed)
    ax = [torch.linspace(-1, 1, case[k], device=DEV) for k in ("nz", "ny", "nx")]
    b = torch.zeros((case["nz"], case["ny"], case["nx"]), device=DEV)
    for _ in range(8):
        c, r = rng.uniform(-0.6, 0.6, 3), rng.uniform(0.15, 0.5)
        d2 = (ax[0][:, None, None] - c[0]) ** 2 + (ax[1][None, :, None] - c[1]) ** 2 + (ax[2][None, None, :] - c[2]) ** 2
        b = torch.where(d2 <= r * r, torch.full_like(b, float(rng.uniform(2.0, 12.0))), b)
    return b + 1.5 * torch.randn(b.shape, device=DEV, generator=torch.Generator(device=DEV).manual_seed(seed))


def _tv_lambda():
    return TV_WEIGHT * (2.0 * math.pi / WAVELENGTH) ** 2


# ---- the calls ------------------------------------------------------------------------------------


def run(state):
    from qoraholo_b200 import capi

    kind = state["kind"]
    if kind == "unwrap":
        c = state["case"]
        capi.unwrap_noalloc(state["in"].data_ptr(), state["out"].data_ptr(), c["count"], c["ny"], c["nx"], _stream())
        return state["out"]
    if kind == "unwrap_batch":
        state["plan"].run(state["in"].data_ptr(), state["out"].data_ptr(), _stream())
        return state["out"]
    if kind == "tv":
        c, b = state["case"], state["b"]
        state["work"][:3].zero_()  # a cold start of the dual
        capi.tv_prox_workspace(b.data_ptr(), state["x"].data_ptr(), state["work"].data_ptr(), 12, c["nz"], c["ny"], c["nx"],
                               _tv_lambda(), c["inner"], _stream())
        return state["x"], state["work"][:3]
    if kind == "bpm":
        ri = state["ri"]
        ri.grad = None
        fields = state["model"](ri)
        fields.backward((fields.detach() - state["data"]) / state["model"].count)
        return fields.detach(), ri.grad
    if kind == "numpy":
        return state["plan"].run(state["in"])
    if state["batch"] > 1:
        state["plan"].process_device_graph(state["in"].data_ptr(), state["out"].data_ptr(), _stream())
    else:
        state["plan"].process_device(state["in"].data_ptr(), state["out"].data_ptr(), _stream())
    return state["out"]


# ---- what a call cannot do without ---------------------------------------------------------------


def _fft_flops(points):
    return 5.0 * points * math.log2(max(points, 2))


def work(case):
    kind = case["kind"]
    if kind in ("unwrap", "unwrap_batch"):
        shapes = _sides(case) if kind == "unwrap_batch" else [(case["ny"], case["nx"])] * case["count"]
        px = sum(y * x for y, x in shapes)
        # Two real 2D cosine transforms (half a complex transform each), the divergence and the constant.
        return {"bytes": 8.0 * px, "flops": sum(_fft_flops(y * x) + 30.0 * y * x for y, x in shapes)}
    if kind == "tv":
        v = case["nz"] * case["ny"] * case["nx"]
        return {"bytes": 4.0 * v * (1 + 1 + 3 + 3), "flops": 36.0 * v * case["inner"] + 8.0 * v}
    if kind == "bpm":
        v, f = case["nz"] * case["n"] ** 2, case["count"] * case["n"] ** 2
        # Per slice and view: two transforms forward and two backward, the screens and propagators.
        flops = case["nz"] * case["count"] * (4 * _fft_flops(case["n"] ** 2) + 60.0 * case["n"] ** 2)
        return {"bytes": 4.0 * 2 * v + 8.0 * 2 * f, "flops": flops}
    count, n, m, nz, b = case["count"], case["holo"], case["m"], case["nz"], case["batch"]
    v = nz * m * m
    f = count * m * m
    flops = count * (_fft_flops(n * n) / 2 + 4 * _fft_flops(m * m)) + 20.0 * f  # fields, unwrap, spectra
    if case["solver"] in ("direct", "c2c"):
        flops += _fft_flops(v) * (1 + 2 * case["iterations"])
    else:
        flops += _fft_flops(v) / 2 * (1 + 2 * case["iterations"])
    flops += case["iterations"] * case["inner"] * 36.0 * v
    return {"bytes": b * (4.0 * count * n * n + 4.0 * v) + 8.0 * f, "flops": b * flops}


def tolerance(case):
    """About four times what the present code shows against `exact`, or, where that is dominated by what
    every 32-bit form shares (the unwrap's eigenvalues), against itself with the sums in another order."""
    kind = case["kind"]
    if kind in ("unwrap", "unwrap_batch"):  # transposed images: rel 2e-7 to 1.3e-6, max 9e-7 to 4e-6
        return {"rel": 5e-6, "max": 2e-5}
    if kind == "tv":  # x 4.5e-8, dual 1.6e-7; max 1.2e-6
        return {"rel": 6e-7, "max": 5e-6}
    if kind == "bpm":  # fields 1e-6 to 9e-6, gradient 2e-6 to 1.6e-5; max 4e-5
        return {"rel": 4e-5, "max": 2e-4}
    # Index volumes (1.337 everywhere, the contrast a few hundredths): 3e-8 to 1.3e-6, max 5e-7 to 1.3e-4.
    return {"rel": 2e-6, "max": 2e-4}


# ---- the same in 64 bits, in plain torch ----------------------------------------------------------


def _wrap(p):
    return p - 2.0 * math.pi * torch.floor((p + math.pi) / (2.0 * math.pi))


def _unwrap64(psi):
    """Least-squares unwrap of (count, ny, nx): the Neumann Poisson problem, by an even extension and its
    Fourier transform, then the constant that agrees with the input modulo 2 pi."""
    psi = psi.to(F64)
    _, ny, nx = psi.shape
    dx, dy = _wrap(psi[:, :, 1:] - psi[:, :, :-1]), _wrap(psi[:, 1:] - psi[:, :-1])
    rho = torch.zeros_like(psi)
    rho[:, :, :-1] += dx
    rho[:, :, 1:] -= dx
    rho[:, :-1] += dy
    rho[:, 1:] -= dy
    ext = torch.cat([rho, rho.flip(2)], 2)
    ext = torch.cat([ext, ext.flip(1)], 1)
    ky = 2.0 * torch.cos(math.pi * torch.arange(2 * ny, device=DEV, dtype=F64) / ny)
    kx = 2.0 * torch.cos(math.pi * torch.arange(nx + 1, device=DEV, dtype=F64) / nx)
    ev = ky[:, None] + kx[None, :] - 4.0
    ev[0, 0] = 1.0
    spec = torch.fft.rfft2(ext) / ev
    spec[:, 0, 0] = 0.0
    phi = torch.fft.irfft2(spec, s=(2 * ny, 2 * nx))[:, :ny, :nx]
    acc = torch.polar(torch.ones_like(phi), psi - phi).sum((1, 2))
    return phi + torch.angle(acc)[:, None, None]


def _extract64(holo, case):
    """Fields (count, m, m) of holograms: the sideband cut out with a disc, moved to the origin."""
    n, m, c = case["holo"], case["m"], _carrier(case)
    r2 = _radius(case) ** 2
    ar = torch.arange(n, device=DEV)
    par = (1.0 - 2.0 * ((ar[:, None] + ar[None, :]) % 2)).to(F64)
    d = torch.arange(m, device=DEV) - m // 2
    at = n // 2 + c + d
    inside = (d[:, None] ** 2 + d[None, :] ** 2 <= r2) & ((at >= 0) & (at < n))[:, None] & ((at >= 0) & (at < n))[None, :]
    at = at.clamp(0, n - 1)
    out = []
    for h in holo:
        spec = torch.fft.fft2(h.to(F64) * par)[at][:, at]
        out.append(torch.fft.ifft2(torch.where(inside, spec, torch.zeros_like(spec))) * (m * m / (n * n)) * par[:m, :m])
    return torch.stack(out)


def _bins(fy_i, fx_i, n, nz):
    """The axial bin of every lateral bin of a view and whether it has one, chosen in float32 as the model
    defines it (a choice of indices, not a computed value)."""
    f = np.float32
    fm, fna = f(N_MEDIUM) / f(WAVELENGTH), f(NA) / f(WAVELENGTH)
    fm2, fna2 = fm * fm, fna * fna
    df = f(1.0) / (f(n) * f(FIELD_PIXEL))
    dfz = f(1.0) / (f(nz) * f(FIELD_PIXEL))
    sb = np.arange(n)
    sb = np.where(sb < n // 2, sb, sb - n).astype(f) * df
    fy, fx = (sb + f(fy_i))[:, None], (sb + f(fx_i))[None, :]
    rho2 = fy * fy + fx * fx
    ok = ~((rho2 > fna2) | (rho2 >= fm2))
    nuz = np.sqrt(np.where(ok, fm2 - rho2, f(0.0)))
    fiz = np.sqrt(fm2 - f(fy_i) * f(fy_i) - f(fx_i) * f(fx_i))
    k = np.floor((nuz - fiz) / dfz + f(0.5)).astype(np.int64)
    ok &= (k >= -(nz // 2)) & (k < nz // 2)
    return np.where(k < 0, k + nz, k), ok


def _map64(spectra, case):
    n, nz = case["m"], case["nz"]
    gain = 4.0 * math.pi / FIELD_PIXEL
    fm2 = (N_MEDIUM / WAVELENGTH) ** 2
    sb = torch.fft.fftfreq(n, d=1.0 / n, dtype=F64, device=DEV) / (n * FIELD_PIXEL)
    pot = torch.zeros(nz * n * n, dtype=C128, device=DEV)
    weight = torch.zeros(nz * n * n, dtype=F64, device=DEV)
    for a, (fy, fx) in enumerate(_circular_scan(case["count"])):
        kz, ok = _bins(fy, fx, n, nz)
        kz, ok = torch.from_numpy(kz).to(DEV), torch.from_numpy(ok).to(DEV)
        nuz = torch.sqrt((fm2 - (sb[:, None] + float(fy)) ** 2 - (sb[None, :] + float(fx)) ** 2).clamp_min(0.0))
        v = -1j * gain * nuz * spectra[a] * (1.0 - 2.0 * (kz % 2))
        flat = (kz * n * n + torch.arange(n * n, device=DEV).reshape(n, n))[ok]  # each voxel at most once a view
        pot[flat] += v[ok]
        weight[flat] += 1.0
    pot = torch.where(weight > 0, pot / weight.clamp_min(1.0), pot)
    return pot.reshape(nz, n, n), (weight > 0).reshape(nz, n, n)


def _divergence64(q):
    s = torch.zeros_like(q[0])
    for axis in range(3):
        k = q[axis].shape[axis] - 1
        lo = q[axis].narrow(axis, 0, k)
        s.narrow(axis, 0, k).add_(lo)
        s.narrow(axis, 1, k).sub_(lo)
    return s


def _tv_prox64(b, p, lam, inner):
    """Fast gradient projection on the dual p (a list of three volumes), from p; the new x and p."""
    r, t = [c.clone() for c in p], 1.0
    for _ in range(inner):
        x = (b - lam * _divergence64(r)).clamp_min(0.0)
        tn = 0.5 * (1.0 + math.sqrt(1.0 + 4.0 * t * t))
        mom, t = (t - 1.0) / tn, tn
        for axis in range(3):
            k = x.shape[axis] - 1
            r[axis].narrow(axis, 0, k).add_((x.narrow(axis, 0, k) - x.narrow(axis, 1, k)) / (12.0 * lam))
        scale = torch.rsqrt((r[0] ** 2 + r[1] ** 2 + r[2] ** 2).clamp_min(1.0))
        for axis in range(3):
            nxt = r[axis] * scale
            r[axis] = nxt + mom * (nxt - p[axis])
            p[axis] = nxt
    return (b - lam * _divergence64(p)).clamp_min(0.0), p


def _solve64(spectra, case):
    m, nz, it = case["m"], case["nz"], case["iterations"]
    k02 = (2.0 * math.pi / WAVELENGTH) ** 2
    pot, filled = _map64(spectra, case)
    imag = torch.zeros((), dtype=F64, device=DEV)
    if case["solver"] in ("direct", "c2c"):
        x = torch.fft.ifftn(pot)
        for _ in range(it):
            x = torch.fft.ifftn(torch.where(filled, pot, torch.fft.fftn(x.real.clamp_min(0.0))))
        real, imag = x.real, x.imag
    else:
        h = m // 2 + 1
        flip = lambda v: torch.roll(v.flip(0, 1, 2), (1, 1, 1), (0, 1, 2))  # noqa: E731  k -> -k
        a = (0.5 * (pot + flip(pot).conj()))[:, :, :h]
        keep = 1.0 - 0.5 * (filled.to(F64) + flip(filled).to(F64))[:, :, :h]
        del pot, filled
        inverse = lambda e: torch.fft.irfftn(e, s=(nz, m, m))  # noqa: E731
        y = inverse(a)
        if case["solver"] == "gp":
            for _ in range(it):
                y = inverse(a + keep * torch.fft.rfftn(y.clamp_min(0.0)))
            real = y
        else:
            prev, t = y.clone(), 1.0
            p = [torch.zeros_like(y) for _ in range(3)]
            for _ in range(it):
                x, p = _tv_prox64(inverse(a + keep * torch.fft.rfftn(y)), p, _tv_lambda(), case["inner"])
                tn = 0.5 * (1.0 + math.sqrt(1.0 + 4.0 * t * t))
                y = x + (t - 1.0) / tn * (x - prev)
                prev, t = x, tn
            real = prev
    re = N_MEDIUM ** 2 + real / k02
    return torch.sqrt(0.5 * (torch.hypot(re, (imag / k02).expand_as(re)) + re))


def _bpm_forward(contrast, case, dtype=C128):
    """Multi-slice beam propagation of the contrast (nz, n, n): field ratios (count, n, n) at z = 0."""
    n, nz = case["n"], case["nz"]
    il = _circular_scan(case["count"]).astype(np.float64)
    fm, fna = N_MEDIUM / WAVELENGTH, NA / WAVELENGTH
    sb = torch.fft.fftfreq(n, d=1.0 / n, dtype=F64, device=DEV) / (n * BPM_PIXEL)
    fy = sb[None, :, None] + torch.from_numpy(il[:, 0]).to(DEV)[:, None, None]
    fx = sb[None, None, :] + torch.from_numpy(il[:, 1]).to(DEV)[:, None, None]
    fiz = torch.from_numpy(np.sqrt(fm * fm - (il ** 2).sum(1))).to(DEV)[:, None, None]
    rho2 = fy * fy + fx * fx
    inside = rho2 < fm * fm
    nuz = torch.sqrt(torch.where(inside, fm * fm - rho2, torch.zeros_like(rho2)))
    angle = 2.0 * math.pi * (nuz - fiz)
    back = -(nz - 1 - nz // 2) * BPM_PIXEL
    step = torch.where(inside, torch.exp(1j * angle * BPM_PIXEL), torch.zeros((), dtype=C128, device=DEV)).to(dtype)
    last = torch.where(inside & (rho2 <= fna * fna), torch.exp(1j * angle * back), torch.zeros((), dtype=C128, device=DEV)).to(dtype)
    least = math.sqrt(max(fm * fm - fna * fna, 0.01 * fm * fm))
    q = torch.where(inside, fm / nuz.clamp_min(least), torch.ones_like(nuz)).to(contrast.dtype)
    del fy, fx, rho2, inside, nuz, angle
    phase = 2.0 * math.pi / WAVELENGTH * BPM_PIXEL
    s = torch.zeros((case["count"], n, n), dtype=dtype, device=DEV)
    s[:, 0, 0] = n * n
    w = torch.ones((), dtype=dtype, device=DEV)
    for k in range(nz):
        if k:
            w = torch.fft.ifft2(s)
        v = torch.fft.fft2(torch.polar(torch.ones_like(contrast[k]), phase * contrast[k]) * w.expand_as(s))
        s = (last if k == nz - 1 else step) * (q * v + (1.0 - q) * s)
    return torch.fft.ifft2(s)


def exact(case, seed):
    kind = case["kind"]
    if kind == "unwrap":
        return _unwrap64(torch.stack(_phase_maps([(case["ny"], case["nx"])] * case["count"], seed)))
    if kind == "unwrap_batch":
        return torch.cat([_unwrap64(m[None]).reshape(-1) for m in _phase_maps(_sides(case), seed)])
    if kind == "tv":
        b = _tv_input(case, seed).to(F64)
        x, p = _tv_prox64(b, [torch.zeros_like(b) for _ in range(3)], float(np.float32(_tv_lambda())), case["inner"])
        return x, torch.stack(p)
    if kind == "bpm":
        start, data = _bpm_inputs(case, seed)
        ri = N_MEDIUM + start  # rounded as the caller holds it
        contrast = (ri.to(F64) - N_MEDIUM).requires_grad_(True)
        fields = _bpm_forward(contrast, case)
        fields.backward((fields.detach() - data) / case["count"])
        return fields.detach(), contrast.grad
    holo, background = _stacks(case, seed)
    base = _extract64(background, case)
    out = []
    for h in holo.split(case["count"]):
        ratio = _extract64(h, case) / base
        phase = _unwrap64(torch.angle(ratio))
        edge = torch.ones(phase.shape[1:], dtype=F64, device=DEV)
        edge[1:-1, 1:-1] = 0.0
        mean = (phase * edge).sum((1, 2)) / edge.sum()
        phase = phase - (2.0 * math.pi * torch.round(mean / (2.0 * math.pi)))[:, None, None]
        out.append(_solve64(torch.fft.fft2(torch.complex(torch.log(ratio.abs()), phase)), case))
    index = torch.stack(out) if case["batch"] > 1 else out[0]
    return index.cpu().numpy() if kind == "numpy" else index
