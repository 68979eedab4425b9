"""The calls that stand for the work of a program built on this package.

A case is one iteration's evaluation of a reconstruction (data loss and gradients of the
object and of the probe, pupil or coded surface), or one registration of a measured stack,
through the package's public entry points.  ``listed`` names the cases, ``draw`` gives more of
the same ranges, ``prepare`` makes what a program holds before the call (seeded, on the GPU),
``run`` makes the call, ``work`` counts what the call cannot do without and ``exact`` evaluates
it in 64 bits with plain torch.

The inputs follow the synthetic workloads of the benchmark: objects with amplitude U[0.8, 1]
and phase U[-pi/2, pi/2], Gaussian probes under a smooth random phase screen, circular pupils
over an LED grid, angular-spectrum propagators, binary coded surfaces, and Poisson counts of
the forward model as uint16.  The current estimate is that of an early iteration: the truth
under 30% complex noise, its brightness off by a fifth (the illumination's power is not known).
"""

from __future__ import annotations

import math

import numpy as np
import torch
import torch.nn.functional as F

import ptychox_b200 as px
from ptychox_b200 import registration, synth

NOISE, BRIGHTNESS = 0.3, 0.8  # relative complex noise and amplitude of the current estimate


def listed():
    def raster(name, kind, p, obj, grid, step, origin, jitter, photons):
        return {"name": name, "kind": kind, "ph": p, "pw": p, "oh": obj, "ow": obj, "gy": grid, "gx": grid,
                "step": step, "origin": origin, "jitter": jitter, "photons": photons}

    def fpm(name, n, h, grid):
        return {"name": name, "kind": "fourier", "oh": n, "ow": n, "ph": h, "pw": h, "gy": grid, "gx": grid,
                "photons": 5e3}

    def field(name, kind, n, count, loss, shifts):
        return {"name": name, "kind": kind, "n": n, "count": count, "ds": 4, "loss": loss, "shift_grad": shifts,
                "photons": 2e3}

    return [
        # a mini-batch of small diffraction patterns: the smallest call, where launches count
        raster("base-16x32", "base", 32, 128, 4, 24, 2, 2, 1e4),
        # a small far-field scan, the size of the drivers' own example
        raster("base-121x128", "base", 128, 512, 11, 32, 8, 2, 1e4),
        # the headline scan: a 512-pixel detector over a 2048-pixel object
        raster("base-900x512", "base", 512, 2048, 30, 48, 64, 3, 1e5),
        # a detector crop that is no power of two
        raster("base-400x640", "base", 640, 2048, 20, 64, 64, 3, 1e5),
        # the reference drivers' own loop: the plain operator on a mini-batch of positions,
        # torch's mean squared error on its amplitudes, backward
        raster("operator-36x96", "operator", 96, 320, 6, 32, 8, 2, 1e4),
        # the headline scan with real-valued (interferometer) positions
        raster("subpixel-900x512", "subpixel", 512, 2048, 30, 48, 64, 3, 1e5),
        # a 15x15 LED-array microscope, and a smaller one with sides that are no powers of two
        fpm("fourier-225x256", 1024, 256, 15),
        fpm("fourier-169x240", 960, 240, 13),
        # lensless coded ptychography at full field
        field("coded-64x1024", "coded", 1024, 64, "mse", False),
        # near-field scan at a camera crop that is no power of two, its positions refined as well
        field("nearfield-32x960", "nearfield", 960, 32, "mse", True),
        # a region of interest under the coded driver's finite-difference loss
        field("coded-fd-16x256", "coded", 256, 16, "fd-isotropic", False),
        # positional tracking and refinement of a near-field stack before its reconstruction
        {"name": "track-200x512", "kind": "track", "h": 512, "w": 512, "count": 200},
    ]


def _smooth(lo, hi):
    """Every 2^a 3^b 5^c in [lo, hi]."""
    out = []
    for n in range(lo, hi + 1):
        m = n
        for p in (2, 3, 5):
            while m % p == 0:
                m //= p
        if m == 1:
            out.append(n)
    return out


def _near(rng, sides, lo, hi):
    """A side of `sides`, spread over the logarithm of [lo, hi]."""
    want = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(sides, key=lambda s: abs(math.log(s / want)))


def draw(rng):
    """One more case: any of the kinds above at any supported side, odd and rectangular ones
    among them, small mini-batches to full scans."""
    kind = rng.choice(["base", "base", "operator", "subpixel", "fourier", "coded", "nearfield", "track"])
    if kind in ("base", "operator", "subpixel"):
        sides = _smooth(16, 640)
        ph = _near(rng, sides, 16, 640)
        pw = ph if rng.random() < 0.7 else _near(rng, sides, max(16, ph // 2), min(640, 2 * ph))
        step = max(2, int(max(ph, pw) * rng.uniform(0.08, 0.35)))
        most = 120e6 if kind == "base" else 60e6 if kind == "subpixel" else 20e6  # pattern pixels of a call
        top = max(2, int(min(30, math.sqrt(most / (ph * pw)), (2000 - max(ph, pw)) / step)))
        gy = round(math.exp(rng.uniform(math.log(2), math.log(top))))
        gx = max(1, gy + rng.choice([-1, 0, 0, 1]))
        jitter = min(3, step // 2)
        origin = jitter + rng.randint(1, 20)
        oh = 2 * origin + (gy - 1) * step + ph + rng.randint(0, 9)
        ow = 2 * origin + (gx - 1) * step + pw + rng.randint(0, 9)
        # a few photons a pixel in the mean, as in the listed scans
        photons = float(round(ph * pw * rng.uniform(0.4, 2.0)))
        return {"kind": kind, "ph": ph, "pw": pw, "oh": oh, "ow": ow, "gy": gy, "gx": gx, "step": step,
                "origin": origin, "jitter": jitter, "photons": photons}
    if kind == "fourier":
        ph = _near(rng, _smooth(48, 256), 48, 256)
        n = _near(rng, [s for s in _smooth(96, 1024) if 3.4 * ph <= s <= 4.6 * ph], 3.4 * ph, min(1024, 4.6 * ph))
        g = rng.randint(3, 15)
        return {"kind": kind, "oh": n, "ow": n, "ph": ph, "pw": ph, "gy": g, "gx": g, "photons": 5e3}
    if kind in ("coded", "nearfield"):
        ds = rng.choice([2, 4])
        n = _near(rng, [s for s in _smooth(96, 1024) if s % ds == 0], 96, 1024)
        count = round(math.exp(rng.uniform(math.log(4), math.log(max(5, min(64, 40e6 / n**2))))))
        return {"kind": kind, "n": n, "count": count, "ds": ds,
                "loss": rng.choice(["mse", "mse", "fd-isotropic"]), "shift_grad": rng.random() < 0.3, "photons": 2e3}
    h = rng.randint(100, 420)
    return {"kind": kind, "h": h, "w": max(100, h + rng.randint(-40, 40)), "count": rng.randint(5, 100)}


# ---------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _object(h, w, gen):
    amp = 0.8 + 0.2 * torch.rand(h, w, generator=gen, device="cuda")
    return torch.polar(amp, math.pi * (torch.rand(h, w, generator=gen, device="cuda") - 0.5))


def _estimate(truth, gen):
    noise = torch.randn(*truth.shape, 2, generator=gen, device="cuda")
    return (BRIGHTNESS * truth * (1 + NOISE * torch.view_as_complex(noise))).contiguous()


def _low_pass(h, w, corr, gen):
    f = torch.fft.fft2(torch.randn(h, w, generator=gen, device="cuda"))
    fy, fx = torch.fft.fftfreq(h, device="cuda")[:, None], torch.fft.fftfreq(w, device="cuda")[None, :]
    out = torch.fft.ifft2(f * torch.exp(-(fx**2 + fy**2) * corr**2 * 2 * math.pi**2)).real
    return out / out.std()


def _probe(h, w, gen):
    y = torch.arange(h, device="cuda")[:, None] - (h - 1) / 2
    x = torch.arange(w, device="cuda")[None, :] - (w - 1) / 2
    amp = torch.exp(-0.5 * ((y / (0.2 * h)) ** 2 + (x / (0.2 * w)) ** 2))
    return torch.polar(amp, 2.0 * _low_pass(h, w, 0.03 * max(h, w), gen)).contiguous()


def _positions(case, seed):
    rng = np.random.default_rng(seed)
    make = synth.raster_positions_subpixel if case["kind"] == "subpixel" else synth.raster_positions
    pos = make(case["gy"], case["step"], case["origin"], case["jitter"], rng, grid_x=case["gx"])
    return torch.from_numpy(pos).cuda()


def _transfer(n, distance, pixel=1.85e-6, wavelength=0.5e-6):
    f = torch.fft.fftfreq(n, d=pixel, dtype=torch.float64, device="cuda")
    kz2 = 1 / wavelength**2 - f[:, None] ** 2 - f[None, :] ** 2
    phase = 2 * math.pi * distance * kz2.clamp(min=0).sqrt()
    return torch.polar((kz2 >= 0).double(), phase).to(torch.complex64)


def _counts(amplitudes, photons, gen):
    """uint16 Poisson counts of the amplitudes' squares and the scale that decodes them;
    `photons(intensity)` is the scale."""
    inten = amplitudes.double() ** 2
    scale = float(np.float32(photons(inten)))
    counts = torch.empty(inten.shape, dtype=torch.uint16, device="cuda")
    for b in range(0, len(inten), 64):
        counts[b:b + 64] = torch.poisson(inten[b:b + 64] / scale, generator=gen).clamp(max=65535).to(torch.int32).to(
            torch.uint16)
    return counts, scale


def prepare(case, seed):
    gen, kind = _generator(seed), case["kind"]
    if kind == "track":
        return {"kind": kind, "stack": _stack(case, gen)}
    if kind in ("coded", "nearfield"):
        n = case["n"]
        truth = _object(n, n, gen)
        aux = (torch.rand(n, n, generator=gen, device="cuda") < 0.5).to(torch.complex64)
        where = (40 * torch.rand(case["count"], 2, generator=gen, device="cuda") - 20) / n
        fixed = {"t1": _transfer(n, 396.95e-6) if kind == "coded" else None, "t2": _transfer(n, 2e-3),
                 "ds": case["ds"], "loss": case["loss"]}
    elif kind == "fourier":
        truth = _object(case["oh"], case["ow"], gen)
        aux = torch.from_numpy(synth.circular_pupil(case["ph"], 0.3)).cuda()
        dx = synth.fpm_dx_for_pupil(case["oh"], case["ph"], 0.1, 0.532, 0.3)
        where = torch.from_numpy(synth.fpm_led_windows(case["oh"], case["ph"], case["gy"], 4.0, 90.0, 0.532, dx)).cuda()
        fixed = {}
    else:
        truth = _object(case["oh"], case["ow"], gen)
        aux = _probe(case["ph"], case["pw"], gen)
        where = _positions(case, seed)
        fixed = {}
    with torch.no_grad():
        amp = torch.cat([_model(kind, truth, aux, where[b:b + 32], fixed) for b in range(0, len(where), 32)])
    if kind in ("base", "operator", "subpixel"):
        counts, scale = _counts(amp, lambda i: float(i.sum(dim=(1, 2)).mean()) / case["photons"], gen)
    elif kind == "fourier":
        counts, scale = _counts(amp, lambda i: float(i.mean(dim=(1, 2)).max()) / case["photons"], gen)
    else:
        counts, scale = _counts(amp, lambda i: float(i.mean()) / case["photons"], gen)
    state = {"kind": kind, "object": _estimate(truth, gen).requires_grad_(True), "aux": aux.requires_grad_(True),
             "where": where.requires_grad_(bool(case.get("shift_grad"))), "counts": counts, "scale": scale, **fixed}
    if kind == "operator":  # the reference's loop keeps the observed amplitudes
        state["observed"] = torch.sqrt(counts.to(torch.float32) * scale)
    return state


def _stack(case, gen):
    """Measured speckle images [count, h, w] under shifts of a few pixels, Poisson noise."""
    h, w, n = case["h"], case["w"], case["count"]
    base = 1 + 0.25 * _low_pass(h, w, 0.8, gen).clamp(-3, 3)
    by = 12 * torch.rand(n, 2, generator=gen, device="cuda", dtype=torch.float64) - 6
    by[0] = 0
    fy, fx = torch.fft.fftfreq(h, device="cuda")[:, None], torch.fft.fftfreq(w, device="cuda")[None, :]
    spec = torch.fft.fft2(base)
    out = torch.empty(n, h, w, device="cuda")
    for b in range(0, n, 32):
        s = by[b:b + 32].float()
        ramp = torch.polar(torch.ones(1, device="cuda"),
                           -2 * math.pi * (fy * s[:, 0, None, None] + fx * s[:, 1, None, None]))
        out[b:b + 32] = torch.poisson(2e3 * torch.fft.ifft2(spec * ramp).real.clamp(min=0), generator=gen)
    return out


# ---------------------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------------------


def run(state):
    """One evaluation: the loss (kept in 32 bits, as the drivers' own) and the gradients."""
    kind = state["kind"]
    if kind == "track":
        x0, y0 = registration.track_position(state["stack"])
        x, y = registration.refine_position(state["stack"], x0, y0)
        return {"track_x": x0, "track_y": y0, "refine_x": x, "refine_y": y}
    obj, aux, where = state["object"], state["aux"], state["where"]
    obj.grad = aux.grad = where.grad = None
    out = {}
    if kind == "operator":
        amp = px.ptychoX_base(obj, aux, where)
        loss = F.mse_loss(amp, state["observed"])
        out["amplitude"] = amp.detach()
    elif kind == "base":
        loss = px.ptychoX_base_loss(obj, aux, where, state["counts"], state["scale"])
    elif kind == "subpixel":
        loss = px.ptychoX_base_subpixel_loss(obj, aux, where, state["counts"], state["scale"])
    elif kind == "fourier":
        loss = px.ptychoX_fourier_loss(obj, aux, where, state["counts"], state["scale"])
    elif kind == "coded":
        loss = px.ptychoX_coded_loss(obj, aux, state["t1"], state["t2"], where, state["ds"], state["counts"],
                                     state["scale"], loss=state["loss"])
    else:
        loss = px.ptychoX_nearfield_loss(obj, aux, state["t2"], where, state["ds"], state["counts"], state["scale"],
                                         loss=state["loss"])
    loss.backward()
    out.update(loss=loss.detach().to(torch.float32), grad_object=obj.grad, grad_aux=aux.grad)
    if where.grad is not None:
        out["grad_shifts"] = where.grad
    return out


def work(case):
    """Bytes: every input read once and every output written once.  Operations: the transforms
    (5 n log2 n each) and about 40 operations a pattern pixel around them."""

    def fft2(h, w):
        return 5.0 * h * w * math.log2(h * w)

    kind = case["kind"]
    if kind == "track":
        h, w, n = case["h"], case["w"], case["count"]
        ch, cw = h - 40, w - 40
        # two registrations: the crop's transform, the doubled correlation's inverse transform, and
        # the upsampled patch, whose smooth separable phase factors have a numerical rank of about 20
        ops = 2 * n * (fft2(ch, cw) + fft2(2 * ch, 2 * cw) + 130.0 * ch * cw) + 2 * n * fft2(h, w)
        ops += sum(n * 84.0 * (1.5 * u) ** 2 for u in (600, 100))
        return {"bytes": 4.0 * n * h * w + 32.0 * n, "flops": ops}
    if kind in ("coded", "nearfield"):
        n, b, low = case["n"], case["count"], (case["n"] // case["ds"]) ** 2
        fields = 6 if kind == "coded" else 5  # object, surface and propagators in, two gradients out
        return {"bytes": 8.0 * n * n * fields + 2.0 * b * low,
                "flops": b * (8 * fft2(n, n) + 100.0 * n * n) + 2 * fft2(n, n)}
    b, p2, o2 = case["gy"] * case["gx"], case["ph"] * case["pw"], case["oh"] * case["ow"]
    counts = 8.0 if kind == "operator" else 2.0  # the operator reads and writes float amplitudes
    transforms = 6 if kind == "subpixel" else 2
    ops = b * (transforms * fft2(case["ph"], case["pw"]) + 40.0 * p2)
    if kind == "fourier":
        ops += 2 * fft2(case["oh"], case["ow"])
    return {"bytes": counts * b * p2 + 16.0 * (o2 + p2), "flops": ops}


# ---------------------------------------------------------------------------------------
# the same in 64 bits, with plain torch
# ---------------------------------------------------------------------------------------


def _crop_windows(obj, pos, ph, pw):
    y = pos[:, 1, None] + torch.arange(ph, device=pos.device)
    x = pos[:, 0, None] + torch.arange(pw, device=pos.device)
    return obj[y[:, :, None], x[:, None, :]]


def _frequencies(n, like):
    return torch.fft.fftfreq(n, d=1.0 / n, dtype=torch.float64, device=like.device)


def _model(kind, obj, aux, where, fixed):
    """Forward amplitudes of some scan units, in the precision of the inputs."""
    if kind in ("base", "operator", "subpixel"):
        ph, pw = aux.shape
        if kind == "subpixel":
            corner = torch.floor(where + 0.5)
            frac = where - corner
            turns = (frac[:, 0, None, None] * _frequencies(pw, aux)[None, None, :] / pw
                     + frac[:, 1, None, None] * _frequencies(ph, aux)[None, :, None] / ph)
            patch = _crop_windows(obj, corner.long(), ph, pw)
            ramp = torch.polar(torch.ones_like(turns), 2 * math.pi * turns).to(obj.dtype)
            patch = torch.fft.ifft2(torch.fft.fft2(patch) * ramp)
        else:
            patch = _crop_windows(obj, where, ph, pw)
        return torch.fft.fftshift(torch.fft.fft2(patch * aux), dim=(-2, -1)).abs()
    if kind == "fourier":
        centred = torch.roll(torch.fft.fft2(obj), (-(obj.shape[0] // 2), -(obj.shape[1] // 2)), dims=(0, 1))
        sub = _crop_windows(centred, where, *aux.shape)
        return torch.fft.ifft2(torch.fft.fftshift(sub * aux, dim=(-2, -1))).abs()
    n, ds = obj.shape[0], fixed["ds"]
    f = _frequencies(n, obj)
    turns = where[:, 0, None, None] * f[None, None, :] + where[:, 1, None, None] * f[None, :, None]
    spec = torch.fft.fft2(obj) * torch.polar(torch.ones_like(turns), 2 * math.pi * turns).to(obj.dtype)
    if fixed["t1"] is not None:
        spec = spec * fixed["t1"]
    s = torch.fft.ifft2(torch.fft.fft2(torch.fft.ifft2(spec) * aux) * fixed["t2"])
    power = (s.real**2 + s.imag**2).reshape(len(s), n // ds, ds, n // ds, ds)
    return power.mean(dim=(2, 4)).sqrt()


def exact(case, seed):
    state = prepare(case, seed)
    kind = state["kind"]
    if kind == "track":
        return _exact_track(state["stack"])
    obj, aux = (state[k].detach().to(torch.complex128).requires_grad_(True) for k in ("object", "aux"))
    where = state["where"].detach()
    refine = state["where"].requires_grad
    where = where.double().requires_grad_(refine) if where.is_floating_point() else where
    fixed = {k: state[k] for k in ("t1", "t2", "ds", "loss") if k in state}
    for k in ("t1", "t2"):
        if fixed.get(k) is not None:
            fixed[k] = fixed[k].to(torch.complex128)
    counts, total, amps = state["counts"], 0.0, []
    observed = state.get("observed")
    chunk = max(1, int(2**25 // (aux.numel())))
    for b in range(0, len(where), chunk):
        amp = _model(kind, obj, aux, where[b:b + chunk], fixed)
        y = observed[b:b + chunk].double() if observed is not None else torch.sqrt(
            counts[b:b + chunk].to(torch.float64) * state["scale"])
        if fixed.get("loss", "mse") == "mse":
            part = ((amp - y) ** 2).sum() / counts.numel()
        else:  # the coded driver's isotropic periodic finite differences
            d = amp - y
            dx, dy = torch.roll(d, -1, dims=2) - d, torch.roll(d, -1, dims=1) - d
            part = torch.sqrt(dx**2 + dy**2 + 1e-5).sum()
        part.backward()
        total += float(part.detach())
        if kind == "operator":
            amps.append(amp.detach())
    out = {"loss": total, "grad_object": obj.grad, "grad_aux": aux.grad}
    if kind == "operator":
        out["amplitude"] = torch.cat(amps)
    if refine:
        out["grad_shifts"] = where.grad
    return out


def _centred(n):
    return torch.fft.ifftshift(torch.arange(-(n // 2), (n + 1) // 2, device="cuda")).double()


def _peak(a):
    """(row, col) of each slice's first maximum in column-major order."""
    i = a.transpose(1, 2).reshape(len(a), -1).argmax(dim=1)
    return i % a.shape[1], i // a.shape[1]


def _register(ref, spectra, usfac):
    """Shifts (col, row) of each spectrum against `ref`: the doubled cross-correlation's peak,
    then the peak of its transform upsampled by `usfac` around it."""
    n, nr, nc = spectra.shape
    xs, ys = [], []
    size = math.ceil(1.5 * usfac)
    mid = size // 2
    for b in range(0, n, 8):
        q = spectra[b:b + 8] * ref.conj()
        pad = torch.zeros(len(q), 2 * nr, 2 * nc, dtype=q.dtype, device="cuda")
        r0, c0 = nr - nr // 2, nc - nc // 2
        pad[:, r0:r0 + nr, c0:c0 + nc] = torch.fft.fftshift(q.conj(), dim=(-2, -1))
        r, c = _peak(torch.fft.ifft2(torch.fft.ifftshift(pad, dim=(-2, -1))).abs())
        half_r, half_c = (torch.fft.ifftshift(torch.arange(-m, m, device="cuda")).double() / 2 for m in (nr, nc))
        at_r, at_c = half_r[r], half_c[c]
        cr, cc = (torch.sign(v * usfac) * torch.floor((v * usfac).abs() + 0.5) for v in (at_r, at_c))
        grid = torch.arange(size, device="cuda").double()

        def kernel(count, centre):
            turns = _centred(count)[None, :, None] * (grid[None, None, :] - mid + centre[:, None, None])
            return torch.polar(torch.ones_like(turns), -2 * math.pi * torch.fmod(turns, count * usfac) / (count * usfac))

        up = kernel(nr, cr).transpose(1, 2) @ (q @ kernel(nc, cc))
        r, c = _peak(up.abs())
        xs.append((cc + (c - mid)) / usfac)
        ys.append((cr + (r - mid)) / usfac)
    return torch.cat(xs), torch.cat(ys)


def _exact_track(stack):
    stack, edge = stack.double(), 20

    def spectra(images):
        return torch.fft.fft2(images[..., edge:images.shape[-2] - edge, edge:images.shape[-1] - edge])

    spec = spectra(stack)
    x0, y0 = _register(spec[0], spec, 600)
    stack = stack / stack.mean(dim=0, keepdim=True)
    n, h, w = stack.shape
    ref = torch.zeros(h, w, dtype=torch.complex128, device="cuda")
    for i in torch.nonzero((x0.abs() > 2) & (y0.abs() > 2)).flatten().tolist():
        turns = _centred(w)[None, :] * x0[i] / w + _centred(h)[:, None] * y0[i] / h
        ref += torch.fft.ifft2(torch.fft.fft2(stack[i]) * torch.polar(torch.ones_like(turns), -2 * math.pi * turns))
    x, y = _register(spectra(ref.abs() / n), spectra(stack), 100)
    return {"track_x": x0, "track_y": y0, "refine_x": x, "refine_y": y}
