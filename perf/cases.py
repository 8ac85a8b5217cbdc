"""Timed cases of the framework: what its users have it do, through its public
entry points, from one thin 128^2 specimen to a 1024-probe frozen-phonon scan.

``listed()`` names twelve calls and ``draw(rng)`` gives more of the same
ranges; ``prepare`` makes a call's inputs on the GPU from a seed, ``run`` is
one call, ``exact`` the same results in 64 bits from plain torch, ``work`` the
bytes and operations that the call cannot do without.

Kinds of calls:

``ms``     ``simulate_fresnel_as``: one probe, a scan of one probe over
           positions (optionally frozen-phonon draws summed per position,
           optionally a detector window), or a batch of different waves
``wpm``    ``simulate_wpm``: adaptive binning, one probe or a few
``grad``   ``simulate_fresnel_as_differentiable`` and its backward: one step
           of an inverse problem, the loss on the patterns
"""
from __future__ import annotations

import math

import numpy as np
import torch

import wideanglepropagation_b200 as wap
from wideanglepropagation_b200.autograd import simulate_fresnel_as_differentiable

# CODATA 2014, as ase.units has them
_H, _C, _ME, _QE = 6.626070040e-34, 299792458.0, 9.10938356e-31, 1.6021766208e-19


def listed():
    return [
        # the smallest call: a thin specimen on a 128^2 window, the reference's defaults (every wavefront returned)
        _ms("fresnel_128_thin", 128, 128, 20, method="fresnel", ps=0.1, dz=2.0, energy=200e3, stack=True),
        # the reference's first example: one convergent probe, 256^2, 20 slices
        _ms("fresnel_256_probe", 256, 256, 20, method="fresnel", ps=0.1, dz=2.0, energy=200e3, stack=True),
        # high-resolution image: a plane wave through 100 slices of a 1024^2 cell, only the exit wave kept
        _ms("as_1024_plane", 1024, 1024, 100, wave="plane"),
        # a notebook's grid: 100 points per side, 100 slices, wavefronts returned
        _ms("as_100_notebook", 100, 100, 100, ps=0.1, stack=True),
        # a small scan on a ragged cell (an orthogonal cell at equal sampling is rarely square)
        _ms("as_240x300_scan", 240, 300, 40, probes=16, ps=0.08),
        # 4D-STEM: 16 x 16 positions x 4 frozen-phonon draws, patterns summed per position
        _ms("scan_256_phonons", 256, 256, 80, probes=1024, draws=4, accumulate=True),
        # 4D-STEM on a wider window, patterns cropped to the detector
        _ms("scan_512_detector", 512, 512, 150, probes=64, max_angle=50.0),
        # partially coherent illumination: a batch of different incident waves
        _ms("modes_256", 256, 256, 80, probes=16, per_probe=True),
        # inverse problem: one gradient step of a 64-probe scan on 512^2
        _grad("grad_512_scan", 512, 64, 64),
        # wide-angle step on a heavy specimen, 16 reference indices evenly spaced
        _wpm("wpm_512_k16", 512, 512, 200, bins=16, power=1.0, amp=80.0, sigma=0.2, dz=2.04, wave="plane"),
        # the reference's own default bins (128, quadratic spacing), a convergent probe, wavefronts returned
        _wpm("wpm_256_default", 256, 256, 40, bins=128, power=2.0, stack=True),
        # a notebook's wide-angle run: 100 points per side, 32 bins
        _wpm("wpm_100_notebook", 100, 100, 100, bins=32, power=2.0, ps=0.1, stack=True),
    ]


def _ms(name, ny, nx, slices, probes=1, draws=1, method="as", wave="probe", per_probe=False, stack=False,
        accumulate=False, max_angle=0.0, ps=0.05, dz=1.3575, energy=300e3, amp=25.0, sigma=0.25):
    return {"kind": "ms", "name": name, "ny": ny, "nx": nx, "slices": slices, "probes": probes, "draws": draws,
            "method": method, "wave": wave, "per_probe": per_probe, "stack": stack, "accumulate": accumulate,
            "max_angle": max_angle, "ps": ps, "dz": dz, "energy": energy, "amp": amp, "sigma": sigma}


def _wpm(name, ny, nx, slices, bins, power, probes=1, wave="probe", stack=False, ps=0.05, dz=1.3575, energy=300e3,
         amp=25.0, sigma=0.25):
    return {"kind": "wpm", "name": name, "ny": ny, "nx": nx, "slices": slices, "probes": probes, "bins": bins,
            "power": power, "wave": wave, "stack": stack, "ps": ps, "dz": dz, "energy": energy, "amp": amp,
            "sigma": sigma}


def _grad(name, n, slices, probes, ckpt=0, ps=0.05, dz=2.0, energy=300e3, amp=20.0, sigma=0.3):
    return {"kind": "grad", "name": name, "ny": n, "nx": n, "slices": slices, "probes": probes, "ckpt": ckpt,
            "ps": ps, "dz": dz, "energy": energy, "amp": amp, "sigma": sigma}


# ---------------------------------------------------------------------------
# drawn cases
# ---------------------------------------------------------------------------
def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _side(rng, lo=32, hi=1024):
    """A grid side: mostly powers of two, else any number of the range (odd ones and primes among them)."""
    p = rng.random()
    if p < 0.5:
        return 1 << rng.randint(int(math.log2(lo)), int(math.log2(hi)))
    if p < 0.75:   # what a user types: a round number
        return max(lo, min(hi, 10 * _log(rng, lo / 10, hi / 10)))
    return _log(rng, lo, hi)


def _pow2(n):
    return n & (n - 1) == 0


def _grid(rng):
    ny = _side(rng)
    nx = ny if rng.random() < 0.7 else max(32, min(1024, _side(rng, 32, 1024)))
    return ny, nx


def draw(rng):
    kind = rng.choices(["ms", "wpm", "grad"], [3, 2, 1])[0]
    energy = rng.choice([80e3, 200e3, 300e3])
    # projected peak of the atoms (V A): light to heavy
    amp = round(math.exp(rng.uniform(math.log(15.0), math.log(400.0))), 1)
    dz = round(rng.uniform(1.0, 4.0), 3)
    ps = round(rng.uniform(0.04, 0.12), 4)
    slices = _log(rng, 5, 200)
    if kind == "grad":
        n = 1 << rng.randint(6, 9)
        probes = _log(rng, 1, 128)
        while probes * slices * n * n > 1.0e9:
            slices = max(5, slices // 2)
            probes = max(1, probes // 2)
        return _drop_name(_grad("", n, slices, probes, rng.choice([0, 0, 1, 4]), ps, dz, energy, min(amp, 60.0), 0.3))
    ny, nx = _grid(rng)
    px = ny * nx
    slow = 1 if _pow2(ny) and _pow2(nx) else 4
    if kind == "wpm":
        bins = rng.choice([4, 8, 16, 16, 32, 64, 128, 128, 256])
        probes = rng.choice([1, 1, 1, 2, 4])
        while probes * bins * px > 1.5e8:
            probes, bins = max(1, probes // 2), bins // 2
        while probes * slices * px * (bins + 1) * slow > 3.0e9 and slices > 1:
            slices = slices // 2
        return _drop_name(_wpm("", ny, nx, slices, bins, rng.choice([1.0, 2.0]), probes, rng.choice(["probe", "plane"]),
                               rng.random() < 0.5 and probes * slices * px < 1.0e8, ps, dz, energy, amp, 0.25))
    shape = rng.choice(["one", "one", "scan", "scan", "modes"])
    probes = 1 if shape == "one" else _log(rng, 2, 1024 if shape == "scan" else 48)
    while probes * px > 6.7e7:
        probes = max(1, probes // 2)
    draws = rng.choice([1, 1, 2, 4]) if shape == "scan" and probes >= 8 else 1
    while (probes * slices * px * slow > 2.5e9 or draws * slices * px > 1.05e8) and slices > 1:
        slices = slices // 2
    return _drop_name(_ms("", ny, nx, slices, probes, draws, rng.choice(["as", "fresnel"]),
                          "probe" if shape != "one" else rng.choice(["probe", "plane"]), shape == "modes",
                          rng.random() < 0.4 and probes * slices * px < 1.0e8, draws > 1,
                          rng.choice([0.0, 0.0, 40.0]), ps, dz, energy, amp, 0.25))


def _drop_name(c):
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _wavelength(energy):
    return _H * _C / math.sqrt(energy * (2 * _ME * _C * _C / _QE + energy)) / _QE * 1.0e10


def _potential(c, g, draws=1):
    """(draws, slices, ny, nx) float32 volts: Gaussian atoms (``amp`` V A, ``sigma`` A) at random places of each
    slice, one per about 9 A^2 as in a crystal's atomic layer, periodic, divided by the slice thickness."""
    dev = _device()
    ny, nx, ps, rows = c["ny"], c["nx"], c["ps"], draws * c["slices"]
    ly, lx = ny * ps, nx * ps
    atoms = max(4, int(ly * lx / 9.0))
    at = torch.rand((rows, atoms, 2), device=dev, generator=g, dtype=torch.float64)

    def profile(n, length, p):
        d = torch.remainder(torch.arange(n, device=dev, dtype=torch.float64) * ps - p[..., None] * length
                            + length / 2, length) - length / 2
        return torch.exp(-d * d / (2 * c["sigma"] ** 2))

    out = torch.empty((rows, ny, nx), device=dev, dtype=torch.float32)
    step = max(1, int(5e7 // (atoms * (ny + nx) + ny * nx)))
    for r in range(0, rows, step):
        gy, gx = profile(ny, ly, at[r:r + step, :, 0]), profile(nx, lx, at[r:r + step, :, 1])
        out[r:r + step] = (c["amp"] / c["dz"]) * torch.bmm(gy.transpose(1, 2), gx)
    return out.reshape(draws, c["slices"], ny, nx)


def _freq2(c):
    dev = _device()
    fy = torch.fft.fftfreq(c["ny"], d=c["ps"], dtype=torch.float64, device=dev)
    fx = torch.fft.fftfreq(c["nx"], d=c["ps"], dtype=torch.float64, device=dev)
    return fy[:, None] ** 2 + fx[None, :] ** 2


def _wave(c, g, count=0):
    """A convergent probe (25 mrad, -50 A) at the grid's centre or a plane wave; ``count`` different probes
    (a random defocus and tilt each) with ``count`` > 0."""
    dev = _device()
    ny, nx = c["ny"], c["nx"]
    if c.get("wave", "probe") == "plane":
        return torch.ones((ny, nx), dtype=torch.complex64, device=dev)
    lam, f2 = _wavelength(c["energy"]), _freq2(c)
    inside = (torch.sqrt(f2) * lam < 0.025).to(torch.float64)
    df = -50.0 - 40.0 * torch.rand((max(1, count), 1, 1), device=dev, generator=g, dtype=torch.float64)
    spectrum = torch.polar(inside.expand(df.shape[0], ny, nx), -math.pi * lam * df * f2)
    p = torch.fft.fftshift(torch.fft.ifft2(spectrum), dim=(-2, -1))
    p = p * (math.sqrt(ny * nx) / torch.linalg.vector_norm(p, dim=(-2, -1), keepdim=True))
    p = p.to(torch.complex64)
    return p if count else p[0]


def _raster(c):
    """Probe centres of the case's scan, repeated for each draw, and which draw and which position each has."""
    per = c["probes"] // c["draws"]
    side = max(1, int(math.floor(math.sqrt(per))))
    rows = -(-per // side)
    y = (np.arange(rows) * c["ny"]) // rows
    x = (np.arange(side) * c["nx"]) // side
    pos = np.stack([np.repeat(y, side), np.tile(x, rows)], 1)[:per].astype(np.int32)
    many = c["probes"]
    which = np.arange(many) % per
    return pos[which], np.minimum(np.arange(many) // per, c["draws"] - 1).astype(np.int32), which.astype(np.int64)


def _inputs(c, seed):
    """The case's arrays, from the seed alone."""
    g = torch.Generator(device=_device())
    g.manual_seed(1_000_003 * int(seed) + 17)
    s = {"case": c}
    if c["kind"] == "ms":
        s["V"] = _potential(c, g, c["draws"])
        s["wave"] = _wave(c, g, c["probes"] if c["per_probe"] else 0)
        if c["probes"] > 1 and not c["per_probe"]:
            pos, draws, which = _raster(c)
            s["positions"] = torch.as_tensor(pos).to(_device())
            s["draw"], s["which"] = draws, which
        return s
    s["V"] = _potential(c, g)
    s["wave"] = _wave(c, g)
    if c["probes"] > 1 or c["kind"] == "grad":
        pos, _, _ = _raster(dict(c, draws=1))
        s["positions"] = torch.as_tensor(pos).to(_device())
    if c["kind"] == "grad":
        # the measured patterns: the bright-field disk, with speckle of a thin specimen and a weak diffuse floor
        disk = torch.fft.fftshift(torch.fft.fft2(s["wave"].to(torch.complex128)).abs() ** 2)
        k = 8
        blur = torch.rand((c["probes"], 1, c["ny"] // k, c["nx"] // k), device=_device(), generator=g)
        speckle = torch.nn.functional.interpolate(blur, scale_factor=k, mode="nearest")[:, 0]
        s["target"] = ((0.5 + speckle) * disk.to(torch.float32) + 1e-3 * float(disk.mean()) * speckle).contiguous()
    return s


def prepare(case, seed):
    s = _inputs(case, seed)
    c = case
    if c["kind"] == "ms":
        kernel = wap.angular_spectrum_propagation_kernel if c["method"] == "as" else wap.fresnel_propagation_kernel
        s["H"] = kernel(c["ny"], c["nx"], (c["ps"], c["ps"]), c["dz"], c["energy"])
        if c["draws"] == 1:
            s["V"] = s["V"][0]
    elif c["kind"] == "grad":
        s["H"] = wap.fresnel_propagation_kernel(c["ny"], c["nx"], (c["ps"], c["ps"]), c["dz"], c["energy"])
        s["V"] = s["V"][0].requires_grad_(True)
    else:
        s["V"] = s["V"][0]
    return s


# ---------------------------------------------------------------------------
# one call
# ---------------------------------------------------------------------------
def run(state):
    s, c = state, state["case"]
    if c["kind"] == "ms":
        options = {}
        if "positions" in s:
            options["positions"] = s["positions"]
        if c["draws"] > 1:
            options["draw"] = s["draw"]
        if c["accumulate"]:
            options["accumulate"] = s["which"]
        if c["max_angle"]:
            options.update(max_angle=c["max_angle"], sampling=(c["ps"], c["ps"]))
        return wap.simulate_fresnel_as(s["V"], s["wave"], s["H"], c["dz"], c["energy"],
                                       return_wavefronts=c["stack"], **options)
    if c["kind"] == "wpm":
        options = {"positions": s["positions"]} if "positions" in s else {}
        return wap.simulate_wpm(s["V"], s["wave"], c["dz"], c["energy"], (c["ps"], c["ps"]), n_bins=c["bins"],
                                power_spacing=c["power"], return_wavefronts=c["stack"], **options)
    s["V"].grad = None
    exit_wave, dp = simulate_fresnel_as_differentiable(s["V"], s["wave"], s["H"], c["dz"], c["energy"],
                                                       positions=s["positions"], ckpt_every=c["ckpt"] or None)
    loss = ((dp - s["target"]) ** 2).sum()
    loss.backward()
    return {"exit": exit_wave.detach(), "dp": dp.detach(), "loss": loss.detach(), "grad": s["V"].grad}


# ---------------------------------------------------------------------------
# what one call cannot do without
# ---------------------------------------------------------------------------
def _pattern_shape(c):
    if not c.get("max_angle"):
        return c["ny"], c["nx"]
    top = c["max_angle"] / (_wavelength(c["energy"]) * 1000.0)
    hy = max(0, min(int(math.floor(top * c["ny"] * c["ps"])), c["ny"] // 2))
    hx = max(0, min(int(math.floor(top * c["nx"] * c["ps"])), c["nx"] // 2))
    return max(1, min(2 * hy + 1, c["ny"])), max(1, min(2 * hx + 1, c["nx"]))


def work(case):
    """Bytes: each input read once, each output written once.  Operations: 5 n log2 n for a transform of n points,
    two per slice step, and the pointwise products beside them (how many reference fields a wide-angle step forms
    is the implementation's matter: counted as one); the gradient sweeps the slices forward once and backward once."""
    c = case
    px, B, N = c["ny"] * c["nx"], c["probes"], c["slices"]
    lg = math.log2(px)
    if c["kind"] == "grad":
        return {"bytes": 8.0 * N * px + 24.0 * px + 16.0 * B * px,
                "flops": B * N * px * 2.0 * (10.0 * lg + 24.0)}
    out = 8.0 * B * px + (8.0 * B * N * px if c["stack"] else 0.0)
    if c["kind"] == "wpm":
        return {"bytes": 4.0 * N * px + 8.0 * px + out + 4.0 * B * px,
                "flops": B * N * px * (10.0 * lg + 30.0)}
    dy, dx = _pattern_shape(c)
    patterns = B // c["draws"] if c["accumulate"] else B
    waves = B if c["per_probe"] else 1
    return {"bytes": 4.0 * c["draws"] * N * px + 16.0 * px + 8.0 * waves * px + out + 4.0 * patterns * dy * dx,
            "flops": B * N * px * (10.0 * lg + 24.0)}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def _rest_energy():
    return _ME * _C * _C / _QE


def _index_minus_one(V, energy):
    """n - 1 of the potential in volts, without cancellation."""
    e0 = _rest_energy()
    r = V * (2 * e0 + 2 * energy + V) / (energy * (2 * e0 + energy))
    return r / (torch.sqrt(1.0 + r) + 1.0)


def _cis(phase):
    return torch.polar(torch.ones_like(phase), phase)


def _transfer(c):
    lam, f2 = _wavelength(c["energy"]), _freq2(c)
    if c.get("method", "fresnel") == "fresnel":
        return _cis(2 * math.pi / lam * c["dz"] - math.pi * lam * c["dz"] * f2)
    q = 1.0 / lam ** 2 - f2
    root = 2 * math.pi * c["dz"] * torch.sqrt(q.abs())
    return torch.where(q >= 0, _cis(root), torch.exp(-root).to(torch.complex128))


def _moved(wave, positions, first, last):
    """The waves of probes first .. last - 1 in complex128."""
    if wave.ndim == 3:
        return wave[first:last].to(torch.complex128)
    w = wave.to(torch.complex128)
    if positions is None:
        return w[None]
    ny, nx = w.shape
    return torch.stack([torch.roll(w, (int(y) - ny // 2, int(x) - nx // 2), (0, 1))
                        for y, x in positions[first:last].cpu().tolist()])


def _intensity(psi):
    return torch.fft.fftshift(torch.fft.fft2(psi).abs() ** 2, dim=(-2, -1))


def _chunk(c):
    return max(1, int(3.3e7 // (c["ny"] * c["nx"])))


def _exact_ms(c, s):
    V, H, B = s["V"], _transfer(c), c["probes"]
    dy, dx = _pattern_shape(c)
    y0, x0 = c["ny"] // 2 - dy // 2, c["nx"] // 2 - dx // 2
    phase = 2 * math.pi * c["dz"] / _wavelength(c["energy"])
    exits, patterns, stacks = [], [], []
    for b in range(0, B, _chunk(c)):
        e = min(B, b + _chunk(c))
        psi = _moved(s["wave"], s.get("positions"), b, e)
        draws = torch.as_tensor(s["draw"][b:e].astype(np.int64), device=V.device) if c["draws"] > 1 else None
        kept = []
        for k in range(c["slices"]):
            t = _cis(phase * _index_minus_one(V[:, k].double(), c["energy"]))
            psi = torch.fft.ifft2(H * torch.fft.fft2(psi * (t[draws] if draws is not None else t[0])))
            if c["stack"]:
                kept.append(psi)
        exits.append(psi)
        patterns.append(_intensity(psi)[..., y0:y0 + dy, x0:x0 + dx])
        if c["stack"]:
            stacks.append(torch.stack(kept, 1))
    dp = torch.cat(patterns)
    if c["accumulate"]:
        which = torch.as_tensor(s["which"], device=dp.device)
        dp = torch.zeros((int(which.max()) + 1, dy, dx), dtype=dp.dtype, device=dp.device).index_add_(0, which, dp)
    exit_wave, stack = torch.cat(exits), torch.cat(stacks) if stacks else None
    if B == 1 and not c["per_probe"]:
        return exit_wave[0], dp[0], stack[0] if stack is not None else None
    return exit_wave, dp, stack


def _exact_wpm(c, s):
    V, K = s["V"][0].double(), c["bins"]
    k0 = 2 * math.pi / _wavelength(c["energy"])
    kp2 = (2 * math.pi) ** 2 * _freq2(c)
    t = torch.from_numpy(np.linspace(0, 1, K) ** c["power"]).to(V.device)
    psi = _moved(s["wave"], s.get("positions"), 0, c["probes"])
    kept = []
    for k in range(c["slices"]):
        d = _index_minus_one(V[k], c["energy"])
        refs = d.min() + (d.max() - d.min()) * t
        right = torch.searchsorted(refs, d.reshape(-1)).reshape(d.shape).clamp(1, K - 1)
        gap = refs[right] - refs[right - 1]
        w = ((d - refs[right - 1]) / torch.where(gap == 0, torch.ones_like(gap), gap)).clamp(0, 1)
        w = w * w * (3 - 2 * w)
        spectrum = torch.fft.fft2(psi)
        new = torch.zeros_like(psi)
        for j in range(K):
            q = ((1.0 + refs[j]) * k0) ** 2 - kp2
            root = c["dz"] * torch.sqrt(q.abs())
            h = torch.where(q >= 0, _cis(root), torch.exp(-root).to(torch.complex128))
            weight = torch.where(right == j, w, torch.zeros_like(w)) + torch.where(right - 1 == j, 1 - w,
                                                                                   torch.zeros_like(w))
            new += weight * torch.fft.ifft2(h * spectrum)
        psi = new
        if c["stack"]:
            kept.append(psi)
    dp, stack = _intensity(psi), torch.stack(kept, 1) if kept else None
    if c["probes"] == 1:
        return psi[0], dp[0], stack[0] if stack is not None else None
    return psi, dp, stack


def _exact_grad(c, s):
    V, H = s["V"][0].double(), _transfer(dict(c, method="fresnel"))
    px, N, E = c["ny"] * c["nx"], c["slices"], c["energy"]
    phase, e0 = 2 * math.pi * c["dz"] / _wavelength(E), _rest_energy()
    grad = torch.zeros_like(V)
    exits, patterns, loss = [], [], 0.0
    step = max(1, min(c["probes"], int(1.5e8 // (px * N))))
    trans = lambda k: _cis(phase * _index_minus_one(V[k], E))  # noqa: E731
    for b in range(0, c["probes"], step):
        e = min(c["probes"], b + step)
        psi, seen = _moved(s["wave"], s["positions"], b, e), []
        for k in range(N):
            seen.append(psi * trans(k))
            psi = torch.fft.ifft2(H * torch.fft.fft2(seen[-1]))
        z = torch.fft.fft2(psi)
        dp = torch.fft.fftshift(z.abs() ** 2, dim=(-2, -1))
        off = dp - s["target"][b:e].double()
        loss = loss + (off ** 2).sum()
        lam = px * torch.fft.ifft2(torch.fft.ifftshift(2 * off, dim=(-2, -1)) * z)
        for k in reversed(range(N)):
            lam = torch.fft.ifft2(H.conj() * torch.fft.fft2(lam))
            a = seen[k]
            grad[k] += 2.0 * (lam.real * -a.imag + lam.imag * a.real).sum(0)
            lam = lam * trans(k).conj()
        exits.append(psi)
        patterns.append(dp)
    n = 1.0 + _index_minus_one(V, E)
    grad = grad * phase * (E + e0 + V) / (E * (2 * e0 + E)) / n
    return {"exit": torch.cat(exits), "dp": torch.cat(patterns), "loss": loss, "grad": grad}


def exact(case, seed):
    c, s = case, _inputs(case, seed)
    return {"ms": _exact_ms, "wpm": _exact_wpm, "grad": _exact_grad}[c["kind"]](c, s)
