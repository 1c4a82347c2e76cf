"""Timed cases of the angular-spectrum march and of the learned KT step.

Each case is one call that a user's program makes: ``angular_spectrum_solve`` on
a host field (the reference's own entry point, with its screens, sources and
boundary options), ``solve_batch`` on several instances, the learned KT step on
device columns and one training step of its network.  Grids are those of the
repository's validation cases (odd and prime sizes), of its benchmark
workloads (power-of-two and 3*2^k sizes) and round numbers in between.

``exact`` restates the same mathematics in 64 bits with plain torch.
"""
import math

import numpy as np
import torch
import torch.nn.functional as F

from angularspectrum_heterogeneous_gb300 import SolverParams, angular_spectrum_solve, solve_batch
from angularspectrum_heterogeneous_gb300.corrector import (Corrector, init_params, learned_flux)
from angularspectrum_heterogeneous_gb300.sources import CompactPlane

C0, RHO0 = 1540.0, 1000.0

SOLVE = dict(kind="solve", nx=0, ny=0, nt=0, dx=1e-4, dt=1.3e-8, dz=4e-4, prop=0.0, f0=3e6,
             p0=1e6, beta=3.5, alpha0=0.5, split=True, flux="kt", tvd=False, adaptive=True,
             taper="quadratic", band=0.2, fw=False, sa=False, sa_strength=0.8, obl=False,
             source="piston", screens=0, bowl=False, cycles=3.0)


def _solve(name, **kw):
    return dict(SOLVE, name=name, **kw)


def listed():
    return [
        # the smallest grid in use: a broadband plane pulse through a lossy medium on 5 x 5
        # columns (attenuation and dispersion check), 30 steps with a partial last one
        _solve("attenuation_5x5x1001", nx=5, ny=5, nt=1001, dx=1.7111e-4, dt=1 / 60e6,
               dz=6.8444e-4, prop=20e-3, beta=0.0, alpha0=1.0, taper="", adaptive=False,
               source="plane"),
        # boundary study: a wide aperture toward the edges with every boundary extra on
        _solve("reflection_81x81x101", nx=81, ny=81, nt=101, prop=30 * 4e-4, beta=0.0, alpha0=-1.0,
               flux="rusanov", adaptive=False, taper="wendland", band=0.15, fw=True, sa=True,
               sa_strength=0.5, cycles=1.5, p0=1e3),
        # step-size study: a strongly nonlinear aperture pulse, KT, no absorbing layer
        _solve("convergence_51x51x401", nx=51, ny=51, nt=401, prop=24 * 4e-4, p0=1.5e6, taper="",
               adaptive=False, cycles=1.5),
        # analytic comparison: a focused piston in a linear lossless medium, sequential steps
        _solve("focused_257x257x601", nx=257, ny=257, nt=601, dx=7.5e-5, dt=1e-8, dz=1.5e-4,
               prop=6 * 1.5e-4, f0=4e6, beta=0.0, alpha0=0.0, split=False, flux="rusanov",
               adaptive=False, taper="", p0=3e5),
        # a tissue model on a grid of round numbers: KT, all boundary extras, two phase screens
        _solve("tissue_200x180x400", nx=200, ny=180, nt=400, prop=10 * 4e-4, fw=True, sa=True,
               screens=2),
        # nonlinearity scaled by the beam's obliquity on a mid-size grid
        _solve("oblique_96x96x192", nx=96, ny=96, nt=192, prop=20 * 4e-4, taper="wendland",
               obl=True),
        # the CPU-sized piston workload: Strang, TVD-Rusanov, Wendland taper
        _solve("piston_128x128x256", nx=128, ny=128, nt=256, dx=3.08e-4, dt=4e-8, dz=2.5e-4,
               prop=24 * 2.5e-4, f0=1e6, p0=4e5, flux="rusanov", tvd=True, taper="wendland"),
        # transcranial bowl: source planes injected slice by slice, skull-like screens, linear
        # water (26 of its 260 steps)
        _solve("bowl_384x384x512", nx=384, ny=384, nt=512, dx=3.08e-4, dt=4e-8, dz=3.08e-4,
               prop=26 * 3.08e-4, f0=1e6, p0=4e5, beta=0.0, alpha0=-1.0, flux="rusanov",
               taper="wendland", band=0.15, fw=True, sa=True, sa_strength=0.5, screens=6,
               bowl=True),
        # the shock-forming workload at full size (10 of its 700 steps)
        _solve("shock_512x512x1024", nx=512, ny=512, nt=1024, dx=1.5e-4, dt=1e-8, dz=1e-4,
               prop=10 * 1e-4, f0=2e6, p0=2e6, fw=True, sa=True, cycles=5.0),
        # independent instances of uneven size marched together, KT sub-cycled per column
        dict(name="batch_8", kind="batch", count=8, steps=8, largest=256, cfl=0.002),
        # the learned KT step on a batch of columns
        dict(name="learned_16384x1024", kind="learned", cols=16384, nt=1024),
        # one training step of its network
        dict(name="train_1024x1024", kind="train", cols=1024, nt=1024),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["solve"] * 9 + ["batch", "learned", "train"])
    if what == "batch":
        return dict(kind="batch", count=rng.randint(2, 8), steps=rng.randint(4, 8),
                    largest=rng.choice([192, 256]), cfl=rng.uniform(0.001, 0.004))
    if what in ("learned", "train"):
        nt = 128 * rng.randint(1, 8)
        return dict(kind=what, cols=_spread(rng, 64, 16384 if what == "learned" else 1024), nt=nt)
    style = rng.choice(["odd", "odd", "round", "fast"])
    if style == "fast":  # sizes with the benchmark's factors
        nx = ny = rng.choice([64, 96, 128, 192, 256, 384])
        nt = rng.choice([128, 192, 256, 384, 512, 768, 1024])
    else:
        nx, ny, nt = _spread(rng, 9, 300), _spread(rng, 9, 300), _spread(rng, 64, 1000)
        if rng.random() < 0.5:
            ny = nx
        if style == "odd":
            nx, ny, nt = nx | 1, ny | 1, nt | 1
        else:
            nx, ny, nt = 10 * (nx // 10 + 1), 10 * (ny // 10 + 1), 10 * (nt // 10 + 1)
    # steps: what a call marches in about the time of the listed cases
    steps = max(2, min(16, int((3e8 if style == "fast" else 6e7) / (nx * ny * nt))))
    flux, tvd = rng.choice([("kt", False), ("rusanov", True), ("rusanov", False)])
    fw = rng.random() < 0.5
    return dict(SOLVE, nx=nx, ny=ny, nt=nt, prop=steps * 4e-4, flux=flux, tvd=tvd,
                split=rng.random() < 0.8, taper=rng.choice(["quadratic", "wendland"]), fw=fw,
                sa=fw and rng.random() < 0.7, obl=rng.random() < 0.15,
                screens=rng.choice([0, 0, 0, 2]), p0=rng.uniform(2e5, 1e6))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _axis(n, d):
    return (torch.arange(n, device="cuda", dtype=torch.float64) - (n - 1) / 2.0) * d


def _field(c, rng):
    """A pulse of the aperture: focused piston, or a plane wave; amplitude, focus and carrier
    phase vary with the seed."""
    x, y, t = _axis(c["nx"], c["dx"]), _axis(c["ny"], c["dx"]), _axis(c["nt"], c["dt"])
    amp, phase = c["p0"] * rng.uniform(0.9, 1.0), rng.uniform(0.0, math.pi)
    w0 = 2 * math.pi * c["f0"]

    def pulse(tau):
        return amp * torch.exp(-(1.05 * tau * w0 / (c["cycles"] * math.pi)) ** 4) * \
            torch.sin(w0 * tau + phase)

    if c["source"] == "plane":
        u = (amp * torch.exp(-0.5 * (t * c["f0"] / 0.15) ** 2) * torch.sin(w0 * t + phase))
        return u.float().expand(c["nx"], c["ny"], c["nt"]).cpu().contiguous().numpy()
    width = min(c["nx"], c["ny"]) * c["dx"]
    r2 = x[:, None] ** 2 + y[None, :] ** 2
    ap = r2 <= (rng.uniform(0.28, 0.32) * width) ** 2
    delay = r2 / (2 * rng.uniform(1.5, 2.0) * width * C0)
    delay = torch.where(ap, delay - delay[ap].mean(), torch.zeros_like(delay))
    u = torch.zeros((c["nx"], c["ny"], c["nt"]), device="cuda", dtype=torch.float32)
    for i in range(0, c["nx"], 64):
        s = slice(i, i + 64)
        u[s] = (pulse(t[None, None, :] + delay[s][:, :, None]) * ap[s][:, :, None]).float()
    return u.cpu().numpy()


def _smooth(nx, ny, rng):
    """A smooth random map in [-1, 1]."""
    x = torch.linspace(-1, 1, nx, device="cuda", dtype=torch.float64)[:, None]
    y = torch.linspace(-1, 1, ny, device="cuda", dtype=torch.float64)[None, :]
    m = 0.0
    for _ in range(6):
        kx, ky, ph = rng.uniform(-12, 12), rng.uniform(-12, 12), rng.uniform(0, 2 * math.pi)
        m = m + torch.sin(kx * x + ky * y + ph) / 6
    return m


def _screens(c, rng):
    steps = int(round(c["prop"] / c["dz"]))
    out = []
    for k in range(c["screens"]):
        z = c["dz"] * (0.5 + (k + 1) * steps // (c["screens"] + 1))
        ph = (1.5 * _smooth(c["nx"], c["ny"], rng)).float().cpu().numpy()
        amp = (0.85 + 0.15 * _smooth(c["nx"], c["ny"], rng)).float().cpu().numpy()
        out.append((z, ph, amp) if k % 2 == 0 else (z, ph))
    return out


def _bowl(c, rng):
    """Compact source planes of a spherical cap (80 mm radius of curvature) sliced by dz: each
    slice drives its annulus of columns with a delayed pulse."""
    roc, f0 = 80e-3, c["f0"]
    x, y, t = _axis(c["nx"], c["dx"]), _axis(c["ny"], c["dx"]), _axis(c["nt"], c["dt"])
    r2 = x[:, None] ** 2 + y[None, :] ** 2
    depth = (roc - torch.sqrt(torch.clamp(roc ** 2 - r2, min=0.0))).reshape(-1)
    amp, phase, w0 = c["p0"] * rng.uniform(0.9, 1.0), rng.uniform(0, math.pi), 2 * math.pi * f0
    out = []
    for k in range(1, int(round(c["prop"] / c["dz"]))):
        cols = torch.nonzero((depth > k * c["dz"]) & (depth <= (k + 1) * c["dz"])).reshape(-1)
        tau = t[None, :] - (depth[cols][:, None] - k * c["dz"]) / C0
        v = amp * torch.exp(-(1.05 * tau * w0 / (3 * math.pi)) ** 4) * torch.sin(w0 * tau + phase)
        out.append((k * c["dz"], CompactPlane(shape=(c["nx"], c["ny"], c["nt"]),
                                              cols=cols.int().cpu().numpy(),
                                              values=v.float().cpu().numpy())))
    return out


def _params(c):
    return SolverParams(
        dX=c["dx"], dY=c["dx"], dT=c["dt"], c0=C0, rho0=RHO0, beta=c["beta"], alpha0=c["alpha0"],
        attenPow=1.0, f0=c["f0"], propDist=c["prop"], boundaryFactor=c["band"],
        useSplitStep=c["split"], useAdaptiveFiltering=c["adaptive"], useTVD=c["tvd"],
        dZmin=c["dz"], useBoundaryLayer=c["taper"] != "",
        boundaryProfile=c["taper"] or "quadratic", useFreqWeightedBoundary=c["fw"],
        useSuperAbsorbing=c["sa"], superAbsorbingStrength=c["sa_strength"],
        fluxScheme="kt" if c["flux"] == "kt" else "rusanov", useNonlinearityObliquity=c["obl"])


def _instances(c):
    """The grids of a batch, uneven: the largest first."""
    sizes = [n for n in (256, 192, 128) if n <= c["largest"]]
    out = []
    for i in range(c["count"]):
        n, nt = sizes[i % len(sizes)], (256, 512, 1024)[(i // 2) % 3]
        out.append(dict(SOLVE, nx=n, ny=n, nt=nt, dx=3.08e-4, dt=4e-8, dz=2.5e-4,
                        prop=c["steps"] * 2.5e-4, f0=1e6, p0=2.5e6 / (1 + i % 4),
                        taper="wendland"))
    return out


LEARN = dict(beta=3.5, dz=2e-3, dt=1e-8, cfl=0.01, min_sub=10, shock=0.5)


def _columns(cols, nt, rng):
    """Columns of a focused beam: pulses of 0.2 to 3 MPa, 1 to 3 MHz, steepened by their second
    harmonic."""
    g = torch.Generator().manual_seed(rng.randrange(1 << 30))
    p, f, ph, k = torch.rand((4, cols, 1), generator=g, dtype=torch.float64).cuda()
    t = _axis(nt, LEARN["dt"])[None, :]
    w = 2 * math.pi * (1e6 + 2e6 * f)
    env = torch.exp(-(t / (0.3 * nt * LEARN["dt"])) ** 4)
    s = torch.sin(w * t + 6.28 * ph) + 0.3 * k * torch.sin(2 * w * t + 12.57 * ph)
    return ((0.2e6 + 2.8e6 * p) * env * s).float().contiguous()


def _theta(rng):
    """Weights of a network that corrects: the last layer's size gives corrections of order one."""
    return init_params(seed=rng.randrange(1 << 30), last_scale=0.3)


def _training(c, rng):
    g = torch.Generator().manual_seed(rng.randrange(1 << 30))
    u = _columns(c["cols"], c["nt"], rng)
    x = (u / 1e6).contiguous()
    y = (torch.roll(x, 1, 1) - 2 * x + torch.roll(x, -1, 1)).contiguous()
    m = (torch.rand((c["cols"], 1), generator=g) < 0.7).float().cuda().expand_as(x).contiguous()
    m[:, 0] = 0.0
    m[:, -1] = 0.0
    return x, y, m


def _rng(seed):
    import random
    return random.Random(seed)


def prepare(case, seed):
    rng = _rng(seed)
    if case["kind"] == "solve":
        prm = _params(case)
        u = _field(case, rng)
        if case["screens"]:
            prm.phaseScreens = _screens(case, rng)
        if case["bowl"]:
            prm.sourcePlanes = _bowl(case, rng)
        return dict(kind="solve", field=u, params=prm)
    if case["kind"] == "batch":
        inst = _instances(case)
        return dict(kind="batch", fields=[_field(i, rng) for i in inst],
                    params=[_params(i) for i in inst], cfl=case["cfl"])
    if case["kind"] == "learned":
        net = Corrector(theta=_theta(rng))
        net.set_output_scale(0.5)
        return dict(kind="learned", net=net, cols=_columns(case["cols"], case["nt"], rng))
    net = Corrector(theta=_theta(rng))
    return dict(kind="train", net=net, batch=_training(case, rng))


def run(state):
    if state["kind"] == "solve":
        return angular_spectrum_solve(state["field"], state["params"], verbose=False)
    if state["kind"] == "batch":
        return solve_batch(state["fields"], state["params"], kt_cfl_target=state["cfl"],
                           kt_max_subcycles=256)
    if state["kind"] == "learned":
        out, n = learned_flux(state["net"], state["cols"], _n_coef(LEARN["beta"]), LEARN["dz"],
                              LEARN["dt"], LEARN["cfl"], LEARN["min_sub"], LEARN["shock"])
        return out, n
    x, y, m = state["batch"]
    return state["net"].train_step(x, y, m, 1e-6, want_grad=True)


# ---------------------------------------------------------------------------
# the work of one pass
# ---------------------------------------------------------------------------
def _solve_work(c):
    v = c["nx"] * c["ny"] * c["nt"]
    steps = math.ceil(c["prop"] / c["dz"] - 1e-9)
    # per step: 3 (Strang) or 2 spectral stages of a forward and an inverse real 3-D
    # transform, 2.5 log2(v) each per sample, and about 60 operations of the Burgers step
    stages = 3 if c["split"] else 2
    flops = steps * v * (stages * 2 * 2.5 * math.log2(v) + 60)
    return 4 * (2 * v + 4 * c["nx"] * c["ny"] * steps + c["nt"] * steps), flops


def work(case):
    if case["kind"] in ("solve", "batch"):
        each = [_solve_work(c) for c in ([case] if case["kind"] == "solve" else _instances(case))]
        return {"bytes": sum(b for b, _ in each), "flops": sum(f for _, f in each)}
    n = case["cols"] * case["nt"]
    if case["kind"] == "learned":
        return {"bytes": 8 * n, "flops": n * 83200}
    return {"bytes": 12 * n, "flops": 3 * n * 83200}


# ---------------------------------------------------------------------------
# the same mathematics in 64 bits
# ---------------------------------------------------------------------------
def _n_coef(beta):
    return beta / (2 * C0 ** 3 * RHO0)


def _dev(a):
    return torch.as_tensor(np.asarray(a, np.float64), device="cuda")


def _grid(n, d):
    """The solver's centred wavenumber grid, spacing 2 pi / ((n - 1) d), in FFT bin order."""
    g = np.arange(n) / (n - 1) / d * 2 * np.pi
    return np.fft.ifftshift(g - g.mean())


def _edge(n, m):
    s, i = np.full(n, np.nan), np.arange(n)
    s[:m] = (m - 1 - i[:m]) / m
    s[n - m:] = (i[n - m:] - (n - m - 1)) / m
    return s


def _taper(n, c):
    s = _edge(n, max(round(n * c["band"]), 1))
    z = np.nan_to_num(s)
    v = np.clip(1 - 10 * z ** 3 + 15 * z ** 4 - 6 * z ** 5, 0, 1) if c["taper"] == "wendland" \
        else 1 - z ** 2
    return np.where(np.isnan(s), 1.0, v)


def _weights(n, c):
    return np.nan_to_num(_edge(n, max(round(n * c["band"]), 1)))


class _Exact:
    def __init__(self, c):
        self.c = c
        nx, ny, nt = self.shape = (c["nx"], c["ny"], c["nt"])
        self.nf = nt // 2 + 1
        self.kk = _dev(_grid(nx, c["dx"]) ** 2)[:, None] + _dev(_grid(ny, c["dx"]) ** 2)[None, :]
        self.N = _n_coef(c["beta"])
        self.freq = np.arange(self.nf) / (nt * c["dt"])
        if c["taper"]:
            axy = _dev(_taper(nx, c))[:, None] * _dev(_taper(ny, c))[None, :]
            self.abl = (axy, _dev(_taper(nt, c)))

    def spectral(self, u, table):
        """irfft of ifft2 of table(bin) times the transform of u, bin by bin."""
        S = torch.fft.rfft(u, dim=2)
        for f in range(self.nf):
            h = table(f)
            if h is None:
                S[:, :, f] = 0
            else:
                S[:, :, f] = torch.fft.ifft2(torch.fft.fft2(S[:, :, f]) * h)
        return torch.fft.irfft(S, n=self.shape[2], dim=2)

    def diffract(self, dz, scale):
        c, (nx, ny, nt) = self.c, self.shape
        kt = np.arange(nt) / (nt - 1) / c["dt"] * 2 * np.pi / C0
        kt = kt - kt.mean()
        kmax, lam = np.pi / c["dx"], C0 / np.mean(np.abs(kt[kt != 0]))
        if c["adaptive"]:
            top = min(kmax * (1 - 0.05 * (1 + 0.7 * (dz / lam) * 5)), kmax * 0.95)
            low = 0.8 * top
        else:
            top = kmax * 0.95
            low = 0.9 * top
        kr = torch.sqrt(self.kk)
        mask = torch.where(kr > low, 0.5 * (1 + torch.cos(np.pi * (kr - low) / (top - low))), 1.0)
        mask = torch.where(kr > top, 0.0, mask)

        def table(f):
            if f == 0 or 2 * f == nt:
                return None
            k = kt[f + nt // 2]
            d = k * k - self.kk
            q = torch.sqrt(d.abs())
            ph = torch.where(d > 0, k - q, torch.full_like(q, k)) * (dz * scale)
            mag = mask * torch.where(d > 0, torch.ones_like(q), torch.exp(-q * dz * scale))
            return torch.polar(mag, ph)
        return table

    def attenuate(self, dz, scale):
        c, nt = self.c, self.shape[2]
        f = self.freq
        if c["alpha0"] < 0:
            conv = 2.17e-3 / 1e12 * 1e2 / (20 * np.log10(np.e))
            al = conv * f ** 2
            s0 = conv / (2 * np.pi) ** 2 * np.tan(np.pi) * 2 * np.pi * (f - c["f0"])
        else:
            conv = c["alpha0"] / 1e6 * 1e2 / (20 * np.log10(np.e))
            al = conv * f
            fs = np.where(f == 0, f[1] / 2, f)
            s0 = -2 * conv / (2 * np.pi) / np.pi * (np.log(2 * np.pi * fs)
                                                     - np.log(2 * np.pi * c["f0"]))
        st = 2 * np.pi * s0 * f

        def table(i):
            if i == 0:
                return torch.ones_like(self.kk)
            km = 2 * np.pi * f[i] / C0
            d = km * km - self.kk
            kz = torch.clamp(torch.sqrt(torch.clamp(d, min=0.0)), min=km * 1e-6)
            o = torch.where(d > 0, km / kz, torch.zeros_like(kz)) * (dz * scale)
            h = torch.polar(torch.exp(-al[i] * o), -st[i] * o)
            if c["alpha0"] < 0:
                h = torch.where(h.real < 0, torch.zeros_like(h), h)
            return h
        return table

    def edges(self, S, f):
        """Frequency-weighted damping and Engquist-Majda edges of one bin."""
        c, nt = self.c, self.shape[2]
        real = f == 0 or 2 * f == nt
        if c["fw"]:
            fr = self.freq
            e = float(np.clip(c["f0"] / max(fr[f], fr[1]), 0.1, 10.0))
            S = S * self.abl_fw ** e
            S = S.real + 0j if real else S
        if c["sa"]:
            co = 0j if f == 0 else -1j * C0 / (2 * np.pi * self.freq[f])
            S = S.real + 0j if real else S
            for ax in (0, 1):
                S = S if ax == 0 else S.transpose(0, 1)
                n, w = S.shape[0], self.sa_w[ax]
                G = torch.empty_like(S)
                G[1:-1] = (S[2:] - S[:-2]) / (2 * c["dx"])
                G[0], G[-1] = (S[1] - S[0]) / c["dx"], (S[-1] - S[-2]) / c["dx"]
                sg = torch.where(torch.arange(n, device="cuda") < n // 2, 1.0, -1.0)[:, None]
                S = S - c["sa_strength"] * w[:, None] * 0.5 * (S + sg * co * G)
                S = S if ax == 0 else S.transpose(0, 1)
            S = S.real + 0j if real else S
        return S

    def per_bin(self, u, fn):
        S = torch.fft.rfft(u, dim=2)
        for f in range(self.nf):
            S[:, :, f] = fn(S[:, :, f].clone(), f)
        return torch.fft.irfft(S, n=self.shape[2], dim=2)

    def obliquity(self, u):
        S, num, den = torch.fft.rfft(u, dim=2), 0.0, 0.0
        for f in range(1, self.nf):
            km = 2 * np.pi * self.freq[f] / C0
            d = km * km - self.kk
            kz = torch.clamp(torch.sqrt(torch.clamp(d, min=0.0)), min=km * 1e-6)
            P = torch.where(d > 0, torch.fft.fft2(S[:, :, f]).abs() ** 2, 0.0)
            num, den = num + (P * km / kz).sum(), den + P.sum()
        return float(num / (den + 1e-30))

    def burgers(self, u, dz, N, cfl=0.0):
        c = self.c
        out = torch.empty_like(u)
        for i in range(0, u.shape[0], 32):
            s = slice(i, i + 32)
            if c["split"] and c["flux"] == "kt":
                out[s] = _kt(u[s], N, dz, c["dt"], cfl)
            elif c["split"] and c["tvd"]:
                bt = max(1.0, 2.0 - 0.7 * (dz / (C0 / c["f0"])) * 10)
                out[s] = _rusanov_tvd(u[s], N * dz / c["dt"], bt)
            else:
                out[s] = _rusanov(u[s], N * dz / c["dt"])
        return out

    def taper(self, u, half):
        if not self.c["taper"]:
            return u
        axy, at = self.abl
        if half:
            axy, at = axy.sqrt(), at.sqrt()
        return u * axy[:, :, None] * at

    def march(self, u0, screens, sources, cfl=0.0):
        c, (nx, ny, nt) = self.c, self.shape
        u = torch.as_tensor(u0, device="cuda").double()
        if c["fw"]:
            self.abl_fw = self.abl[0]
        if c["sa"]:
            self.sa_w = [_dev(_weights(nx, c)), _dev(_weights(ny, c))]
        zs, acc, pax = [], [], []
        before = (u ** 2).sum(2)
        made = None
        while math.fsum(zs) < c["prop"] - 1e-15:
            z = math.fsum(zs)
            dz = min(c["dz"], c["prop"] - z)
            if made is None or abs(made[0] - dz) > 1e-15:
                sc = 0.5 if c["split"] else 1.0
                # the k-space filter is sized from the full step
                made = (dz, self.diffract(dz, sc), self.attenuate(dz, sc))
            P, A = made[1:]
            if c["split"]:
                u = self.spectral(u, A)
            u = self.taper(self.spectral(u, P), c["split"])
            N = self.N * self.obliquity(u) if c["obl"] else self.N
            u = self.burgers(u, dz, N, cfl)
            if c["split"]:
                u = self.taper(self.spectral(u, P), True)
            u = self.spectral(u, A)
            if c["fw"] or c["sa"]:
                u = self.per_bin(u, self.edges)
            f0b = max(c["f0"] * nt * c["dt"], 1.0)
            for scr in screens or []:
                if z < scr[0] <= z + dz:
                    ph = _dev(scr[1])
                    am = torch.clamp(_dev(scr[2]), 1e-6, 1.0) if len(scr) > 2 else None

                    def screen(S, f):
                        m = torch.ones_like(ph) if am is None else am ** (f / f0b)
                        return S * torch.polar(m, -ph * (f / f0b))
                    u = self.per_bin(u, screen)
            for sz, pl in sources or []:
                if z < sz <= z + dz:
                    cols = torch.as_tensor(pl.cols, device="cuda").long()
                    u.reshape(nx * ny, nt)[cols] += _dev(pl.values)
            after = (u ** 2).sum(2)
            acc.append([v.cpu() for v in (u.amin(2), u.amax(2), after,
                                          torch.clamp(before - after, min=0.0))])
            pax.append(u[nx // 2, ny // 2].cpu())
            before = after
            zs.append(dz)
        pnp, ppp, pI, loss = (torch.stack([a[k] for a in acc], 2).numpy() for k in range(4))
        return u.cpu().numpy(), pnp, ppp, pI, loss, np.cumsum(zs), torch.stack(pax, 1).numpy()


def _rusanov(u, k):
    a, b = u[..., :-1], u[..., 1:]
    h = -(a * a + b * b) / 2 - torch.maximum(a.abs(), b.abs()) * (b - a)
    out = u.clone()
    out[..., 1:-1] -= k * (h[..., 1:] - h[..., :-1])
    return out


def _rusanov_tvd(u, k, bt):
    a, b = u[..., :-1], u[..., 1:]
    h = 0.5 * (-0.5 * (a * a + b * b)) - 0.5 * torch.maximum(a.abs(), b.abs()) * (b - a)
    dm, dp = (b - a)[..., :-1], (b - a)[..., 1:]
    eps = 1e-30

    def lim(r):
        return torch.clamp(torch.minimum(torch.clamp(bt * r, max=1.0), torch.clamp(r, max=bt)),
                           min=0.0)
    phi = 0.5 * (lim(dp / (dm + eps * torch.sign(dm + eps)))
                 + lim(dm / (dp + eps * torch.sign(dp + eps))))
    out = u.clone()
    out[..., 1:-1] -= k * phi * (h[..., 1:] - h[..., :-1])
    return out


def _kt_rhs(u, k):
    dm, dp = u[..., 1:-1] - u[..., :-2], u[..., 2:] - u[..., 1:-1]
    m = torch.minimum(torch.minimum(2 * dm.abs(), 0.5 * (dm + dp).abs()), 2 * dp.abs())
    s = F.pad(torch.where(dm * dp > 0, torch.sign(dm) * m, torch.zeros_like(m)), (1, 1))
    um, up = u[..., :-1] + 0.5 * s[..., :-1], u[..., 1:] - 0.5 * s[..., 1:]
    ap = torch.clamp(torch.maximum(-um, -up), min=0.0)
    am = torch.clamp(torch.minimum(-um, -up), max=0.0)
    den = ap - am
    ok = den >= 1e-14
    h = (ap * (-0.5 * um * um) - am * (-0.5 * up * up) - ap * am * (up - um)) / \
        torch.where(ok, den, 1.0)
    h = torch.where(ok, h, torch.zeros_like(h))
    return F.pad(-k * (h[..., 1:] - h[..., :-1]), (1, 1))


def _kt_once(u, k):
    s = u + _kt_rhs(u, k)
    return 0.5 * u + 0.5 * (s + _kt_rhs(s, k))


def _kt(u, N, dz, dt, cfl):
    """KT with each column sub-cycled at the CFL target (0: one step)."""
    if cfl <= 0:
        return _kt_once(u, N * dz / dt)
    v = u.reshape(-1, u.shape[-1])
    peak = v.abs().amax(1)
    n = torch.clamp(torch.ceil(N / dt * peak * dz / cfl), min=1).long()
    out = torch.empty_like(v)
    for k in torch.unique(n).tolist():
        at = torch.nonzero(n == k).reshape(-1)
        w = v[at]
        for _ in range(k):
            w = _kt_once(w, N * dz / k / dt)
        out[at] = w
    return out.reshape(u.shape)


def _layers(theta):
    out, o = [], 0
    for shp in [(64, 1, 5), (64,), (64, 64, 5), (64,), (64, 64, 5), (64,), (1, 64, 5), (1,)]:
        n = int(np.prod(shp))
        out.append(_dev(theta[o:o + n]).reshape(shp).requires_grad_(True))
        o += n
    return out


def _net(x, w):
    h = x[:, None, :]
    for k in range(4):
        h = F.conv1d(h, w[2 * k], w[2 * k + 1], padding=2)
        h = F.gelu(h, approximate="tanh") if k < 3 else h
    return h[:, 0, :]


def exact(case, seed):
    rng = _rng(seed)
    if case["kind"] == "solve":
        u = _field(case, rng)
        screens = _screens(case, rng) if case["screens"] else None
        sources = _bowl(case, rng) if case["bowl"] else None
        return _Exact(case).march(u, screens, sources)
    if case["kind"] == "batch":
        inst = _instances(case)
        return [_Exact(i).march(_field(i, rng), None, None, case["cfl"]) for i in inst]
    if case["kind"] == "learned":
        w = _layers(_theta(rng))
        u = _columns(case["cols"], case["nt"], rng).double()
        L, N = LEARN, _n_coef(LEARN["beta"])
        k = N / L["dt"] * L["dz"]
        s = u.abs().amax(1)
        n = torch.clamp(torch.ceil(k * s / L["cfl"]), min=1)
        pick = (n >= L["min_sub"]) & ((u[:, 1:] - u[:, :-1]).abs().amax(1) <= L["shock"] * s) & \
            (k * s <= 0.5)
        out = _kt(u, N, L["dz"], L["dt"], L["cfl"])
        at = torch.nonzero(pick).reshape(-1)
        with torch.no_grad():
            for i in at.split(1024):
                coarse = _kt_once(u[i], k)
                y = _net(coarse * (k / 0.3), w) * (s[i] * 0.5 * (k * s[i]) ** 3)[:, None]
                y[:, 0] = 0
                y[:, -1] = 0
                out[i] = coarse + y
        return out, int(at.numel())
    w = _layers(_theta(rng))
    x, y, m = (v.double() for v in _training(case, rng))
    total, n = 0.0, m.sum()
    for i in range(0, x.shape[0], 128):
        j = slice(i, i + 128)
        part = (((_net(x[j], w) - y[j]) ** 2) * m[j]).sum() / n
        part.backward()
        total += float(part.detach())
    return total, torch.cat([v.grad.reshape(-1) for v in w])
