"""Timed cases of the constant-stratification step: what a user of the package has it do.

A case names an operation, a grid, a precision and its options; prepare() builds
the kernel handle and a seeded state as a model run has them in hand, run() makes
one pass through the package's public interface, and exact() restates the operation
in plain torch FP64 (dense vertical matrices, torch.fft in x and y).

States: Gaussian amplitudes with uniform random phases, velocity amplitude
(Kh^2 + m^2)^(-3/4), 0.1 m/s rms, on 3.125 km x 3.125 km cells over 4000 m depth
(the benchmark's family of grids); steps of half the fastest wave period's limit.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "wave-vortex-model_gb300"))
import wvgpu as wv  # noqa: E402

PI = math.pi
URMS = 0.1
T0, T = 0.0, 43200.0  # reference time and model time of the pass
GM = 9.81             # gravity of the modal normalization


def _case(op, grid, precision="fp64", hydrostatic=False, damping=False, steps=1, **more):
    Nx, Ny, Nz = grid
    return dict(op=op, Nx=Nx, Ny=Ny, Nz=Nz, precision=precision, hydrostatic=hydrostatic, damping=damping, steps=steps,
                **more)


def listed():
    return [
        # the smallest call: one right-hand side on a unit-test sized box, all latency and launches
        dict(_case("flux", (16, 16, 9)), name="flux_16x16x9"),
        # a short integration on a laptop-sized grid, state resident on the GPU
        dict(_case("rk4", (64, 64, 33), steps=4), name="rk4_64x64x33"),
        # the headline workload: one step of the FP64 drop-in
        dict(_case("rk4", (256, 256, 129)), name="rk4_256x256x129"),
        # the gateway's way in: host arrays in, host arrays out, every call
        dict(_case("rk4_host", (128, 128, 65), steps=2), name="rk4_host_128x128x65"),
        # a scheduled right-hand side as a hydrostatic model with adaptive damping evaluates it, ragged grid
        dict(_case("rhs", (60, 50, 31), hydrostatic=True, damping=True), name="rhs_damped_hydro_60x50x31"),
        # diagnostics and output: the physical fields of a state
        dict(_case("inverse", (192, 192, 97)), name="inverse_192x192x97"),
        # initialisation from physical fields, hydrostatic transform
        dict(_case("forward", (256, 256, 65), hydrostatic=True), name="forward_hydro_256x256x65"),
        # the backward direction: one flux VJP of a gradient computation
        dict(_case("vjp", (128, 128, 65)), name="vjp_128x128x65"),
        # a passive tracer's tendency in given velocity fields
        dict(_case("scalar", (96, 64, 33)), name="scalar_96x64x33"),
        # the paired-FP32 form of the headline step
        dict(_case("rk4", (256, 256, 129), precision="fp32x2"), name="rk4_fp32x2_256x256x129"),
        # the mixed form of the headline step
        dict(_case("rk4", (256, 256, 129), precision="mixed"), name="rk4_mixed_256x256x129"),
        # an ensemble of small uneven grids stepped in one graph launch
        dict(_case("ensemble", (48, 48, 25), steps=4, members=4, Nx2=64, Nz2=33), name="ensemble_48_64"),
    ]


def draw(rng):
    def size(lo, hi):
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        kind = rng.random()
        if kind < 0.35:  # powers of two and three times them, as models are usually run
            return min((16, 24, 32, 48, 64, 96, 128, 192), key=lambda v: abs(math.log(v / n)))
        return n if kind < 0.6 else 2 * max(1, n // 2)

    op = rng.choice(["flux", "rhs", "rk4", "rk4_host", "inverse", "forward", "vjp", "adjoint", "scalar", "ensemble"])
    small = op in ("adjoint", "ensemble", "scalar")
    Nx, Ny = size(12, 96 if small else 192), size(12, 96 if small else 192)
    Nz = int(round(math.exp(rng.uniform(math.log(7), math.log(49 if small else 97)))))
    if rng.random() < 0.4:
        Nz = min((9, 17, 25, 33, 49, 65, 97), key=lambda v: abs(math.log(v / Nz)))
    precision = rng.choice(["fp64", "fp64", "fp32x2"])
    case = _case(op, (Nx, Ny, Nz), precision, hydrostatic=rng.random() < 0.3,
                 damping=op in ("rhs", "rk4") and rng.random() < 0.5,
                 steps=rng.choice([1, 2, 3]) if op in ("rk4", "rk4_host", "adjoint", "ensemble") else 1)
    if op == "ensemble":
        case.update(members=rng.choice([1, 2, 5]), Nx2=size(16, 64), Nz2=rng.choice([9, 13, 17, 33]))
    return case


# ---- grid, modes and coefficients (plain numpy) -----------------------------------


def _grids(case):
    first = (case["Nx"], case["Ny"], case["Nz"])
    return [first, (case["Nx2"], case["Nx2"], case["Nz2"])] if case["op"] == "ensemble" else [first]


def _configuration(case, grid):
    Nx, Ny, Nz = grid
    return wv.Configuration(Nx=Nx, Ny=Ny, Nz=Nz, Nj=max(1, 2 * (Nz - 1) // 3), Lx=3125.0 * Nx, Ly=3125.0 * Ny, Lz=4000.0,
                            isHydrostatic=case["hydrostatic"])


class _Modes:
    """Retained (k, l) modes in canonical order and the half-spectrum rows they live in."""

    def __init__(self, c):
        self.c = c
        Nx, Ny = c.Nx, c.Ny
        dft = lambda n: np.array(list(range((n + 1) // 2)) + [-v for v in range(n // 2, 0, -1)])  # noqa: E731
        L, K = (a.ravel() for a in np.meshgrid(dft(Ny), dft(Nx), indexing="ij"))
        nyx = (K == -(Nx // 2)) if Nx % 2 == 0 else np.zeros(K.shape, bool)
        nyy = (L == -(Ny // 2)) if Ny % 2 == 0 else np.zeros(L.shape, bool)
        primary = (L > 0) | (((L == 0) | nyy) & ((K > 0) | (K == 0) | nyx))
        k, l = 2.0 * PI * (K / c.Lx), 2.0 * PI * (L / c.Ly)
        Kh = np.sqrt(k * k + l * l)
        keep = primary & ~nyx & ~nyy & (Kh <= 2.0 * (2.0 * PI * (Nx // 2 / c.Lx)) / 3.0)
        at = np.flatnonzero(keep)
        at = at[np.lexsort((L[at], K[at], Kh[at]))]
        self.K, self.L, self.k, self.l, self.Kh = K[at], L[at], k[at], l[at], Kh[at]
        self.half = Nx // 2 + 1
        self.conj = self.K < 0
        kk, ll = np.where(self.conj, -self.K, self.K), np.where(self.conj, -self.L, self.L)
        self.row = kk + self.half * (ll % Ny)
        have = np.zeros(Ny * self.half, bool)
        have[self.row] = True
        self.comp = [(self.half * i, self.half * (-i % Ny)) for i in range(Ny)
                     if not have[self.half * i] and have[self.half * (-i % Ny)]]
        self.real = [self.half * i for i in range(Ny) if (i == 0 or 2 * i == Ny) and have[self.half * i]]
        self.m = np.arange(c.Nj) * PI / c.Lz


def _coefficients(g):
    """Field factors and projection factors per (mode, j), arrays (Nkl, Nj)."""
    c = g.c
    f = 2.0 * c.rotationRate * math.sin(c.latitude * PI / 180.0)
    f2, N2 = f * f, c.N0 ** 2
    j = np.arange(c.Nj)
    sign = np.where(j % 2 == 0, 1.0, -1.0)
    m = g.m
    with np.errstate(divide="ignore", invalid="ignore"):
        h0 = np.where(j == 0, c.Lz, N2 / (c.g * m * m))
        Fg = np.where(j == 0, 2.0, sign * h0 * m * math.sqrt(2.0 * GM / (c.Lz * N2)))
        Gg = np.where(j == 0, 1.0, sign * math.sqrt(2.0 * GM / (c.Lz * N2)))
        Kh = g.Kh[:, None]
        K2 = Kh * Kh
        nonhydro = sign * math.sqrt(2.0 * GM / (c.Lz * (N2 - f2)))
        if c.isHydrostatic:
            h = np.broadcast_to(np.where(j == 0, 1.0, N2 / (c.g * m * m)), (len(g.Kh), c.Nj))
            Fw, Gw = np.broadcast_to(Fg, h.shape), Gg
        else:
            h = np.where(j == 0, 1.0, (N2 - f2) / (c.g * (m * m + K2)))
            Fw, Gw = np.where(j == 0, 2.0, nonhydro * h * m), np.where(j == 0, 1.0, nonhydro)
        w = np.sqrt(c.g * h * K2 + f2)
        cosA, sinA = (np.where(Kh > 0, v[:, None] / Kh, 0.0) for v in (g.k, g.l))
        wave, inert, geo, mda = (Kh > 0) & (j > 0), (Kh == 0) & (j >= 0), (Kh > 0) & (j >= 0), (Kh == 0) & (j > 0)
        a = dict(omega=w, U=np.where(wave, cosA - 1j * (f / w) * sinA, np.where(inert, 1.0, 0.0)) * Fw,
                 V=np.where(wave, sinA + 1j * (f / w) * cosA, np.where(inert, 1j, 0.0)) * Fw,
                 W=np.where(wave, -1j * Kh * h, 0.0) * Gw, N=np.where(wave, -Kh * h / w, 0.0) * Gw)
        lr = np.where(j == 0, 0.0, f2 / (c.g * h0))
        den = K2 + lr
        a["U0"] = np.where(geo, 1j * g.l[:, None] / den * Fg, 0.0)
        a["V0"] = np.where(geo, -1j * g.k[:, None] / den * Fg, 0.0)
        a["N0"] = np.where(geo & (j > 0), -(f / c.g) / den * Gg, np.where(mda, Gg, 0.0))
        a["vort"] = np.where(geo, 1.0 / Fg, np.where(mda, f2 / (2.0 * h0) / Fg, 0.0))
        a["buoy"] = np.where(geo & (j > 0), (-f / h0) / Gg, np.where(mda, 1.0 / Gg, 0.0))
        a["ApmN"] = np.where(wave, -w / (2.0 * Kh * h) / Gw, 0.0)
        if c.isHydrostatic:
            a["div"] = np.where(wave, -1j / (2.0 * Kh * h) * h0 / Fg * Gg / Gw, 0.0)
            a["Cu"], a["Cv"], a["Cw"] = a["div"] * 1j * g.k[:, None], a["div"] * 1j * g.l[:, None], 0.0 * a["div"]
        else:
            pre = sign * math.sqrt(c.g * c.Lz / (2.0 * (N2 - f2)))
            a["Cu"], a["Cv"], a["Cw"] = cosA * (m / 2.0) * pre, sinA * (m / 2.0) * pre, 1j * (Kh / 2.0) * pre
        a["inert"] = 0.5 / Fw[0]
    return a, f


def _damping(g, f):
    c = g.c
    top = max(np.max(np.abs(g.k)), np.max(np.abs(g.l)))
    res, lowest = PI / top, min(2.0 * PI / c.Lx, 2.0 * PI / c.Ly)

    def ramp(v, cut, most):
        with np.errstate(divide="ignore", over="ignore"):
            mid = np.exp(-((v - most) / (v - cut)) ** 2)
        return np.where(v < cut, 0.0, np.where(v > most, 1.0, mid))

    h0 = np.where(g.m == 0, c.Lz, c.N0 ** 2 / (c.g * np.maximum(g.m, 1e-300) ** 2))
    pxy = res / PI ** 2
    pz = PI ** 2 * (c.g * h0[-1] / f ** 2) / res ** 2 * pxy
    qk = ramp(g.Kh, lowest * (top / lowest) ** 0.75, top)
    jmax = c.Nj - 1.0
    qj = ramp(np.arange(c.Nj) * 1.0, jmax ** 0.75, jmax) if c.Nj > 2 else np.ones(c.Nj)
    lr = np.where(g.m == 0, 0.0, f ** 2 / (c.g * h0))
    return -pxy * (qk * g.Kh ** 2)[:, None] - pz * (qj * lr)[None, :]


def _state(g, a, rng):
    """(Ap, Am, A0) of a random flow at URMS."""
    K2 = g.Kh[:, None] ** 2 + g.m[None, :] ** 2
    env = np.where(K2 > 0, np.maximum(K2, 1e-300) ** -0.75, 0.0)
    parts = []
    for factor in (a["U"], a["U"], a["U0"]):
        size = np.sqrt(np.abs(factor) ** 2 + np.abs(a["V"] if factor is a["U"] else a["V0"]) ** 2)
        z = rng.standard_normal(K2.shape) * np.exp(2j * PI * rng.random(K2.shape)) * env
        parts.append((z, np.divide(1.0, size, out=np.zeros_like(size), where=size > 0)))
    scale = URMS / math.sqrt(sum(float(np.sum(np.abs(z[s > 0]) ** 2)) for z, s in parts))
    Ap, Am, A0 = (scale * z * s for z, s in parts)
    still = g.Kh == 0  # inertial oscillations are one real vector rotating; no mean buoyancy mode
    Am[still] = np.conj(Ap[still])
    return [np.ascontiguousarray(v, dtype=np.complex128) for v in (Ap, Am, A0)]


def _inputs(case, seed):
    """Per grid: geometry, factors and the seeded host arrays of the pass."""
    rng = np.random.Generator(np.random.PCG64(seed))
    out = []
    for grid in _grids(case):
        c = _configuration(case, grid)
        g = _Modes(c)
        a, f = _coefficients(g)
        members = [_state(g, a, rng) for _ in range(case.get("members", 1))]
        i = dict(g=g, a=a, f=f, members=members, dt=min(0.45 * 3125.0, PI / float(np.max(a["omega"]))))
        shape = (grid[2], grid[1], grid[0])
        if case["op"] in ("vjp", "adjoint"):
            i["bars"] = [v / URMS for v in _state(g, a, rng)]
        if case["op"] in ("forward", "scalar"):
            i["fields"] = _smooth(rng, 4 if case["op"] == "scalar" else 3 if case["hydrostatic"] else 4, shape)
        out.append(i)
    return out


def _smooth(rng, channels, shape):
    """Multi-scale physical fields: noise times a k^-2 horizontal filter plus a vertical profile."""
    Nz, Ny, Nx = shape
    noise = torch.from_numpy(rng.standard_normal((channels, Nz, Ny, Nx), dtype=np.float32)).cuda().double()
    ky = torch.fft.fftfreq(Ny, 1.0 / Ny, device="cuda", dtype=torch.float64)[:, None]
    kx = torch.arange(Nx // 2 + 1, device="cuda", dtype=torch.float64)[None, :]
    out = torch.fft.irfft2(torch.fft.rfft2(noise) / (1.0 + kx * kx + ky * ky), s=(Ny, Nx))
    out = out / out.std()
    z = torch.linspace(-1.0, 0.0, Nz, device="cuda", dtype=torch.float64)[None, :, None, None]
    amplitude = torch.tensor([URMS, URMS, 1e-3, 5.0], device="cuda", dtype=torch.float64)[:channels, None, None, None]
    return (amplitude * out * (1.0 + torch.cos(PI * z))).cpu().numpy()


# ---- the passes ----------------------------------------------------------------------


def prepare(case, seed):
    case = dict(case)
    ins = _inputs(case, seed)
    s = dict(case=case, op=case["op"])
    dev = lambda v: torch.from_numpy(np.ascontiguousarray(v)).cuda()  # noqa: E731
    if case["op"] == "ensemble":
        s["handle"] = wv.WVEnsemble([i["g"].c for i in ins], [len(i["members"]) for i in ins], precision=case["precision"],
                                    autotune=False)
        s["start"] = [dev(np.stack([np.stack(m) for m in i["members"]])) for i in ins]
        s["work"] = [torch.empty_like(v) for v in s["start"]]
        s["dt"] = [i["dt"] for i in ins]
        return s
    i = ins[0]
    s["handle"] = k = wv.WVTransformConstantStratificationKernel(i["g"].c, precision=case["precision"])
    if case["damping"]:
        k.set_forcing(nonlinear=True, adaptive_damping=True)
    s["dt"] = i["dt"]
    s["A"] = i["members"][0] if case["op"] == "rk4_host" else [dev(v) for v in i["members"][0]]
    if case["op"] == "rk4":
        s["work"] = [torch.empty_like(v) for v in s["A"]]
    if "bars" in i:
        s["bars"] = [dev(v) for v in i["bars"]]
    if "fields" in i:
        s["fields"] = dev(i["fields"])
    return s


def run(state):
    s, op, k = state, state["op"], state["handle"]
    steps = s["case"]["steps"]
    if op == "flux":
        return k.nonlinearFlux(T, T0, *s["A"])
    if op == "rhs":
        return k.evaluateRightHandSide(T, T0, *s["A"])
    if op == "rk4":  # in place on the model's state; every pass from the same one
        for w, v in zip(s["work"], s["A"]):
            w.copy_(v)
        k.rk4(*s["work"], T, T0, s["dt"], steps)
        return s["work"]
    if op == "rk4_host":
        return k.rk4(*s["A"], T, T0, s["dt"], steps)[:3]
    if op == "inverse":
        return k.transformWaveVortexToUVWEta(T, T0, *s["A"])
    if op == "forward":
        f = k.transformUVEtaToWaveVortex if s["case"]["hydrostatic"] else k.transformUVWEtaToWaveVortex
        return f(s["fields"], T, T0)
    if op == "vjp":
        return k.flux_vjp(T, T0, *s["A"], *s["bars"])
    if op == "adjoint":
        return k.rk4_adjoint(*s["A"], T, T0, s["dt"], steps, 2, *s["bars"])
    if op == "scalar":
        return k.advectFGridScalar(s["fields"][3], s["fields"][:3], True)
    for w, v in zip(s["work"], s["start"]):
        w.copy_(v)
    k.rk4(s["work"], T, T0, s["dt"], steps)
    return s["work"]


def work(case):
    """Inputs read and outputs written once; FFT operations counted as 2.5 n log2 n per
    real row pair of transforms and 5 n log2 n per complex vertical line."""
    bytes_, flops = 0.0, 0.0
    for Nx, Ny, Nz in _grids(case):
        g = _Modes(_configuration(case, (Nx, Ny, Nz)))
        M, R = len(g.Kh) * g.c.Nj, Nx * Ny * Nz
        nt = 3 if case["hydrostatic"] else 4
        plane = 2.5 * R * math.log2(Nx * Ny)
        line = 2.5 * len(g.Kh) * 2 * (Nz - 1) * math.log2(2 * (Nz - 1))
        flux = (3 + 4 * nt) * plane + (4 + 2 * nt) * line + 6 * nt * R + 150 * M
        op, n = case["op"], case["steps"] * case.get("members", 1)
        if op in ("flux", "rhs"):
            b, f = 96.0 * M, flux
        elif op in ("rk4", "rk4_host", "ensemble"):
            b, f = 96.0 * M * case.get("members", 1), 4 * n * flux
        elif op == "inverse":
            b, f = 48.0 * M + 32.0 * R, 4 * plane + 4 * line + 60 * M
        elif op == "forward":
            b, f = 48.0 * M + 8.0 * nt * R, nt * plane + nt * line + 60 * M
        elif op == "vjp":
            b, f = 144.0 * M, 2.6 * flux
        elif op == "adjoint":
            b, f = 144.0 * M, 4 * n * 3.6 * flux
        else:
            b, f = 40.0 * R, 5 * plane + 8 * R + 2 * 2.0 * Nz * R
        bytes_ += b
        flops += f
    return {"bytes": bytes_, "flops": flops}


# ---- the same operations in plain torch FP64 --------------------------------------------


class _Exact:
    def __init__(self, i):
        g, a = i["g"], i["a"]
        c = g.c
        self.c, self.g = c, g
        t = lambda v: torch.from_numpy(np.ascontiguousarray(v)).cuda()  # noqa: E731
        self.a = {n: t(v) for n, v in a.items()}
        self.row, self.conj, self.real = t(g.row), t(g.conj)[:, None], t(np.array(g.real, dtype=np.int64))
        self.to, self.src = (t(np.array([p[q] for p in g.comp], dtype=np.int64)) for q in (0, 1))
        self.m, self.k, self.l = t(g.m), t(g.k)[:, None], t(g.l)[:, None]
        L = c.Nz - 1
        jn = (np.arange(c.Nj)[:, None] * np.arange(c.Nz)[None, :]) % (2 * L)
        cos, sin = np.cos(PI * jn / L), np.sin(PI * jn / L)
        sin[jn % L == 0] = 0.0
        ends = np.where((np.arange(c.Nz) % L) == 0, 1.0, 2.0) / L
        self.cos = t(np.where(np.arange(c.Nj)[:, None] == 0, 0.5, cos))
        self.sin = t(sin)
        self.fcos, self.fsin = t((cos * ends).T), t((2.0 / L * sin).T)
        self.kx = 2.0 * PI / c.Lx * torch.arange(g.half, device="cuda", dtype=torch.float64)
        ly = np.arange(c.Ny)
        self.ly = t(2.0 * PI / c.Ly * np.where(2 * ly <= c.Ny, ly, ly - c.Ny))[:, None]
        self.damp = t(_damping(g, i["f"]))
        self.hs = 1.0 / (c.Nx * c.Ny)
        self.targets = (0, 1, 3) if c.isHydrostatic else (0, 1, 2, 3)

    def _columns(self, spec, matrix):
        return torch.complex(spec.real @ matrix, spec.imag @ matrix)

    def _half(self, cols):
        """Retained columns (Nkl, Nz) -> half spectrum (Nz, Ny, NxHalf)."""
        c = self.c
        h = torch.zeros((c.Ny * self.g.half, c.Nz), dtype=torch.complex128, device="cuda")
        h = h.index_copy(0, self.row, torch.where(self.conj, cols.conj().resolve_conj(), cols))
        if len(self.to):
            h = h.index_copy(0, self.to, h[self.src].conj().resolve_conj())
        if len(self.real):
            r = h[self.real].real
            h = h.index_copy(0, self.real, torch.complex(r, torch.zeros_like(r)))
        return h.reshape(c.Ny, self.g.half, c.Nz).permute(2, 0, 1)

    def _space(self, half):
        return torch.fft.irfft2(half, s=(self.c.Ny, self.c.Nx), norm="forward")

    def _modes(self, field, matrix):
        h = torch.fft.rfft2(field).permute(1, 2, 0).reshape(-1, self.c.Nz)[self.row]
        return self.hs * self._columns(torch.where(self.conj, h.conj().resolve_conj(), h), matrix)

    def _phase(self, t):
        w = self.a["omega"] * (t - T0)
        return torch.complex(torch.cos(w), torch.sin(w))

    def spectra(self, A, t):
        a, p = self.a, self._phase(t)
        ap, am, a0 = A[0] * p, A[1] * p.conj(), A[2]
        return (a["U"] * ap + a["U"].conj() * am + a["U0"] * a0, a["V"] * ap + a["V"].conj() * am + a["V0"] * a0,
                a["W"] * (ap + am), a["N"] * (ap - am) + a["N0"] * a0)

    def fields(self, A, t):
        return [self._space(self._half(self._columns(f, self.cos if q < 2 else self.sin)))
                for q, f in enumerate(self.spectra(A, t))]

    def project(self, U, V, W, N, t):
        a, p = self.a, self._phase(t)
        a0 = 1j * (self.k * V - self.l * U) * a["vort"] + N * a["buoy"]
        b = (N - a["N0"] * a0) * a["ApmN"]
        wave = a["Cu"] * U + a["Cv"] * V + a["Cw"] * W
        still = torch.from_numpy(self.g.Kh == 0).cuda()[:, None]
        inert = (U - 1j * V) * a["inert"]
        cp = torch.where(still, inert, wave + b)
        cm = torch.where(still, inert.conj().resolve_conj(), wave - b)
        return cp * p.conj(), cm * p, a0

    def flux(self, A, t, damping=False):
        spec = self.spectra(A, t)
        half = [self._half(self._columns(f, self.cos if q < 2 else self.sin)) for q, f in enumerate(spec)]
        u, v, w = (self._space(half[q]) for q in range(3))
        S = []
        for q in range(4):
            if q not in self.targets:
                S.append(torch.zeros_like(self.a["ApmN"]) + 0j)
                continue
            fz = self._columns(-self.m * spec[q], self.sin) if q < 2 else self._columns(self.m * spec[q], self.cos)
            product = u * self._space(1j * self.kx * half[q]) + v * self._space(1j * self.ly * half[q]) + w * self._space(self._half(fz))
            S.append(self._modes(-product, self.fcos if q < 2 else self.fsin))
        F = self.project(*S, t)
        if not damping:
            return F
        speed = torch.sqrt(torch.max(u * u + v * v))
        return tuple(f + x * (speed * self.damp) for f, x in zip(F, A))

    def step(self, A, t, h, damping=False):
        add = lambda x, s, y: tuple(p + s * q for p, q in zip(x, y))  # noqa: E731
        k1 = self.flux(A, t, damping)
        k2 = self.flux(add(A, 0.5 * h, k1), t + 0.5 * h, damping)
        k3 = self.flux(add(A, 0.5 * h, k2), t + 0.5 * h, damping)
        k4 = self.flux(add(A, h, k3), t + h, damping)
        return add(add(add(add(A, h / 6, k1), h / 3, k2), h / 3, k3), h / 6, k4)

    def steps(self, A, t, h, n, damping=False):
        for _ in range(n):
            A, t = self.step(A, t, h, damping), t + h
        return list(A)

    def scalar(self, s, adv):
        c = self.c
        L = c.Nz - 1
        jn = np.arange(c.Nz)[:, None] * np.arange(c.Nz)[None, :] % (2 * L)
        ends = np.where(np.arange(c.Nz) % L == 0, 1.0, 2.0) / L
        mid = np.arange(c.Nz) % L != 0
        m = PI * np.arange(c.Nz) / c.Lz
        D = (np.sin(PI * jn / L) * mid[:, None] * mid[None, :]) @ ((-m * mid)[:, None] * np.cos(PI * jn / L) * ends[None, :])
        h = torch.fft.rfft2(s)
        kx = self.kx.clone()
        if c.Nx % 2 == 0:
            kx[-1] = 0.0
        ly = np.arange(c.Ny)
        ly = torch.from_numpy(2.0 * PI / c.Ly * np.where(2 * ly < c.Ny, ly, ly - c.Ny)).cuda()[:, None]
        hz = torch.tensordot(torch.from_numpy(D).cuda() + 0j, h, dims=1)
        back = lambda v: torch.fft.irfft2(v, s=(c.Ny, c.Nx))  # noqa: E731
        spec = [1j * kx * h, 1j * ly * h, hz]
        ky0 = self.real // self.g.half
        for v in spec:  # self-conjugate rows are real
            v[:, ky0, 0] = v[:, ky0, 0].real + 0j
        out = -(adv[0] * back(spec[0]) + adv[1] * back(spec[1]) + adv[2] * back(spec[2]))
        keep = torch.zeros(c.Ny * self.g.half, dtype=torch.bool, device="cuda")
        for rows in (self.row, self.to, self.src):
            keep[rows] = True
        return back(torch.fft.rfft2(out) * keep.reshape(c.Ny, self.g.half))


def exact(case, seed):
    op, n = case["op"], case["steps"]
    ins = _inputs(case, seed)
    dev = lambda vs: [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in vs]  # noqa: E731
    if op == "ensemble":
        out = []
        for i in ins:
            x = _Exact(i)
            out.append(torch.stack([torch.stack(x.steps(dev(m), T, i["dt"], n)) for m in i["members"]]))
        return out
    i = ins[0]
    x, A = _Exact(i), dev(i["members"][0])
    if op in ("flux", "rhs"):
        return list(x.flux(A, T, case["damping"]))
    if op in ("rk4", "rk4_host"):
        return x.steps(A, T, i["dt"], n, case["damping"])
    if op == "inverse":
        return torch.stack(x.fields(A, T))
    if op == "forward":
        f = dev([i["fields"]])[0]
        f = [f[0], f[1], None, f[2]] if case["hydrostatic"] else list(f)
        spec = [torch.zeros_like(x.a["ApmN"]) + 0j if v is None else x._modes(v, x.fcos if q < 2 else x.fsin)
                for q, v in enumerate(f)]
        return list(x.project(*spec, T))
    if op in ("vjp", "adjoint"):
        leaf = [v.requires_grad_(True) for v in A]
        out = x.flux(leaf, T) if op == "vjp" else x.steps(leaf, T, i["dt"], n)
        return list(torch.autograd.grad(sum((b.conj() * f).real.sum() for b, f in zip(dev(i["bars"]), out)), leaf))
    f = dev([i["fields"]])[0]
    return x.scalar(f[3], f[:3])
