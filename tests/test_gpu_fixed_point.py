"""FP64 transforms on 64-bit fixed-point lines against the oracle: every lane-held
length (16 to 256 points, one or three times a power of two) on each axis, lengths
that take the run-time stages (odd, prime factors, short, just past a lane length),
rows past the fixed-point x pass's 512 points, and states of extreme size or holding
NaN and infinity.  Tolerances: 1e-12, or three times the oracle's own FP64 noise
(two orderings of its vertical sums) where that is larger.  On the smallest grids the
reference is the oracle in long double: there its FP64 rounding along x and y, which
the two orderings share, is as large as the tolerance (8.4e-13 of F0 at 6x8x5)."""
import types

import numpy as np
import pytest
import scipy.fft

import wv_oracle as O
from _cases import parity_tolerance, rel_err

pytestmark = pytest.mark.gpu

# (Nx, Ny, Nz): z lines have 2 (Nz - 1) points
LANES = [(16, 24, 17), (24, 16, 13), (32, 48, 25), (48, 32, 9), (64, 96, 33), (96, 64, 49), (128, 192, 7),
         (192, 128, 8), (256, 16, 97), (16, 256, 65), (24, 20, 129)]
ANY = [(6, 8, 5), (10, 14, 12), (15, 13, 8), (22, 26, 11), (34, 17, 18), (300, 12, 9), (12, 300, 9), (516, 8, 7)]


@pytest.fixture(scope="module")
def wv():
    import torch
    import wvgpu
    from wvgpu import build
    assert torch.cuda.is_available()
    build.build()
    return wvgpu


def _setup(wv, shape, hydro=False, antialias=True, precision="fp64"):
    Nx, Ny, Nz = shape
    c = O.Config(Nx=Nx, Ny=Ny, Nz=Nz, Nj=O.default_nj(Nz), Lx=400e3, Ly=400e3 * Ny / Nx, Lz=4000.0, latitude=33.0,
                 isHydrostatic=hydro, shouldAntialias=antialias)
    cfg = wv.Configuration(Nx=Nx, Ny=Ny, Nz=Nz, Nj=c.Nj, Lx=c.Lx, Ly=c.Ly, Lz=c.Lz, N0=c.N0, rho0=c.rho0, g=c.g,
                           planetaryRadius=c.planetaryRadius, rotationRate=c.rotationRate, latitude=c.latitude,
                           isHydrostatic=hydro, shouldAntialias=antialias)
    d = O.build_descriptor(c)
    return c, d, O.random_state(d, 7, 1e-3), wv.WVTransformConstantStratificationKernel(cfg, precision=precision)


@pytest.fixture(scope="module")
def extended():
    """The oracle evaluated in long double (its coefficient tables stay FP64, as on the GPU)."""
    ld = np.longdouble
    m = types.ModuleType("wv_oracle_extended")
    m.__file__ = O.__file__
    import sys
    sys.modules[m.__name__] = m  # (dataclasses look their module up)
    with open(O.__file__) as f:
        exec(compile(f.read().replace("np.complex128", "np.clongdouble"), m.__name__, "exec"), m.__dict__)
    fft, ifft, rfft, irfft = scipy.fft.fft, scipy.fft.ifft, scipy.fft.rfft, scipy.fft.irfft
    m._rfft2 = lambda x, workers: fft(rfft(np.asarray(x, ld), axis=-1), axis=-2)
    m._irfft2 = lambda x, s, workers: irfft(ifft(x, axis=-2, norm="forward"), n=s[1], axis=-1, norm="forward")
    m._dct1 = lambda x, axis: scipy.fft.dct(np.ascontiguousarray(x, ld), type=1, axis=axis)
    m._dst1 = lambda x, axis: scipy.fft.dst(np.ascontiguousarray(x, ld), type=1, axis=axis)

    def phase(desc, t, t0):
        angle = (desc.arrays["omega"] * (t - t0)).astype(ld)
        return np.cos(angle) + 1j * np.sin(angle)

    m.phase = phase
    yield m
    del sys.modules[m.__name__]


def _close(got, ref, floors):
    for a, b, fl in zip(got, ref, floors):
        a = a.cpu().numpy() if hasattr(a, "cpu") else a
        assert rel_err(a, b) <= parity_tolerance(fl), (rel_err(a, b), fl)


@pytest.mark.parametrize("i,shape", list(enumerate(LANES + ANY)))
def test_transforms_flux_and_vjp_match_oracle(wv, extended, i, shape):
    import torch
    hydro, antialias = i % 3 == 2, i % 4 != 3
    c, d, A, k = _setup(wv, shape, hydro, antialias)
    t, t0 = 1234.5, 10.0
    ref, floors = O.noise_floor(O.nonlinear_flux, d, *A, t, t0)
    if np.prod(shape) < 2000:
        ref = [x.astype(np.complex128) for x in extended.nonlinear_flux(d, *[a.astype(np.clongdouble) for a in A], t, t0)]
    _close(k.nonlinearFlux(t, t0, *A), ref, floors)
    ref, floors = O.noise_floor(lambda *a: (O.inverse_uvweta(*a),), d, *A, t, t0)
    _close((k.transformWaveVortexToUVWEta(t, t0, *A),), ref, floors)
    rng = np.random.default_rng(5)
    R = (shape[2], shape[1], shape[0])
    f = rng.standard_normal((3 if hydro else 4,) + R)
    fwd = k.transformUVEtaToWaveVortex if hydro else k.transformUVWEtaToWaveVortex
    _close(fwd(f, t, t0), *O.noise_floor(O.forward, d, f, t, t0))
    Fb = [rng.standard_normal((d.Nkl, c.Nj)) + 1j * rng.standard_normal((d.Nkl, c.Nj)) for _ in range(3)]
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()
    _close(k.flux_vjp(t, t0, *map(dev, A), *map(dev, Fb)), *O.noise_floor(O.flux_vjp, d, *A, t, t0, *Fb))
    s, adv = rng.standard_normal(R), 0.1 * rng.standard_normal((3,) + R)
    ref, floors = O.noise_floor(lambda *a: (O.advect_fgrid_scalar(*a),), d, s, adv, antialias)
    _close((k.advectFGridScalar(dev(s), dev(adv), antialias),), ref, floors)
    k.close()


@pytest.mark.parametrize("shape", [(32, 48, 17), (20, 18, 11)])
@pytest.mark.parametrize("power", [-600, -130, 130, 600])
def test_scaled_states_give_scaled_fields(wv, shape, power):
    """The transforms are linear, and a power of two moves only the lines' exponents:
    past float range the line bounds come from exponents relative to the largest
    entry, so only roundings (three passes, each within 2^-50 of the line's bound)
    may differ: 2e-14 of the largest value."""
    import torch
    c, d, A, k = _setup(wv, shape)
    s = 2.0 ** power
    f = k.transformWaveVortexToUVWEta(300.0, 0.0, *A)
    g = k.transformWaveVortexToUVWEta(300.0, 0.0, *[s * x for x in A])
    assert np.isfinite(g).all()
    for a, b in zip(g, f):
        assert np.max(np.abs(a / s - b)) <= 2e-14 * np.max(np.abs(b))
    rng = np.random.default_rng(6)
    R = (shape[2], shape[1], shape[0])
    f = rng.standard_normal((4,) + R)
    B = k.transformUVWEtaToWaveVortex(f, 300.0, 0.0)
    S = k.transformUVWEtaToWaveVortex(s * f, 300.0, 0.0)
    for a, b in zip(S, B):
        assert np.max(np.abs(a / s - b)) <= 1e-13 * np.max(np.abs(b))
    q, adv = rng.standard_normal(R), 0.1 * rng.standard_normal((3,) + R)
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()
    one = k.advectFGridScalar(dev(q), dev(adv), False).cpu().numpy()
    big = k.advectFGridScalar(dev(s * q), dev(adv), False).cpu().numpy()
    assert np.max(np.abs(big / s - one)) <= 1e-13 * np.max(np.abs(one))
    k.close()


@pytest.mark.parametrize("shape", [(32, 48, 17), (20, 18, 11)])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_nan_and_infinity_reach_every_field_value(wv, shape, bad):
    c, d, A, k = _setup(wv, shape)
    A = [np.array(x) for x in A]
    A[0][3, 2] = bad
    f = k.transformWaveVortexToUVWEta(0.0, 0.0, *A)
    for channel in (0, 1, 3):
        assert not np.isfinite(f[channel][1:-1]).any()
    F = k.nonlinearFlux(0.0, 0.0, *A)
    assert not any(np.isfinite(x).any() for x in F[:2])
    k.close()


@pytest.mark.parametrize("shape", [(16, 24, 17), (48, 32, 13), (192, 32, 9), (30, 16, 9)])
def test_fp32x2_routes_match_oracle(wv, shape):
    """FP32X2 handles: fixed-point lines at lane lengths (the flux then meets FP64's
    tolerance), paired FP32 elsewhere and in the adjoint (1e-9 of the largest value),
    and after a choice of kernels the paired-FP32 flux."""
    import torch
    c, d, A, k = _setup(wv, shape, precision="fp32x2")
    ref, floors = O.noise_floor(O.nonlinear_flux, d, *A, 50.0, 0.0)
    if shape[0] in (16, 48):
        _close(k.nonlinearFlux(50.0, 0.0, *A), ref, floors)
    rng = np.random.default_rng(8)
    Fb = [rng.standard_normal((d.Nkl, c.Nj)) + 1j * rng.standard_normal((d.Nkl, c.Nj)) for _ in range(3)]
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()
    vjp, vfl = O.noise_floor(O.flux_vjp, d, *A, 50.0, 0.0, *Fb)
    for a, b, fl in zip(k.flux_vjp(50.0, 0.0, *map(dev, A), *map(dev, Fb)), vjp, vfl):
        assert rel_err(a.cpu().numpy(), b) <= max(1e-9, parity_tolerance(fl))
    k.set_fft_variants("register", "register")
    for a, b in zip(k.nonlinearFlux(50.0, 0.0, *A), ref):
        assert rel_err(a, b) <= 1e-9
    k.close()
