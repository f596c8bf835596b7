"""Where the fixed-point lines of FP64 handles could lose what plain doubles keep:
advecting velocities that are identically zero, values near both ends of a double's
range, phases of very small angles, and lines of several hundred points; and the memory
that their VJP takes."""
import numpy as np
import pytest

import wv_oracle as O
from test_gpu_fixed_point import extended  # noqa: F401 (a fixture)

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def wv():
    import torch
    import wvgpu
    from wvgpu import build
    assert torch.cuda.is_available()
    build.build()
    return wvgpu


def _setup(wv, shape, hydro=False):
    Nx, Ny, Nz = shape
    c = O.Config(Nx=Nx, Ny=Ny, Nz=Nz, Nj=O.default_nj(Nz), Lx=400e3, Ly=400e3 * Ny / Nx, Lz=4000.0, latitude=33.0,
                 isHydrostatic=hydro)
    cfg = wv.Configuration(Nx=Nx, Ny=Ny, Nz=Nz, Nj=c.Nj, Lx=c.Lx, Ly=c.Ly, Lz=c.Lz, N0=c.N0, rho0=c.rho0, g=c.g,
                           planetaryRadius=c.planetaryRadius, rotationRate=c.rotationRate, latitude=c.latitude,
                           isHydrostatic=hydro)
    d = O.build_descriptor(c)
    return c, d, O.random_state(d, 7, 1e-3), wv.WVTransformConstantStratificationKernel(cfg)


# lane-held, run-time and block-wide lines of the x pass
@pytest.mark.parametrize("shape", [(64, 64, 33), (128, 48, 33), (60, 50, 21), (516, 8, 7)])
def test_still_velocity_component_advects_nothing(wv, shape):
    """A geostrophic flow has no vertical velocity: the flux advected by the fields
    that the flux returns (w zero everywhere) is the same flux, bit for bit."""
    c, d, A, k = _setup(wv, shape)
    A = [0.0 * A[0], 0.0 * A[1], A[2]]
    F = k.nonlinearFlux(50.0, 0.0, *A)
    own, adv = k.nonlinearFluxWithAdvectionFields(50.0, 0.0, *A)
    assert not adv[2].any() and adv[0].any()
    for a, b in zip(k.nonlinearFluxUsingAdvectionFields(50.0, 0.0, *A, adv), F):
        assert np.array_equal(a, b)
    k.close()


@pytest.mark.parametrize("shape", [(64, 64, 33), (192, 32, 13), (256, 16, 9), (60, 50, 21), (300, 12, 9)])
def test_own_advection_fields_give_the_flux_bit_for_bit(wv, shape):
    """The returned velocities are the ones the flux used, to the last bit."""
    c, d, A, k = _setup(wv, shape)
    F, adv = k.nonlinearFluxWithAdvectionFields(50.0, 0.0, *A)
    for a, b, f in zip(k.nonlinearFluxUsingAdvectionFields(50.0, 0.0, *A, adv), F, k.nonlinearFlux(50.0, 0.0, *A)):
        assert np.array_equal(a, b) and np.array_equal(b, f)
    k.close()


@pytest.mark.parametrize("shape", [(32, 48, 17), (20, 18, 11), (516, 8, 7)])
@pytest.mark.parametrize("power", [-900, 960])
def test_values_near_the_ends_of_the_range(wv, shape, power):
    """A power of two moves only exponents (tolerances of
    test_scaled_states_give_scaled_fields): lines bounded by 2^-892 and less or by
    2^938 and more keep their values; the flux is quadratic, so half the power there."""
    import torch
    c, d, A, k = _setup(wv, shape)
    s, h = 2.0 ** power, 2.0 ** (power // 2)
    f = k.transformWaveVortexToUVWEta(300.0, 0.0, *A)
    g = k.transformWaveVortexToUVWEta(300.0, 0.0, *[s * x for x in A])
    for a, b in zip(g, f):
        assert np.max(np.abs(a / s - b)) <= 2e-14 * np.max(np.abs(b))
    for a, b in zip(k.nonlinearFlux(300.0, 0.0, *[h * x for x in A]), k.nonlinearFlux(300.0, 0.0, *A)):
        assert np.max(np.abs(a / h / h - b)) <= 1e-13 * np.max(np.abs(b))
    rng = np.random.default_rng(6)
    R = (shape[2], shape[1], shape[0])
    f = rng.standard_normal((4,) + R)
    B = k.transformUVWEtaToWaveVortex(f, 300.0, 0.0)
    S = k.transformUVWEtaToWaveVortex(s * f, 300.0, 0.0)
    for a, b in zip(S, B):
        assert np.max(np.abs(a / s - b)) <= 1e-13 * np.max(np.abs(b))
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()
    q, adv = rng.standard_normal(R), 0.1 * rng.standard_normal((3,) + R)
    one = k.advectFGridScalar(dev(q), dev(adv), True).cpu().numpy()
    big = k.advectFGridScalar(dev(s * q), dev(adv), True).cpu().numpy()
    assert np.max(np.abs(big / s - one)) <= 1e-13 * np.max(np.abs(one))
    u = [dev(s * x) for x in A]  # the VJP is linear in the cotangents
    for a, b in zip(k.flux_vjp(300.0, 0.0, *map(dev, A), *u), k.flux_vjp(300.0, 0.0, *map(dev, A), *map(dev, A))):
        a, b = a.cpu().numpy(), b.cpu().numpy()
        assert np.max(np.abs(a / s - b)) <= 1e-13 * np.max(np.abs(b))
    k.close()


@pytest.mark.parametrize("shape", [(32, 48, 17), (20, 18, 11)])
@pytest.mark.parametrize("angle", [1e-12, 1e-7, 1.9e-3, 1.5e-2, 1.6e-2, 0.3])
def test_sines_of_small_angles_keep_their_digits(wv, shape, angle):
    """A wave along x with Ap = -Am has u = 2 i sin(omega t) cos(kx) times its factor: the
    channel holds nothing but the sine, so its relative error is the sine's."""
    c, d, A, k = _setup(wv, shape)
    omega = d.arrays["omega"]
    l, kk = d.l, d.k
    mode = int(np.flatnonzero((np.abs(l) == 0.0) & (kk > 0.0))[0])
    A = [0.0 * a for a in A]
    A[0][mode, 1], A[1][mode, 1] = 1e-3, -1e-3
    t = angle / float(omega[mode, 1])
    f = k.transformWaveVortexToUVWEta(t, 0.0, *A)
    ref = O.inverse_uvweta(d, *A, t, 0.0)
    assert np.max(np.abs(f[0] - ref[0])) <= 1e-12 * np.max(np.abs(ref[0]))
    k.close()


# y, x and z lines (2 (Nz - 1) points) past 192, on run-time and block-wide stages, and lane-held 256
@pytest.mark.parametrize("shape", [(16, 384, 9), (12, 640, 7), (420, 10, 9), (1000, 8, 7), (10, 12, 161), (8, 10, 257),
                                   (256, 12, 9), (12, 256, 9), (10, 12, 129)])
def test_long_lines_against_long_double(wv, extended, shape):  # noqa: F811
    """Largest error against the oracle in long double at most twice that of the oracle
    in doubles, whose FFTs round alike (1e-16 to 2e-16 of a line), plus 1e-15."""
    c, d, A, k = _setup(wv, shape)
    wide = [a.astype(np.clongdouble) for a in A]
    rng = np.random.default_rng(8)
    fields = rng.standard_normal((4, shape[2], shape[1], shape[0]))

    def check(got, plain, ref):
        for a, b, r in zip(got, plain, ref):
            scale = np.max(np.abs(r))
            far = lambda x: float(np.max(np.abs(np.asarray(x).astype(r.dtype) - r)) / scale)
            assert far(a) <= 2.0 * far(b) + 1e-15, (far(a), far(b))

    check(k.nonlinearFlux(123.0, 0.0, *A), O.nonlinear_flux(d, *A, 123.0, 0.0), extended.nonlinear_flux(d, *wide, 123.0, 0.0))
    check(k.transformWaveVortexToUVWEta(123.0, 0.0, *A), O.inverse_uvweta(d, *A, 123.0, 0.0),
          extended.inverse_uvweta(d, *wide, 123.0, 0.0))
    check(k.transformUVWEtaToWaveVortex(fields, 123.0, 0.0), O.forward(d, fields, 123.0, 0.0),
          extended.forward(d, fields.astype(np.longdouble), 123.0, 0.0))
    k.close()


# lane-held and run-time rows
@pytest.mark.parametrize("shape", [(32, 32, 17), (30, 20, 9)])
def test_rows_of_the_vjp_are_allocated_when_first_needed(wv, shape):
    """A VJP of a state transform and a checkpointed adjoint (which keeps rows of its own)
    do without them; a flux VJP without memory for them gives the same gradient (block
    kernel against lines: the tolerance of the VJP against FP64's own noise, 1e-11)."""
    import torch
    c, d, A, k = _setup(wv, shape)
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()  # noqa: E731
    state = list(map(dev, A))
    k.inverse_vjp(10.0, 0.0, dev(np.ones((4, shape[2], shape[1], shape[0]))))
    ready = k.metrics()["device_bytes"]
    k._lib.wv_test_fail_allocation_after(0)
    try:
        without = k.flux_vjp(10.0, 0.0, *state, *state)
    finally:
        k._lib.wv_test_fail_allocation_after(-1)
    assert k.metrics()["device_bytes"] == ready
    k.close()
    c, d, A, k = _setup(wv, shape)
    k.rk4_adjoint(*state, 0.0, 0.0, 60.0, 2, 1, *state)
    kept = k.metrics()["device_bytes"]
    rows = k.flux_vjp(10.0, 0.0, *state, *state)
    assert k.metrics()["device_bytes"] - kept == 15 * shape[0] * shape[1] * shape[2] * 8
    for a, b in zip(without, rows):
        a, b = a.cpu().numpy(), b.cpu().numpy()
        assert np.max(np.abs(a - b)) <= 1e-11 * np.max(np.abs(b))
    k.close()


@pytest.mark.parametrize("shape", [(256, 200, 9), (512, 16, 7), (16, 512, 7), (12, 10, 129), (10, 12, 201), (516, 8, 7)])
def test_equal_samples_at_the_exponent_boundary(wv, shape):
    """Fields of one modulus near a power of two of the lines' bounds (tests of the lines
    alone: test_fixed_point_lines_cpu.py): the transform scales with the fields."""
    c, d, A, k = _setup(wv, shape)
    sign = np.random.default_rng(9).choice([-1.0, 1.0], (4, shape[2], shape[1], shape[0]))
    ref = k.transformUVWEtaToWaveVortex(0.7 * sign, 0.0, 0.0)
    for step in (-40, -8, -3, -1, 0, 1, 3, 8, 40):
        f = (1.0 + step * 2.0 ** -23) / 1.0025
        for a, b in zip(k.transformUVWEtaToWaveVortex(f * sign, 0.0, 0.0), ref):
            assert np.max(np.abs(a - b * (f / 0.7))) <= 1e-12 * np.max(np.abs(b))
    k.close()
