"""Which arithmetic an FP32X2 handle runs (wv_get_fixed_point), how to choose it, and the
accuracy of the paired-FP32 step where fixed-point lines are the default."""
import numpy as np
import pytest

import wv_oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def wv():
    import torch
    import wvgpu
    from wvgpu import build
    assert torch.cuda.is_available()
    build.build()
    return wvgpu


def _handle(wv, shape, precision="fp32x2", hydro=False):
    Nx, Ny, Nz = shape
    return wv.WVTransformConstantStratificationKernel(
        wv.Configuration(Nx=Nx, Ny=Ny, Nz=Nz, Nj=O.default_nj(Nz), Lx=3125.0 * Nx, Ly=3125.0 * Ny, Lz=4000.0, latitude=33.0,
                         isHydrostatic=hydro), precision=precision)


def _state(wv, k, seed=3):
    import torch
    return [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in wv.synthetic_state(k, seed=seed, urms=0.1)]


# lane-held lines on every axis; below 65536 points only where y or z lines are not warp
# registers (multiples of 32 points); not with 192 points along x or y; no run-time lengths
@pytest.mark.parametrize("shape,fixed", [((64, 64, 17), True), ((64, 32, 17), False), ((32, 32, 33), False), ((48, 48, 25), True),
                                         ((16, 16, 9), True), ((24, 64, 13), True), ((128, 64, 33), True), ((192, 96, 49), False),
                                         ((96, 192, 49), False), ((96, 96, 97), True), ((60, 64, 33), False), ((64, 64, 31), False)])
def test_default_route(wv, shape, fixed):
    k = _handle(wv, shape)
    assert k.fixed_point() == fixed
    k.close()


@pytest.mark.parametrize("precision,fixed", [("fp64", True), ("mixed", False)])
def test_other_handles_have_one_route(wv, precision, fixed):
    k = _handle(wv, (64, 64, 33), precision)
    assert k.fixed_point() == fixed
    k.set_fixed_point(fixed)
    with pytest.raises(wv.WVKernelError):
        k.set_fixed_point(not fixed)
    assert k.fixed_point() == fixed
    k.close()


def test_choosing_a_route_and_going_back(wv):
    k = _handle(wv, (64, 64, 33))
    A = _state(wv, k)
    flux = lambda: [f.cpu().numpy() for f in k.nonlinearFlux(50.0, 0.0, *A)]  # noqa: E731
    fixed = flux()
    exact = _handle(wv, (64, 64, 33), "fp64")
    for a, b in zip(exact.nonlinearFlux(50.0, 0.0, *A), fixed):
        assert np.array_equal(a.cpu().numpy(), b)
    exact.close()
    variants = k.fft_variants()
    k.set_fft_variants(*variants)  # as reported: paired FP32 all the same
    assert not k.fixed_point() and k.fft_variants() == variants
    paired = flux()
    assert any(not np.array_equal(a, b) for a, b in zip(paired, fixed))
    k.set_fixed_point()
    assert k.fixed_point()
    assert all(np.array_equal(a, b) for a, b in zip(flux(), fixed))
    k.set_vertical_kernels("cuda", "cuda")
    assert not k.fixed_point()
    k.set_fixed_point(True)  # the vertical transforms come along
    assert k.vertical_kernels() == ("fft", "fft")
    assert all(np.array_equal(a, b) for a, b in zip(flux(), fixed))
    k.set_fixed_point(False)
    assert all(np.array_equal(a, b) for a, b in zip(flux(), paired))
    k.close()
    k = _handle(wv, (60, 50, 31))
    with pytest.raises(wv.WVKernelError):
        k.set_fixed_point()
    k.close()


@pytest.mark.parametrize("shape", [(64, 64, 33), (96, 96, 49), (60, 50, 31)])
@pytest.mark.parametrize("hydro", [False, True])
def test_paired_steps_match_fp64(wv, shape, hydro):
    """Twenty RK4 steps of a turbulent state in paired FP32, chosen or default: every field
    within 1e-8 of FP64's in relative L2, as test_fp32x2_fields_after_rk4_steps_match_fp64."""
    import torch
    fields = []
    for precision in ("fp64", "fp32x2"):
        k = _handle(wv, shape, precision, hydro)
        A = wv.synthetic_state(k, seed=5, urms=0.1)
        dt = wv.cfl_time_step(k, *A)
        A = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in A]
        if precision == "fp32x2":
            k.set_fft_variants(*k.fft_variants())
            assert not k.fixed_point()
        k.rk4(*A, 0.0, 0.0, dt, 20)
        fields.append(k.transformWaveVortexToUVWEta(20 * dt, 0.0, *A).cpu().numpy())
        k.close()
    for q in (0, 1, 3) if hydro else range(4):
        a, b = fields[0][q], fields[1][q]
        assert np.linalg.norm(b - a) <= 1e-8 * np.linalg.norm(a)
    assert not np.array_equal(*fields)
