"""Where the fixed-point lines of FP64 handles could lose what plain doubles keep:
advecting velocities that are identically zero."""
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
