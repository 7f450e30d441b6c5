"""The double-precision path's line transforms at the lengths where they change form: packed
half-length x lines and odd full ones, half-line first and last stages, every butterfly
(2, 3, 4, 5, 7, 8, 11, 13), caller spectra with a larger prime, extents rounded up past such a
prime, several rows and columns per CTA, rows transformed one line at a time, and rows too
long for the fused pass.  Against the FP64 oracle: with caller spectra within 1e-10 relative
L2 (two FP64 FFTs), with the engine's own tensor within 1e-9 (the ulp of f and g that the
27-point second difference amplifies); five RK4 steps within 1e-9."""
import numpy as np
import pytest

from fullmag_gb300 import FdmBackend, _abi
from helpers import problem, rel_l2

pytestmark = pytest.mark.gpu


def check(gpu, orc, kw, tol):
    f = orc.fields(kw["m0"])
    assert rel_l2(gpu.copy_field(_abi.OBSERVABLE_H_DEMAG), f["h_demag"]) < tol
    assert rel_l2(gpu.copy_field(_abi.OBSERVABLE_H_EFF), f["h_eff"]) < tol
    for _ in range(5):
        gpu.step(5e-14)
        orc.step(5e-14)
    assert np.abs(gpu.copy_field(_abi.OBSERVABLE_M) - orc.get_m()).max() < 1e-9
    assert rel_l2(gpu.copy_field(_abi.OBSERVABLE_H_EFF), orc.fields()["h_eff"]) < 1e-9
    gpu.close()
    orc.close()


@pytest.mark.parametrize("spectra", [True, False])
@pytest.mark.parametrize("grid", [(1, 1, 1), (2, 3, 1), (8, 8, 8), (15, 21, 1), (13, 11, 7), (22, 26, 1), (34, 6, 3),
                                  (157, 3, 1), (64, 64, 2), (5, 300, 2), (96, 640, 1), (2000, 2, 1)])
def test_open_lengths(gpu_lib, oracle, grid, spectra):
    nx, ny, nz = grid
    kw = problem(nx, ny, nz, d=(3e-9, 2.5e-9, 2e-9), seed=31, ku1=3e4, u_axis=(0.3, 0.2, 1.0))
    sp = oracle.newell_spectra(nx, ny, nz, kw["dx"], kw["dy"], kw["dz"], thin_film_2d=nz == 1) if spectra else None
    gpu = FdmBackend(**kw, integrator=_abi.INTEGRATOR_RK4, precision=_abi.PRECISION_DOUBLE, spectra=sp)
    if spectra:
        assert gpu.fft_shape() == (2 * nx, 2 * ny, 1 if nz == 1 else 2 * nz)
    check(gpu, oracle.Problem(**kw, integrator=oracle.RK4), kw, 1e-10 if spectra else 1e-9)


@pytest.mark.parametrize("grid,periodic", [((17, 16, 1), (1, 0, 0)), ((24, 17, 2), (1, 1, 0)), ((34, 9, 1), (1, 1, 0)),
                                           ((4455, 1, 1), (1, 0, 0))])
def test_periodic_lengths(gpu_lib, oracle, grid, periodic):
    nx, ny, nz = grid
    kw = problem(nx, ny, nz, seed=32)
    images = tuple(1 if p else 0 for p in periodic)
    orc = oracle.Problem(**kw, integrator=oracle.RK4, periodic=periodic, image_counts=images)
    gpu = FdmBackend(**kw, integrator=_abi.INTEGRATOR_RK4, precision=_abi.PRECISION_DOUBLE, periodic=periodic,
                     image_counts=images)
    check(gpu, orc, kw, 1e-9)
