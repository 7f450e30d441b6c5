"""Films whose spectra's rows go unpadded (y lines from 2048 points).  Against the FP64 oracle within 1e-6 relative L2: an FP32 transform of length N rounds about
3 log2 N times per axis and direction by 2^-24, at random, which stays below 2e-7 here, and the
tensor's own rounding adds 6e-8."""
import pytest

from fullmag_gb300 import FdmBackend, _abi
from helpers import problem, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,periodic,py", [
    (20, 600, None, 2048), (300, 1030, None, 4096), (60, 700, (1, 0, 0), 2048)])
def test_fields(gpu_lib, oracle, nx, ny, periodic, py):
    kw = problem(nx, ny, 1, d=(3e-9, 2.5e-9, 2e-9), seed=97)
    extra = dict(periodic=periodic, image_counts=tuple(int(p) for p in periodic)) if periodic else {}
    gpu = FdmBackend(**kw, integrator=_abi.INTEGRATOR_RK4, **extra)
    assert gpu.fft_shape()[1] == py
    f = oracle.Problem(**kw, integrator=oracle.RK4, **extra).fields(kw["m0"])
    assert rel_l2(gpu.copy_field(_abi.OBSERVABLE_H_DEMAG), f["h_demag"]) < 1e-6
    assert rel_l2(gpu.copy_field(_abi.OBSERVABLE_H_EFF), f["h_eff"]) < 1e-6
    gpu.close()
