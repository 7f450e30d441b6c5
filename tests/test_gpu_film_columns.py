"""Films with long y lines: on both sides of the number of kx columns where their column pass changes
form, and where the spectra's rows go unpadded (from 2048 points), open and periodic, alone and in a
batch.  Against the FP64 oracle within 1e-6 relative L2: an FP32 transform of length N rounds about
3 log2 N times per axis and direction by 2^-24, at random, which stays below 2e-7 here, and the
tensor's own rounding adds 6e-8."""
import numpy as np
import pytest

from fullmag_gb300 import FdmBackend, FdmBatch, _abi
from helpers import problem, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,periodic,py", [
    (8, 440, None, 1024), (32, 448, None, 1024), (40, 448, None, 896), (32, 512, None, 1024), (40, 500, None, 1024),
    (8, 380, None, 768), (32, 450, (1, 0, 0), 1024), (80, 440, (1, 0, 0), 896), (320, 440, (1, 0, 0), 896),
    (8, 512, (0, 1, 0), 512), (64, 512, (1, 1, 0), 512), (80, 512, (1, 1, 0), 512), (320, 512, (1, 1, 0), 512),
    (64, 896, (1, 1, 0), 896), (320, 896, (1, 1, 0), 896), (16, 1024, (1, 1, 0), 1024), (320, 1024, (1, 1, 0), 1024),
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


def test_batch_member_as_alone(gpu_lib):
    """Twenty small steps on transforms of another length: a few FP32 roundings apart."""
    plans = [dict(problem(nx, ny, 1, seed=98 + ny, alpha=0.1), integrator=_abi.INTEGRATOR_DP45, adaptive_max_error=1e-5,
                  adaptive_dt_max=5e-14) for nx, ny in ((20, 440), (30, 512), (150, 448))]
    batch = FdmBatch(plans)
    batch.step_until(1e-12, 5e-14)
    for i, kw in enumerate(plans):
        one = FdmBackend(**kw)
        t = 0.0
        while t < 1e-12 * (1 - 1e-12):
            t = one.step(min(5e-14, 1e-12 - t))["time_seconds"]
        assert np.abs(batch.copy_field(i) - one.copy_field(_abi.OBSERVABLE_M)).max() < 1e-5
        one.close()
    batch.close()
