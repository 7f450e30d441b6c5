"""The single-precision line transforms at every two-level length (2^a times 1, 5/4, 3/2, 7/4
from 16 to 1024) of each axis: rows, thin films, the three-pass and the fused column passes,
the register, packed and shared-memory z passes, the unpadded (periodic) forms, the batched
kernels and the reverse sweep.  Against the FP64 oracle within 1e-6 relative L2: an FP32
transform of length N rounds about 3 log2 N times per axis and direction by 2^-24, at random,
which stays below 2e-7 here, and the tensor's own rounding adds 6e-8."""
import numpy as np
import pytest

from fullmag_gb300 import FdmBackend, FdmBatch, _abi
from helpers import problem, rel_l2

pytestmark = pytest.mark.gpu

TOL = 1e-6
D = (3e-9, 2.5e-9, 2e-9)


def check(gpu, orc, kw):
    f = orc.fields(kw["m0"])
    assert rel_l2(gpu.copy_field(_abi.OBSERVABLE_H_DEMAG), f["h_demag"]) < TOL
    assert rel_l2(gpu.copy_field(_abi.OBSERVABLE_H_EFF), f["h_eff"]) < TOL
    shape = gpu.fft_shape()
    gpu.close()
    orc.close()
    return shape


def open_box(oracle, nx, ny, nz, seed=41):
    kw = problem(nx, ny, nz, d=D, seed=seed)
    return check(FdmBackend(**kw, integrator=_abi.INTEGRATOR_RK4), oracle.Problem(**kw, integrator=oracle.RK4), kw)


FILMS = [(17, 9, 20, 20), (23, 11, 24, 24), (28, 14, 28, 28), (32, 16, 32, 32), (33, 17, 40, 40), (47, 24, 48, 48),
         (50, 28, 56, 56), (64, 31, 64, 64), (65, 33, 80, 80), (96, 41, 96, 96), (110, 56, 112, 112),
         (128, 57, 128, 128), (129, 65, 160, 160), (190, 96, 192, 192), (193, 97, 224, 224), (256, 128, 256, 256),
         (257, 129, 320, 320), (384, 161, 384, 384), (385, 193, 448, 448), (511, 256, 512, 512), (513, 257, 640, 640),
         (768, 380, 768, 768), (770, 448, 896, 896), (1000, 500, 1024, 1024), (1025, 513, 2048, 2048)]


@pytest.mark.parametrize("nx,ny,half,py", FILMS)
def test_films(gpu_lib, oracle, nx, ny, half, py):
    px, p, _ = open_box(oracle, nx, ny, 1)
    assert (px, p) == (2 * half, py)


@pytest.mark.parametrize("ny", [1, 9, 12, 13, 17, 21, 28, 32, 40, 48, 50, 64, 70, 90, 100, 128, 150, 192, 200, 256, 300, 384, 400, 512])
@pytest.mark.parametrize("fused", [True, False])
def test_y_passes(gpu_lib, oracle, monkeypatch, ny, fused):
    if not fused:
        monkeypatch.setenv("FULLMAG_FDM_NO_FUSED_YZ", "1")
    open_box(oracle, 19, ny, 2)


@pytest.mark.parametrize("nz", [2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12])
@pytest.mark.parametrize("fused", [True, False])
def test_z_in_registers(gpu_lib, oracle, monkeypatch, nz, fused):
    if not fused:
        monkeypatch.setenv("FULLMAG_FDM_NO_FUSED_YZ", "1")
    _, _, pz = open_box(oracle, 21, 18, nz)
    assert pz == (2 * nz if nz <= 8 else 20 if nz <= 10 else 24)


@pytest.mark.parametrize("nz", [13, 16, 17, 24, 28, 31, 40, 45, 56, 64, 70])
@pytest.mark.parametrize("pair", ["0", "1"])
def test_z_in_shared_memory(gpu_lib, oracle, monkeypatch, nz, pair):
    monkeypatch.setenv("FULLMAG_FDM_Z_PAIR", pair)
    open_box(oracle, 9, 260, nz)  # py = 640: the plane does not fit the fused pass


def test_small_plane_beyond_the_register_lengths(gpu_lib, oracle):
    # a small (y, z) plane keeps powers of two there: the general fused y+z pass
    _, py, pz = open_box(oracle, 20, 17, 13)
    assert (py, pz) == (64, 32)


@pytest.mark.parametrize("shape,periodic", [((2 * h, n, 1), (1, 1, 0)) for h, n in
                                            [(16, 16), (20, 24), (28, 40), (48, 56), (80, 96), (112, 128), (160, 192),
                                             (224, 256), (256, 320), (320, 384), (24, 448), (24, 640),
                                             (20, 768), (16, 896), (16, 1024), (33, 34),
                                             (45, 105), (98, 75)]] +
                         [((40, 17, 1), (1, 0, 0)), ((48, 200, 1), (1, 0, 0)), ((33, 64, 1), (0, 1, 0)),
                          ((32, 20, 4), (1, 1, 0)), ((18, 24, 3), (0, 1, 0)), ((40, 11, 10), (1, 0, 0)),
                          ((20, 12, 14), (1, 1, 0))])
def test_periodic_lengths(gpu_lib, oracle, shape, periodic):
    kw = problem(*shape, d=D, seed=42)
    images = tuple(1 if p else 0 for p in periodic)
    check(FdmBackend(**kw, integrator=_abi.INTEGRATOR_RK4, periodic=periodic, image_counts=images),
          oracle.Problem(**kw, integrator=oracle.RK4, periodic=periodic, image_counts=images), kw)


def test_batched_lengths(gpu_lib):
    """Films and small volumes of every batched kernel in one batch against the same problems
    alone: the two sides run the same step control on transforms that differ only in how the
    work is tiled, so after twenty small steps they agree to a few FP32 roundings."""
    shapes = [(300, 8, 1), (20, 170, 1), (33, 17, 1), (8, 8, 5), (9, 170, 2), (24, 40, 3), (400, 20, 2), (13, 20, 13), (600, 9, 1), (10, 300, 1), (10, 260, 2)]
    plans = [dict(problem(*s, seed=50 + i, alpha=0.1), integrator=_abi.INTEGRATOR_DP45, adaptive_max_error=1e-5,
                  adaptive_dt_max=5e-14) for i, s in enumerate(shapes)]
    batch = FdmBatch(plans)
    batch.step_until(1e-12, 5e-14)
    for i, kw in enumerate(plans):
        one = FdmBackend(**kw)
        t = 0.0
        while t < 1e-12 * (1 - 1e-12):
            t = one.step(min(5e-14, 1e-12 - t))["time_seconds"]
        assert np.abs(batch.copy_field(i) - one.copy_field(_abi.OBSERVABLE_M)).max() < 1e-5, shapes[i]
        one.close()
