"""Periodic lines that fill the shared memory of a CTA to the last element: the longest odd film
and z lines of the double-precision path, the longest odd film line of the single-precision one."""
import numpy as np
import pytest

from fullmag_gb300 import FdmBackend, _abi
from helpers import problem, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,periodic,precision,tol", [
    ((3, 2421, 1), (0, 1, 0), _abi.PRECISION_DOUBLE, 1e-9),
    ((2, 2, 2421), (0, 0, 1), _abi.PRECISION_DOUBLE, 1e-9),
    # FP32: 3 log2 N roundings of 2^-24 per axis and direction, and the tensor's own
    ((4, 4557, 1), (0, 1, 0), _abi.PRECISION_SINGLE, 1e-6)])
def test_fields(gpu_lib, oracle, shape, periodic, precision, tol):
    kw = problem(*shape, seed=95)
    images = tuple(1 if p else 0 for p in periodic)
    gpu = FdmBackend(**kw, integrator=_abi.INTEGRATOR_HEUN, precision=precision, periodic=periodic, image_counts=images)
    orc = oracle.Problem(**kw, integrator=oracle.HEUN, periodic=periodic, image_counts=images)
    f = orc.fields(kw["m0"])
    assert rel_l2(gpu.copy_field(_abi.OBSERVABLE_H_DEMAG), f["h_demag"]) < tol
    assert rel_l2(gpu.copy_field(_abi.OBSERVABLE_H_EFF), f["h_eff"]) < tol
    gpu.step(5e-14)
    orc.step(5e-14)
    assert np.abs(gpu.copy_field(_abi.OBSERVABLE_M) - orc.get_m()).max() < 10 * tol
    gpu.close()
    orc.close()
