"""The first-same-as-last derivative of the adaptive integrators changes buffers with the state
parity: a step from any parity, after a refresh, after a rejected attempt and after an upload
agrees with the same step of a new handle that starts from the same state."""
import numpy as np
import pytest

from fullmag_gb300 import FdmBackend, _abi
from helpers import problem, random_unit

pytestmark = pytest.mark.gpu

DT = 5e-14


def step_from(kw, m, dt):
    be = FdmBackend(**dict(kw, m0=m))
    st = be.step(dt)
    out = be.copy_field(_abi.OBSERVABLE_M), st
    be.close()
    return out


def check(be, kw, dt):
    """One step of be against a new handle's: the derivative kept from the last step and the one
    evaluated anew differ by rounding, 6e-10 of the error norm in FP32.  That is a few 1e-6 of the
    norm of a rejected attempt, but may be all of a small step's, whose suggestion follows its
    third or fifth root."""
    want, sw = step_from(kw, be.copy_field(_abi.OBSERVABLE_M), dt)
    st = be.step(dt)
    assert np.abs(be.copy_field(_abi.OBSERVABLE_M) - want).max() < 1e-6
    assert st["dt_seconds"] == pytest.approx(sw["dt_seconds"], rel=1e-5)
    single = kw["precision"] == _abi.PRECISION_SINGLE
    assert st["suggested_next_dt"] == pytest.approx(sw["suggested_next_dt"], rel=0.3 if single else 1e-5)
    assert st["total_energy_joules"] == pytest.approx(sw["total_energy_joules"], rel=1e-5)
    return st


@pytest.mark.parametrize("demag", [True, False])
@pytest.mark.parametrize("precision", [_abi.PRECISION_SINGLE, _abi.PRECISION_DOUBLE])
@pytest.mark.parametrize("integrator", [_abi.INTEGRATOR_RK23, _abi.INTEGRATOR_DP45])
def test_roles(gpu_lib, integrator, precision, demag):
    kw = problem(18, 11, 3, seed=76, alpha=0.1, enable_demag=demag)
    kw.update(integrator=integrator, precision=precision, adaptive_max_error=1e-4, adaptive_dt_max=1e-12)
    be = FdmBackend(**kw)
    for _ in range(3):
        check(be, kw, DT)
    for _ in range(2):
        be.copy_field(_abi.OBSERVABLE_H_EFF)  # evaluates the committed state again
        check(be, kw, DT)
    for _ in range(3):
        st = check(be, kw, 1e-12)
        assert st["dt_seconds"] < 1e-12  # rejected at least once
    for seed in (77, 78):
        be.upload(random_unit(18 * 11 * 3, seed))
        check(be, kw, DT)
        check(be, kw, DT)
        check(be, kw, DT)
    be.close()
