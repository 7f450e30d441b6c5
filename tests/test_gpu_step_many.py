"""Runs of fixed steps (step and step_many) from a state that was replaced in between: every
step starts from the state and the field in hand, whatever the steps before it prepared."""
import numpy as np
import pytest

from fullmag_gb300 import FdmBackend, _abi
from helpers import problem, random_unit

pytestmark = pytest.mark.gpu

DT = 5e-14
INTEGRATORS = [_abi.INTEGRATOR_HEUN, _abi.INTEGRATOR_RK4]


def fresh_then(kw, m, steps, field_map=None):
    """The state that a new handle reaches from m."""
    be = FdmBackend(**dict(kw, m0=m))
    if field_map is not None:
        be.set_field_map(field_map)
    for _ in range(steps):
        be.step(DT)
    out = be.copy_field(_abi.OBSERVABLE_M)
    be.close()
    return out


@pytest.mark.parametrize("demag", [True, False])
@pytest.mark.parametrize("integrator", INTEGRATORS)
def test_step_after_an_upload_or_a_field_map(gpu_lib, integrator, demag):
    kw = problem(24, 10, 3, seed=71, enable_demag=demag)
    kw["integrator"] = integrator
    m1 = random_unit(24 * 10 * 3, 72)
    be = FdmBackend(**kw)
    be.step(DT)
    be.step(DT)
    # two steps back to the same state parity and dt as the prepared stage of the old state
    be.upload(m1)
    be.step(DT)
    assert np.array_equal(be.copy_field(_abi.OBSERVABLE_M), fresh_then(kw, m1, 1))
    h = 4e4 * random_unit(24 * 10 * 3, 73)
    be.upload(m1)
    be.set_field_map(h)
    be.step(DT)
    assert np.array_equal(be.copy_field(_abi.OBSERVABLE_M), fresh_then(kw, m1, 1, h))
    be.close()
