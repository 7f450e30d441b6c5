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


def same_run(a, b, tol=1e-6):
    """States and statistics of two runs of the same steps: their passes with and without
    statistics are compiled apart, so they may round differently by 2^-24 a stage."""
    assert np.abs(a[0] - b[0]).max() < tol
    assert a[1]["step"] == b[1]["step"] and abs(a[1]["time_seconds"] - b[1]["time_seconds"]) < 1e-24
    for k in ("exchange_energy_joules", "total_energy_joules", "max_effective_field_amplitude", "max_rhs_amplitude"):
        assert abs(a[1][k] - b[1][k]) <= 20 * tol * abs(b[1][k]), k


def run(kw, plan):
    """plan: (dt, steps, many) blocks, or an array to upload."""
    be = FdmBackend(**kw)
    st = None
    for block in plan:
        if isinstance(block, np.ndarray):
            be.upload(block)
        elif block[2]:
            st = be.step_many(block[0], block[1])
        else:
            for _ in range(block[1]):
                st = be.step(block[0])
    out = be.copy_field(_abi.OBSERVABLE_M), st
    be.close()
    return out


TERMS = {"plain": dict(), "no_demag": dict(enable_demag=False), "current": dict(oersted_current=1e-3, oersted_radius=2e-8),
         "dmi": dict(dmi_d_interfacial=2e-3)}


@pytest.mark.parametrize("terms", list(TERMS))
@pytest.mark.parametrize("integrator", INTEGRATORS + [_abi.INTEGRATOR_ABM3])
def test_many_steps_as_single_ones(gpu_lib, integrator, terms):
    """Blocks of an odd and of an even number of steps, from either parity, with another step size,
    after single steps and after an upload."""
    kw = problem(25, 12, 2, seed=74, alpha=0.1, **TERMS[terms])
    kw["integrator"] = integrator
    m1 = random_unit(25 * 12 * 2, 75)
    blocks = [(DT, 3, True), (DT, 4, True), (DT, 1, False), (DT, 4, True), (0.5 * DT, 5, True), (0.5 * DT, 2, True), m1,
              (DT, 6, True), (DT, 1, False), (DT, 9, True)]
    for end in (1, 2, 4, 5, 8, len(blocks)):
        plan = blocks[:end]
        singles = [b if isinstance(b, np.ndarray) else (b[0], b[1], False) for b in plan]
        same_run(run(kw, plan), run(kw, singles))
