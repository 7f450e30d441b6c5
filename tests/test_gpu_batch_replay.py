"""A batch that continues with the same problems replays the round it captured: the values after
every call are those of the same problems alone."""
import numpy as np
import pytest

from fullmag_gb300 import FdmBackend, FdmBatch, _abi
from helpers import problem

pytestmark = pytest.mark.gpu


def alone(be, t, dt, t_end):
    while t < t_end * (1 - 1e-12):
        st = be.step(min(dt, t_end - t))
        t, dt = st["time_seconds"], st["suggested_next_dt"]
    return t, dt


def test_values_after_every_call(gpu_lib):
    shapes = [(17, 9, 1), (24, 16, 2), (12, 20, 4), (33, 5, 1), (70, 40, 1), (20, 14, 1)]
    plans = [dict(problem(*s, seed=40 + i, alpha=0.05 + 0.02 * i, b_mt=(20.0 * i, 10.0, 0.0)),
                  integrator=_abi.INTEGRATOR_DP45, adaptive_max_error=1e-5) for i, s in enumerate(shapes)]
    batch = FdmBatch(plans)
    singles = [[FdmBackend(**kw), 0.0, 1e-13] for kw in plans]
    for call, t_end in enumerate((4e-13, 8e-13, 8e-13, 1.3e-12, 2.5e-12)):
        steps, _ = batch.step_until(t_end, 1e-13)
        assert (steps >= 1).all() or call == 2
        assert call != 2 or (steps == 0).all()
        for i, s in enumerate(singles):
            s[1], s[2] = alone(*s, t_end)
            # round after round the step control follows FP32 rounding apart: 1e-6 a call
            assert np.abs(batch.copy_field(i) - s[0].copy_field(_abi.OBSERVABLE_M)).max() < 1e-6 * (call + 1), (call, i)
            assert batch.stats(i)["time_seconds"] == pytest.approx(t_end, rel=1e-12)
            assert batch.stats(i)["total_energy_joules"] == pytest.approx(s[0].stats()["total_energy_joules"], rel=1e-5)
            if call % 2:  # evaluates the member's fields in between
                a, b = batch.copy_field(i, _abi.OBSERVABLE_H_EFF), s[0].copy_field(_abi.OBSERVABLE_H_EFF)
                assert np.linalg.norm(a - b) < 1e-5 * np.linalg.norm(b)
    for s in singles:
        s[0].close()
    batch.close()


def test_a_member_beyond_the_batched_passes(gpu_lib, oracle):
    """A caller's 3 x 60 x 8 spectra: a column of that plane takes more shared memory than the fused y+z
    pass is used for, so the batch runs its problems one by one on their streams."""
    plans = [dict(problem(*s, seed=60 + i, alpha=0.1), integrator=_abi.INTEGRATOR_DP45, adaptive_max_error=1e-5,
                  adaptive_dt_max=5e-14) for i, s in enumerate([(3, 60, 8), (17, 9, 1), (12, 20, 4)])]
    plans[0]["spectra"] = oracle.newell_spectra(3, 60, 8, *[plans[0][k] for k in ("dx", "dy", "dz")])
    batch = FdmBatch(plans)
    singles = [[FdmBackend(**kw), 0.0, 5e-14] for kw in plans]
    assert singles[0][0].fft_shape() == (6, 120, 16)
    for call, t_end in enumerate((5e-13, 1e-12)):
        batch.step_until(t_end, 5e-14)
        for i, s in enumerate(singles):
            s[1], s[2] = alone(*s, t_end)
            assert np.abs(batch.copy_field(i) - s[0].copy_field(_abi.OBSERVABLE_M)).max() < 1e-6 * (call + 1), (call, i)
    for s in singles:
        s[0].close()
    batch.close()
