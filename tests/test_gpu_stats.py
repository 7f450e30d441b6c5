"""Statistics of a step at the CTA counts where their reduction changes form.  The per-cell terms
are the same whatever the rows per CTA, and their compensated float-float sums round by 2^-48 per
addition, 6e-11 over the 18000 cells here, so the energies agree within 1e-10 and the maxima
exactly."""
import pytest

from fullmag_gb300 import FdmBackend, _abi
from helpers import problem

pytestmark = pytest.mark.gpu

ENERGIES = ("exchange_energy_joules", "demag_energy_joules", "external_energy_joules", "anisotropy_energy_joules",
            "total_energy_joules")
MAXIMA = ("max_effective_field_amplitude", "max_demag_field_amplitude", "max_rhs_amplitude")


def compare(a, b, tol):
    scale = max(abs(a[k]) for k in ENERGIES)
    for k in ENERGIES:
        assert abs(a[k] - b[k]) <= tol * scale, (k, a[k], b[k])
    for k in MAXIMA:
        assert a[k] == b[k], (k, a[k], b[k])


@pytest.mark.parametrize("integrator", [_abi.INTEGRATOR_HEUN, _abi.INTEGRATOR_DP45])
@pytest.mark.parametrize("rows", [1, 511, 512, 513, 1024, 1025, 3000])  # in the pass up to 512 CTAs
def test_sums_at_any_number_of_ctas(gpu_lib, monkeypatch, rows, integrator):
    kw = problem(6, rows, 1, seed=91, ku1=2e4, enable_demag=rows <= 1024)
    kw.update(integrator=integrator, adaptive_max_error=1e-3, adaptive_dt_max=5e-14)
    got = []
    for per_cta in ("1", "7"):
        monkeypatch.setenv("FULLMAG_FDM_ROWS_PER_CTA", per_cta)
        be = FdmBackend(**kw)
        assert be.tuning()["rows_per_cta"] == int(per_cta)
        steps = [be.stats()] + [be.step(5e-14) for _ in range(3)]
        got.append(steps)
        be.close()
    for a, b in zip(*got):
        compare(a, b, 1e-10)


@pytest.mark.parametrize("rows,integrator", [(20, _abi.INTEGRATOR_HEUN), (20, _abi.INTEGRATOR_DP45), (600, _abi.INTEGRATOR_RK4)])
def test_kernel_timing_covers_the_reduction(gpu_lib, rows, integrator):
    kw = problem(8, rows, 1, seed=92)
    kw.update(integrator=integrator, adaptive_max_error=1e-3, adaptive_dt_max=5e-14)
    plain, timed = FdmBackend(**kw), FdmBackend(**kw)
    timed.set_kernel_timing(True)
    for n in range(1, 4):
        a, b = plain.step(5e-14), timed.step(5e-14)
        assert [a[k] for k in ENERGIES + MAXIMA] == [b[k] for k in ENERGIES + MAXIMA]  # the same bits
        ms, count = timed.kernel_times()["finalize_stats"]
        assert count == n and ms > 0
    plain.close()
    timed.close()
