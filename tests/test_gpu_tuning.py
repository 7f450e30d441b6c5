"""The launch shapes that a handle runs with are its own: a search made for the fused y+z pass, or
with another choice forced, is not applied to a handle of the same grid that runs other passes."""
import pytest

from fullmag_gb300 import FdmBackend, _abi
from helpers import problem

pytestmark = pytest.mark.gpu


def make(nx, ny, nz, **terms):
    return FdmBackend(**problem(nx, ny, nz, seed=81, **terms), integrator=_abi.INTEGRATOR_RK4)


def test_three_passes_after_the_fused_pass(gpu_lib, monkeypatch):
    make(22, 18, 5).close()  # fused y+z
    monkeypatch.setenv("FULLMAG_FDM_NO_FUSED_YZ", "1")
    be = make(22, 18, 5)
    assert be.tuning()["z_pair"] == 2  # pz = 10: the register z pass
    be.set_kernel_timing(True)
    be.refresh()
    assert be.kernel_times()["z_convolve"][1] == 1 and be.kernel_times()["yz_convolve"][1] == 0
    be.close()


def test_z_pass_after_a_problem_without_demag(gpu_lib, monkeypatch):
    monkeypatch.setenv("FULLMAG_FDM_Z_PAIR", "1")
    assert make(16, 512, 20, enable_demag=False).tuning()["z_pair"] == 0  # same extents, no z pass
    assert make(16, 512, 20).tuning()["z_pair"] == 1


# pz 32 to 128; the plane of 260 rows does not fit the fused pass
@pytest.mark.parametrize("nz", [16, 19, 22, 26, 31, 40, 44, 50, 60])
def test_forced_z_pass(gpu_lib, monkeypatch, nz):
    for forced in ("0", "1", "0"):
        monkeypatch.setenv("FULLMAG_FDM_Z_PAIR", forced)
        be = make(10, 260, nz)
        assert be.tuning()["z_pair"] == int(forced)
        be.close()


def test_forced_rows(gpu_lib, monkeypatch):
    monkeypatch.setenv("FULLMAG_FDM_ROWS_PER_CTA", "5")
    assert make(23, 30, 1).tuning()["rows_per_cta"] == 5
    monkeypatch.delenv("FULLMAG_FDM_ROWS_PER_CTA")
    assert make(23, 30, 1).tuning()["rows_per_cta"] in (1, 2, 4, 8, 16)
