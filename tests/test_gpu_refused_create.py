"""A create that the engine refuses leaves nothing behind for the next one."""
import numpy as np
import pytest

from fullmag_gb300 import FdmBackend, FdmError, _abi
from helpers import problem, random_unit

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [_abi.PRECISION_SINGLE, _abi.PRECISION_DOUBLE])
def test_valid_create_after_a_refused_one(gpu_lib, precision):
    # z lines of 8192 points do not fit the shared memory of a CTA
    with pytest.raises(FdmError):
        FdmBackend(**problem(2, 2, 4096, seed=99), precision=precision)
    for shape in ((12, 1, 5), (12, 9, 1)):
        be = FdmBackend(**problem(*shape, seed=99), precision=precision)
        be.step(5e-14)
        be.upload(random_unit(int(np.prod(shape)), 3))
        be.step(5e-14)
        be.close()
