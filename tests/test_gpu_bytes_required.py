"""sns_bytes_required covers what a handle holds: the server's budget and sns_create's check rest
on it."""
import pytest

from spectral_solver_b200 import Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 12, 16, 24, 32, 48, 64, 96, 128, 256, 512])
@pytest.mark.parametrize("precision", [0, 1])
def test_a_handle_fits_its_requirement(lib, n, precision):
    need = lib.sns_bytes_required(n, precision)
    with Solver(n, precision=precision) as s:
        assert s.device_bytes() <= need
