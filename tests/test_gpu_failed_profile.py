"""A call that fails between two stages leaves work fields that hold the next stage's start; the
calls after it overwrite them, so no step may start from them.  The failure is planted by the
host (the device error word)."""
import numpy as np
import pytest

from spectral_solver_b200 import Solver, _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [16, 64])
@pytest.mark.parametrize("warm", [0, 2, 4])  # later steps: launched, captured after the failure, captured before it
@pytest.mark.parametrize("between", ["max_velocity", "dump_velocity", "forward", "rhs"])
def test_step_after_a_failed_profile(n, between, warm):
    def overwrite(s):
        if between == "forward":
            s.forward(np.ones((n, n, n)))
        elif between == "rhs":
            s.rhs(s.get_state())
        else:
            getattr(s, between)()

    with Solver(n, 400.0, seed=1, pert_amp=0.05, pert_kmax=n // 4) as s:
        s.step(1e-3, warm)
        assert s.lib.sns_debug_set_error_word(s.h, 1) == _lib.SNS_OK
        with pytest.raises(_lib.SnsError):
            s.profile_passes(1e-3, 1)  # fails after its first stage
        state = s.get_state()
        with Solver(n, 400.0) as f:
            f.set_state(state)
            overwrite(s)
            for _ in range(2):
                s.step(1e-3, 2)
                f.step(1e-3, 2)
                assert all(np.array_equal(a, b) for a, b in zip(s.get_state(), f.get_state()))
