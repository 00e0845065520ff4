"""Steps on a stopped clock (one that reached its horizon, or was never started) leave the state
as it is.  A state with content outside the truncation sphere keeps it through them, so nothing
may then be computed as if those modes were zero: the velocity, the diagnostics and the steps that
follow are bit for bit those of a handle that was never stepped."""
import numpy as np
import pytest

from spectral_solver_b200 import Solver

pytestmark = pytest.mark.gpu

NU, DT = 1.0 / 400.0, 1e-3


def unmasked_state(n):
    """A Hermitian spectrum with content at every |m| < N/2 on each axis (corners included)."""
    rng = np.random.default_rng(n)
    m = np.fft.fftfreq(n, 1.0 / n)
    kz, ky, kx = np.meshgrid(m, m, m, indexing="ij")
    weight = 0.3 / (1.0 + kx ** 2 + ky ** 2 + kz ** 2)
    inside = (abs(kx) < n / 2) & (abs(ky) < n / 2) & (abs(kz) < n / 2)
    return [np.fft.fftn(rng.standard_normal((n, n, n))) * weight * inside for _ in range(3)]


def same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


# 48, 128: the four-launch stage, steps replayed from a graph; 256: the streaming passes
@pytest.mark.parametrize("n", [48, 128, 256])
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("form", [0, 1])
def test_idle_steps_are_not_taken(n, precision, form):
    if n == 128 and form != precision:
        pytest.skip("one precision of each form at this size")
    full = unmasked_state(n)

    def solver():
        s = Solver(n, nu=NU, precision=precision)
        if form:
            s.set_nonlinear_form(1)
        s.set_state(full)
        return s

    with solver() as s, solver() as f:
        start = f.get_state()
        s.step_cfl(1)  # the clock was never started
        s.step_cfl(2)
        assert same(s.get_state(), start)
        assert s.max_velocity() == f.max_velocity()
        assert s.diagnostics() == f.diagnostics()
        s.step(DT)
        f.step(DT)
        assert same(s.get_state(), f.get_state())
        # a clock that runs into its horizon between two states
        s.set_clock(0.0, t_end=0.5 * DT, cfl=0.5, dt_max=DT)
        s.step_cfl(1)
        s.set_state(full)
        s.step_cfl(3)
        assert s.clock()["stopped"] and s.clock()["steps"] == 1
        f.set_state(full)
        assert same(s.get_state(), start)
        assert s.diagnostics() == f.diagnostics()
        # a running clock after it
        for x in (s, f):
            x.set_clock(0.0, cfl=0.2, dt_max=DT)
            x.step_cfl(2)
        assert same(s.get_state(), f.get_state())
        s.step(DT, 4)
        f.step(DT, 4)
        assert same(s.get_state(), f.get_state()) and s.diagnostics() == f.diagnostics()
