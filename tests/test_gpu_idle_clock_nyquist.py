"""Steps on a stopped clock leave the plane mx = N/2 as it is too, where a state that was set may hold
more than the mode (N/2, 0, 0); a step that is taken zeroes it."""
import numpy as np
import pytest

from spectral_solver_b200 import Solver

pytestmark = pytest.mark.gpu

NU, DT = 1.0 / 400.0, 1e-3


def full_state(n):
    """A Hermitian spectrum with content at every mode."""
    rng = np.random.default_rng(n)
    m = np.fft.fftfreq(n, 1.0 / n)
    kz, ky, kx = np.meshgrid(m, m, m, indexing="ij")
    weight = 0.3 / (1.0 + kx ** 2 + ky ** 2 + kz ** 2)
    return [np.fft.fftn(rng.standard_normal((n, n, n))) * weight for _ in range(3)]


def same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


# 48, 128: the sweep of the generic passes; 256: the fused forward z and sweep
@pytest.mark.parametrize("n", [48, 128, 256])
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("form", [0, 1])
def test_idle_steps_keep_the_plane(n, precision, form):
    full = full_state(n)

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
        for x in (s, f):
            x.set_clock(0.0, cfl=0.2, dt_max=DT)
            x.step_cfl(2)
        got = s.get_state()
        assert same(got, f.get_state())
        for c in got:
            c = c[:, :, n // 2].copy()
            c[0, 0] = 0.0
            assert not np.any(c)
        s.step(DT, 3)
        f.step(DT, 3)
        assert same(s.get_state(), f.get_state()) and s.diagnostics() == f.diagnostics()
