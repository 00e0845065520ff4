"""Steps of small grids replay a captured graph once a handle has warmed up: the replayed steps
equal steps taken launch by launch (fresh handles, one or two steps each) bit for bit, across a
change of dt, viscosity, nonlinear form, pruning, compensation and state, and next to the
device clock."""
import numpy as np
import pytest

from spectral_solver_b200 import Solver

pytestmark = pytest.mark.gpu


def same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


# 128: the largest grid that replays; 256: launch by launch throughout
@pytest.mark.parametrize("n", [8, 48, 128, 256])
@pytest.mark.parametrize("precision", [0, 1])
def test_replayed_steps_are_the_launched_steps(n, precision):
    def fresh(state, prepare=lambda s: None):
        s = Solver(n, 1600.0, precision=precision)
        s.set_state(state)
        prepare(s)
        return s

    with Solver(n, 1600.0, seed=2, pert_amp=0.05, pert_kmax=max(1, n // 8), precision=precision) as s:
        s.step(1e-3, 3)  # launched, launched, captured

        def check(dt, prepare=lambda s: None):
            before = s.get_state()
            with fresh(before, prepare) as f:
                f.step(dt)  # a new handle's first step is launched
                want = f.get_state()
            prepare(s)
            s.step(dt)
            assert same(s.get_state(), want)

        check(1e-3)
        check(2e-3)
        check(2e-3, lambda s: s._check(s.lib.sns_set_viscosity(s.h, 1.0 / 300.0)))
        check(1e-3, lambda s: (s._check(s.lib.sns_set_viscosity(s.h, 1.0 / 300.0)), s.set_sphere_pruning(False)))
        s._check(s.lib.sns_set_viscosity(s.h, 1.0 / 1600.0))
        s.set_sphere_pruning(True)
        check(1e-3, lambda s: s.set_nonlinear_form(1))
        s.set_nonlinear_form(0)
        # a state from outside drops the sphere flag: its first step is launched, later ones replay
        s.set_state(s.get_state())
        check(1e-3)
        check(1e-3)
        if precision:
            s.set_compensation(False)
            u = s.get_state()
            with fresh(u, lambda f: f.set_compensation(False)) as f:
                f.step(1e-3)
                s.step(1e-3)
                assert same(s.get_state(), f.get_state())
            s.set_compensation(True)
        # the clock's steps replay their own graph; a fixed step between them leaves it alone
        s.set_clock(0.0, cfl=0.4, dt_max=0.5)
        s.step_cfl(3)
        s.step(1e-3)
        t = s.clock()["t"]
        before = s.get_state()
        dt = min(0.5, 0.4 * 2.0 * np.pi / n / s.max_velocity())
        with fresh(before) as f:
            f.step(dt)
            s.step_cfl(1)
            assert same(s.get_state(), f.get_state())
        assert s.clock()["dt"] == dt and s.clock()["t"] == t + dt
