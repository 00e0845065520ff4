"""The four-launch stage of small grids (N <= 128): every grid size and both forms, from a state
with content outside the truncation sphere (the first stage then runs on every pencil, the
later ones on those inside), against the oracle; pruned and unpruned runs agree bit for bit."""
import numpy as np
import pytest

from oracle.ref_r2c import TaylorGreenR2C, full_to_half, half_to_full
from spectral_solver_b200 import Solver

pytestmark = pytest.mark.gpu

NU, DT, STEPS = 1.0 / 400.0, 1e-3, 4


def unmasked_state(n):
    """A Hermitian spectrum with content at every |m| < N/2 on each axis (corners included)."""
    rng = np.random.default_rng(n)
    m = np.fft.fftfreq(n, 1.0 / n)
    kz, ky, kx = np.meshgrid(m, m, m, indexing="ij")
    decay = 0.3 / (1.0 + kx ** 2 + ky ** 2 + kz ** 2)
    inside = (abs(kx) < n / 2) & (abs(ky) < n / 2) & (abs(kz) < n / 2)
    return [np.fft.fftn(rng.standard_normal((n, n, n))) * decay * inside for _ in range(3)]


@pytest.mark.parametrize("n", [8, 12, 16, 24, 32, 48, 64, 96, 128])
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("viscous_mode", [0, 1])
def test_steps_from_an_unmasked_state(n, precision, viscous_mode):
    if viscous_mode and n not in (24, 64):
        pytest.skip("the viscous factor is the sweep's: two sizes cover it")
    full = unmasked_state(n)
    states = []
    for prune in (True, False):
        with Solver(n, nu=NU, precision=precision, viscous_mode=viscous_mode) as s:
            s.set_sphere_pruning(prune)
            s.set_state(full)
            s.step(DT, STEPS)
            states.append(s.get_state())
            vmax = s.max_velocity()
    o = TaylorGreenR2C(n, 1.0 / NU, u_hat0=[full_to_half(c) for c in full], integrating_factor=bool(viscous_mode))
    for _ in range(STEPS):
        o.step(DT)
    ref = [half_to_full(c) for c in o.u_hat]
    num = sum(float(np.sum(np.abs(a - b) ** 2)) for a, b in zip(states[0], ref))
    den = sum(float(np.sum(np.abs(b) ** 2)) for b in ref)
    # the parity tests' bounds: FP64 round-off of a trajectory; FP32 round-off of the state
    assert (num / den) ** 0.5 < (1e-6 if precision else 1e-12)
    assert all(np.array_equal(a, b) for a, b in zip(*states))
    assert abs(vmax - o.max_velocity()) < (2e-6 if precision else 1e-12) * vmax
