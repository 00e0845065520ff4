"""Steps from a state with content outside the truncation sphere (the first stage runs on every
pencil, the later ones on those inside): the rotational form on every small grid against the
oracle, and both forms on a large grid, pruned and unpruned bit for bit."""
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
    kz, ky, kx = np.meshgrid(m, m, m, indexing="ij", sparse=True)
    weight = 0.3 / (1.0 + kx ** 2 + ky ** 2 + kz ** 2)
    weight = weight * ((abs(kx) < n / 2) & (abs(ky) < n / 2) & (abs(kz) < n / 2))
    return [np.fft.fftn(rng.standard_normal((n, n, n))) * weight for _ in range(3)]


def pruned_and_full(n, precision, form, full):
    states = []
    for prune in (True, False):
        with Solver(n, nu=NU, precision=precision) as s:
            s.set_nonlinear_form(form)
            s.set_sphere_pruning(prune)
            s.set_state(full)
            s.step(DT, STEPS)
            states.append(s.get_state())
    assert all(np.array_equal(a, b) for a, b in zip(*states))
    return states[0]


@pytest.mark.parametrize("n", [8, 12, 16, 24, 32, 48, 64, 96, 128])
@pytest.mark.parametrize("precision", [0, 1])
def test_rotational_small_grids(n, precision):
    full = unmasked_state(n)
    got = pruned_and_full(n, precision, 1, full)
    o = TaylorGreenR2C(n, 1.0 / NU, u_hat0=[full_to_half(c) for c in full], rotational=True)
    for _ in range(STEPS):
        o.step(DT)
    ref = [half_to_full(c) for c in o.u_hat]
    num = sum(float(np.sum(np.abs(a - b) ** 2)) for a, b in zip(got, ref))
    den = sum(float(np.sum(np.abs(b) ** 2)) for b in ref)
    # the parity tests' bounds: FP64 round-off of a trajectory; FP32 round-off of the state
    assert (num / den) ** 0.5 < (1e-6 if precision else 1e-12)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("form", [0, 1])
def test_large_grid(precision, form):
    pruned_and_full(256, precision, form, unmasked_state(256))
