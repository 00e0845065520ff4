"""The projected right-hand side runs on five products (u_2^2 subtracted from the diagonal
ones), the unprojected nonlinear term on all six: the two agree after the projection."""
import numpy as np
import pytest

from spectral_solver_b200 import Solver

pytestmark = pytest.mark.gpu


def modes(n):
    m = np.arange(n)
    m = np.where(m <= n // 2, m, m - n).astype(np.float64)
    return m.reshape(1, 1, n), m.reshape(1, n, 1), m.reshape(n, 1, 1)


# 8: the smallest grid; 48, 96: generic x pass; 128, 256: the fused x and z passes of either form
@pytest.mark.parametrize("n", [8, 48, 96, 128, 256])
@pytest.mark.parametrize("precision", [0, 1])
def test_rhs_is_the_projected_nonlinear_term(n, precision):
    nu = 1.0 / 400.0
    with Solver(n, nu=nu, seed=3, pert_amp=0.1, pert_kmax=max(1, n // 4), precision=precision) as s:
        u = s.get_state()
        r = s.rhs(u)
        w = s.nonlinear(u)
    kx, ky, kz = modes(n)
    k2 = kx * kx + ky * ky + kz * kz
    keep = (4 * k2 <= n * n) & (k2 > 0)
    w = [a - nu * k2 * b for a, b in zip(w, u)]
    dot = (kx * w[0] + ky * w[1] + kz * w[2]) / np.where(k2 > 0, k2, 1.0)
    ref = [np.where(keep, a - k * dot, 0.0) for a, k in zip(w, (kx, ky, kz))]
    # the stored half only: the reference's full layout mirrors it
    h = n // 2 + 1
    num = sum(float(np.sum(np.abs(a[..., :h] - b[..., :h]) ** 2)) for a, b in zip(r, ref))
    den = sum(float(np.sum(np.abs(b[..., :h]) ** 2)) for b in ref)
    # round-off of two transforms chains in the form's precision (the right-hand side bounds
    # of the parity tests: 1e-12 and 2e-5)
    assert (num / den) ** 0.5 < (2e-5 if precision else 1e-12)
