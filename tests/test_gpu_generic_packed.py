"""The packed transforms of the generic-shape solver: two real fields to a complex transform, read
through the Hermitian parts of any input and taken apart at the mirror mode.  Shapes cover every
radix (2 .. 8, 12, 16, primes above 7), one, two and three stages, odd axes (no Nyquist index),
axes of length 2 (the only mode pair is 0 and Nyquist) and partial tiles; the states are
arbitrary complex arrays, as the reference's transforms accept them."""
import numpy as np
import pytest

from oracle.legacy import LegacyNS

pytestmark = pytest.mark.gpu

SHAPES = [(2, 2, 2), (3, 2, 5), (16, 12, 7), (45, 33, 14), (72, 17, 10), (13, 64, 9), (30, 22, 96), (26, 6, 80)]


def rel_l2(a, b):
    num = sum(float(np.sum(np.abs(x - y) ** 2)) for x, y in zip(a, b))
    den = sum(float(np.sum(np.abs(y) ** 2)) for y in b)
    return np.sqrt(num / den)


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("dealias", [True, False])
def test_any_state_any_shape(shape, dealias):
    from spectral_solver_b200 import Fft3D
    lengths, nu, dt = (1.7, 3.1, 2.3), 0.01, 1e-4
    o = LegacyNS(shape, lengths, nu, dealias=dealias)
    rng = np.random.default_rng(sum(shape))
    zyx = shape[::-1]
    u = [rng.standard_normal(zyx) + 1j * rng.standard_normal(zyx) for _ in range(3)]
    with Fft3D(shape, lengths) as f:
        # FP64 round-off of the transforms: the bound of the generic path's other tests
        if any(np.abs(r).max() > 0 for r in o.nonlinear_rhs(u)):
            assert rel_l2(f.rhs(u, nu, dealias, full=False), o.nonlinear_rhs(u)) <= 1e-12
        ref = o.rhs(u)
        if any(np.abs(r).max() > 0 for r in ref):
            assert rel_l2(f.rhs(u, nu, dealias, full=True), ref) <= 1e-12
        want = o.step_rk3(o.step_rk3(u, dt), dt)
        got = f.step(u, nu, dt, 2, dealias)
        scale = max(float(np.abs(w).max()) for w in want)
        assert max(float(np.abs(a - b).max()) for a, b in zip(got, want)) <= 1e-12 * scale
        p, q = f.product(u[0], u[2]), o.product_dealiased(u[0], u[2])
        assert np.abs(p - q).max() <= 1e-12 * np.abs(q).max()
