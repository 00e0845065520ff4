"""The generic-shape nonlinear term keeps each component's own accuracy: a velocity component far
smaller than the others (a perturbation of a planar flow), or zero, gets its term to round-off of
that term, with and without the phase-shift pair."""
import numpy as np
import pytest

from oracle.legacy import LegacyNS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(24, 20, 18), (13, 16, 9)])
@pytest.mark.parametrize("dealias", [True, False])
@pytest.mark.parametrize("component", [0, 1, 2])
@pytest.mark.parametrize("size", [1e-9, 0.0])
def test_a_small_component(shape, dealias, component, size):
    from spectral_solver_b200 import Fft3D
    lengths = (1.7, 3.1, 2.3)
    rng = np.random.default_rng(sum(shape) + component)
    u = [np.fft.fftn(rng.standard_normal(shape[::-1])) for _ in range(3)]
    u[component] *= size
    ref = LegacyNS(shape, lengths, 0.01, dealias=dealias).nonlinear_rhs(u)[component]
    with Fft3D(shape, lengths) as f:
        got = f.rhs(u, 0.01, dealias, full=False)[component]
    if size == 0.0:
        assert not np.any(got)
    else:  # FP64 round-off of the transforms: the bound of the generic path's other tests
        assert np.linalg.norm(got - ref) <= 1e-12 * np.linalg.norm(ref)
