"""The unprojected nonlinear term (sns_nonlinear, all six products) on the fused passes: small grids
and the oracle; on large grids the two-stage x pass and the fused forward z + sweep against the
generic one-row x pass and the separate sweep, which a launch shape selects."""
import numpy as np
import pytest

from oracle.ref_r2c import TaylorGreenR2C, full_to_half, half_to_full
from spectral_solver_b200 import Solver

pytestmark = pytest.mark.gpu

# round-off of two transform chains in the form's precision (the right-hand side's parity bounds)
BOUND = (1e-12, 2e-5)


def unmasked_state(n):
    """A Hermitian spectrum with content at every |m| < N/2 on each axis (corners included)."""
    rng = np.random.default_rng(n)
    m = np.fft.fftfreq(n, 1.0 / n)
    kz, ky, kx = np.meshgrid(m, m, m, indexing="ij", sparse=True)
    weight = 0.3 / (1.0 + kx ** 2 + ky ** 2 + kz ** 2)
    weight = weight * ((abs(kx) < n / 2) & (abs(ky) < n / 2) & (abs(kz) < n / 2))
    return [np.fft.fftn(rng.standard_normal((n, n, n))) * weight for _ in range(3)]


def outside(n):
    m = np.fft.fftfreq(n, 1.0 / n)
    kz, ky, kx = np.meshgrid(m, m, m, indexing="ij", sparse=True)
    return 4 * (kx ** 2 + ky ** 2 + kz ** 2) > n * n


def rel_l2(a, b):
    num = sum(float(np.sum(np.abs(x - y) ** 2)) for x, y in zip(a, b))
    den = sum(float(np.sum(np.abs(y) ** 2)) for y in b)
    return (num / den) ** 0.5


@pytest.mark.parametrize("n", [8, 12, 24, 48, 96, 128])
@pytest.mark.parametrize("precision", [0, 1])
def test_small_grids_match_the_oracle(n, precision):
    u = unmasked_state(n)
    o = TaylorGreenR2C(n, 400.0)
    ref = [half_to_full(c) for c in o.nonlinear([full_to_half(c) for c in u])]
    with Solver(n, 400.0, precision=precision) as s:
        s.step(1e-3, 3)  # work fields hold something, outside the sphere too
        got = s.nonlinear(u)
    assert rel_l2(got, ref) < BOUND[precision]
    assert not any(np.any(c[outside(n)]) for c in got)


@pytest.mark.parametrize("n,precision", [(256, 0), (256, 1), (512, 0), (512, 1)])
def test_large_grids_match_the_generic_passes(n, precision, tmp_path):
    cache, generic = str(tmp_path / "shapes.txt"), str(tmp_path / "generic.txt")
    with Solver(n, 400.0, seed=3, pert_amp=0.1, pert_kmax=n // 3, precision=precision) as s:
        assert s.launch_config()["xpass_grid"] > 0 and s.launch_config()["p5_grid"] > 0
        u = unmasked_state(n) if n == 256 else s.get_state()
        got = s.nonlinear(u)
        s.autotune(1, cache)
    words = open(cache).read().split()
    with open(generic, "w") as f:
        f.write(" ".join(words[:5] + ["0", "0"]) + "\n")  # name, N, precision, y/z grid, x pass, forward z + sweep
    with Solver(n, 400.0, precision=precision) as s:
        assert s.autotune(1, generic)["xpass_grid"] == 0 and s.launch_config()["p5_grid"] == 0
        ref = s.nonlinear(u)
    assert rel_l2(got, ref) < BOUND[precision]
    out = outside(n)
    assert not any(np.any(c[out]) for c in got)
