"""bench.py's figures of the bytes that a step moves: the per-pass bytes of three stages are the
per-step figure, and the roofline's fixed model is the six-product one with nothing pruned."""
import pytest

import bench

STAGE = ("p1_zinv_phase", "p2_yinv", "p3_xpass", "p3_nyq", "p4_yfwd", "p5_sweep")


@pytest.mark.parametrize("n", [256, 512])
@pytest.mark.parametrize("w", [8, 4])
def test_passes_add_up_to_the_step(n, w):
    b, live = bench.moved_pass_bytes(n, w)
    assert 3 * sum(b[p] for p in STAGE) == pytest.approx(bench.moved_step_bytes_s(live), rel=1e-12)
    assert all(b[p] <= bench.PASS_BYTES_S[p] for p in STAGE)
    assert bench.moved_step_bytes_s(1.0) == 3 * sum(bench.PASS_BYTES_S[p] for p in STAGE)


def test_the_fixed_model():
    # g counted as read in every stage: one S more per stage than the mean of three
    assert bench.MODEL_BYTES_S == bench.step_bytes_s(1.0) == 3 * (sum(bench.MODEL_PASS_BYTES_S[p] for p in STAGE) + 1)
