"""The two-launch forward transform on device buffers at every size it serves, against numpy:
the mirrored half, the self-mirrored columns 0 and N/2 included."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 12, 16, 24, 32, 48, 64])
def test_matches_numpy(lib, n):
    import torch
    x = np.random.default_rng(n).standard_normal((n, n, n))
    d_in = torch.from_numpy(x).cuda()
    d_out = torch.full((n, n, n), float("nan"), dtype=torch.complex128, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    assert lib.sns_forward_r2c_noalloc(n, C.c_void_p(d_in.data_ptr()), C.c_void_p(d_out.data_ptr()),
                                       C.c_void_p(stream)) == 0
    ref = np.fft.fftn(x)
    # the transform tests' bound
    assert np.max(np.abs(d_out.cpu().numpy() - ref)) <= 1e-12 * np.max(np.abs(ref))
