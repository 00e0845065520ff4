"""The index-checked build on what the bounds test of the conservative steps does not run: every
small grid, the rotational form, device CFL steps, sns_nonlinear, the allocation-free forward
transform, and large grids from a state with content outside the sphere."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = r"""
import ctypes as C, json, sys
import numpy as np
import torch
sys.path.insert(0, sys.argv[1])
from spectral_solver_b200 import _lib, Solver
lib = _lib.load()
assert lib._name.endswith("libsns_b200_check.so"), lib._name
out = {}
for n in (8, 12, 16, 24, 32, 48, 64, 96, 128, 256):
    for prec in (0, 1):
        with Solver(n, 400.0, seed=1, pert_amp=1e-2, pert_kmax=max(1, n // 4), precision=prec) as s:
            s.set_clock(0.0, cfl=0.2, dt_max=1e-3)
            u = s.get_state()
            rng = np.random.default_rng(n)
            u = [c + 1e-4 * np.fft.fftn(rng.standard_normal((n, n, n))) for c in u]  # outside the sphere too
            for form in (0, 1):
                s.set_nonlinear_form(form)
                s.step(1e-3, 2)
                s.step_cfl(2)
                s.rhs(u)
                s.nonlinear(u)
                s.set_state(u)
                s.step_cfl(1)
                s.step(1e-3, 4)
            s.set_nonlinear_form(0)
            s.step(1e-3, 1)
            d = s.diagnostics()
            out[f"E_{n}_{prec}"] = d["kinetic_energy"] if np.isfinite(d["max_velocity"]) else float("nan")
    if n <= 64:
        phys = torch.randn(n, n, n, dtype=torch.float64, device="cuda")
        spec = torch.empty(n, n, n, dtype=torch.complex128, device="cuda")
        torch.cuda.synchronize()
        assert lib.sns_forward_r2c_noalloc(n, phys.data_ptr(), spec.data_ptr(), None) == 0
        err = (spec - torch.fft.fftn(phys)).abs().max() / spec.abs().max()
        out[f"forward_{n}"] = float(err)
cnt, line, idx = C.c_longlong(), C.c_int(), C.c_longlong()
assert lib.sns_debug_bounds(C.byref(cnt), C.byref(line), C.byref(idx)) == 0
out.update(count=cnt.value, line=line.value, index=idx.value)
print(json.dumps(out))
"""


def test_no_index_leaves_its_buffer():
    env = dict(os.environ, SNS_B200_LIB="check")
    r = subprocess.run([sys.executable, "-c", SCRIPT, ROOT], capture_output=True, text=True, timeout=900, env=env,
                       cwd=ROOT)
    assert r.returncode == 0, r.stderr[-3000:]
    res = json.loads(r.stdout.strip().splitlines()[-1])
    assert res["count"] == 0, res
    assert all(0.1 < v < 0.2 for k, v in res.items() if k.startswith("E_")), res
    assert all(v < 1e-12 for k, v in res.items() if k.startswith("forward_")), res
