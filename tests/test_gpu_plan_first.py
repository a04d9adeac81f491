"""A plan as the first work of a process (GPU): its kernels' code and host
memory are set up before the stream capture, which would not survive them."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = r"""
import ctypes, sys
import torch
sys.path.insert(0, sys.argv[1])
import mublis_b200 as mb
lib = mb.load()
mb.check(lib.mublis_b200_init(), lib)
kind, dtype, form = sys.argv[2], sys.argv[3], sys.argv[4]
mb.check(lib.mublis_b200_set_form(dtype.encode(), form.encode()), lib)
dt = torch.float32 if dtype == "s" else torch.float64
a = torch.eye(48, dtype=dt, device="cuda")
b = torch.rand(32, 48, dtype=dt, device="cuda")
c = torch.zeros(32, 48, dtype=dt, device="cuda")
torch.cuda.synchronize()
plan = ctypes.c_void_p()
if kind == "gemm":
    arr = (mb.GemmProblem * 1)(mb.GemmProblem(0, 0, 48, 32, 48, 1.0, 0.0, a.data_ptr(), 48,
                                              b.data_ptr(), 48, c.data_ptr(), 48))
    mb.check(lib.mublis_b200_plan_gemm_grouped(dtype.encode(), arr, 1, ctypes.byref(plan)), lib)
else:
    c.copy_(b)
    torch.cuda.synchronize()
    arr = (mb.TrsmProblem * 1)(mb.TrsmProblem(mb.M_LOWER, 0, mb.M_NON_UNIT, 48, 32, 1.0,
                                              a.data_ptr(), 48, c.data_ptr(), 48))
    mb.check(lib.mublis_b200_plan_trsm_grouped(dtype.encode(), arr, 1, ctypes.byref(plan)), lib)
mb.check(lib.mublis_b200_plan_run(plan), lib)
assert float((c - b).abs().max()) <= 1e-6, "I b = b"
"""


@pytest.mark.parametrize("kind,dtype,form", [("gemm", "s", "fp16x3"), ("gemm", "d", "plain"),
                                             ("trsm", "s", "plain")])
def test_plan_is_the_first_work(kind, dtype, form):
    from tests.conftest import ROOT
    subprocess.run([sys.executable, "-c", CHILD, str(ROOT), kind, dtype, form], check=True,
                   timeout=300)
