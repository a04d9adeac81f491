"""The allocation-free SGEMM as the first product of a process (GPU): what its kernel
needs is claimed when the library starts, so the call maps no memory of the driver's,
neither the device's nor pinned host memory."""
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
n = 256
a = torch.eye(n, device="cuda")
b = torch.arange(n * n, dtype=torch.float32, device="cuda").reshape(n, n)
c = torch.zeros(n, n, device="cuda")
stream = torch.cuda.Stream()
mb.check(lib.mublis_b200_set_stream(stream.cuda_stream), lib)
torch.cuda.synchronize()
def state():
    with open("/proc/self/maps") as f:
        maps = sorted(line.split()[0] for line in f if "rw-s" in line)  # pinned or the driver's
    return maps, torch.cuda.mem_get_info()[0]
state()
before = state()
st = lib.mublis_b200_sgemm_noalloc(0, 0, n, n, n, 1.0, a.data_ptr(), 1, n, b.data_ptr(), 1, n, 0.0,
                                   c.data_ptr(), 1, n)
after = state()
mb.check(st, lib)
assert torch.equal(c, b)
assert after[1] == before[1], "device memory"
assert after[0] == before[0], sorted(set(after[0]) ^ set(before[0]))
"""


def test_first_call_maps_nothing():
    from tests.conftest import ROOT
    subprocess.run([sys.executable, "-c", CHILD, str(ROOT)], check=True, timeout=300)
