"""Which kernel a call runs in (GPU), where a rule on sizes had sent it the slower way
by a factor of 1.2 to 4: from the library's profile, sizes as measured beside the
rules (gemm_direct.cu, trsm.cu)."""
import ctypes
import json

import pytest

import mublis_b200 as mb

pytestmark = pytest.mark.gpu


def kernels(lib, call, *args):
    import torch
    buf = ctypes.create_string_buffer(1 << 16)
    torch.cuda.synchronize()
    lib.mublis_b200_profile_read(buf, len(buf))
    lib.mublis_b200_profile_enable(1)
    st = getattr(lib, call)(*args)
    lib.mublis_b200_profile_enable(0)
    lib.mublis_b200_profile_read(buf, len(buf))
    assert st == 0, mb.last_error(lib)
    return set(json.loads(buf.value.decode()))


@pytest.fixture(scope="module", autouse=True)
def plain_forms(lib):
    assert lib.mublis_b200_init() == 0, mb.last_error(lib)
    lib.mublis_b200_set_form(b"s", b"plain")
    lib.mublis_b200_set_form(b"d", b"plain")


def zeros(p, rows, cols):
    torch = pytest.importorskip("torch")
    return torch.zeros(cols, rows, dtype=torch.float32 if p == "s" else torch.float64, device="cuda")


def ptr(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("p,m,n,kernel", [("s", 256, 40000, "ffma_sgemm"), ("s", 512, 10000, "ffma_sgemm"),
                                          ("s", 128, 40000, "ffma_sgemm"), ("s", 700, 3000, "ffma_sgemm"),
                                          ("s", 200, 300, "direct_sgemm"), ("d", 128, 40000, "dmma_dgemm"),
                                          ("d", 300, 300, "direct_dgemm")])
def test_trmm(lib, p, m, n, kernel):
    a, b = zeros(p, m, m), zeros(p, m, n)
    assert kernel in kernels(lib, f"mublis_{p}trmm", 0, mb.M_LOWER, 0, 0, m, n, 1.0, ptr(a), 1, m, ptr(b), 1, m)


@pytest.mark.parametrize("p,m,n,k,kernel", [
    ("s", 64, 64, 65536, "direct_sgemm"), ("s", 64, 64, 131072, "direct_sgemm"),
    ("d", 64, 64, 65536, "direct_dgemm"), ("d", 16, 16, 100000, "direct_dgemm"),
    ("s", 512, 512, 8192, "ffma_sgemm"), ("s", 1043, 3956, 355, "ffma_sgemm"),
    ("s", 64, 64, 64, "direct_sgemm"), ("d", 301, 177, 211, "direct_dgemm")])
def test_gemm(lib, p, m, n, k, kernel):
    a, b, c = zeros(p, m, k), zeros(p, k, n), zeros(p, m, n)
    assert kernel in kernels(lib, f"mublis_{p}gemm", 0, 0, m, n, k, 1.0, ptr(a), 1, m, ptr(b), 1, k, 0.0,
                             ptr(c), 1, m)


@pytest.mark.parametrize("p,m,n,kernel", [
    ("s", 256, 40000, "trsm_leaf_s"), ("s", 256, 80000, "trsm_inv_s"), ("s", 192, 5000, "trsm_leaf_s"),
    ("s", 144, 4700, "small_strsm"), ("s", 256, 4700, "small_strsm"), ("s", 128, 40000, "small_strsm"), ("s", 256, 100, "small_strsm"),
    ("s", 1024, 5000, "trsm_leaf_s"), ("s", 1024, 40000, "trsm_inv_s"), ("s", 512, 28000, "trsm_leaf_s"),
    ("d", 256, 40000, "small_dtrsm"), ("d", 512, 40000, "trsm_leaf_d")])
def test_trsm(lib, p, m, n, kernel):
    import torch
    a, b = zeros(p, m, m), zeros(p, m, n)
    a += torch.eye(m, dtype=a.dtype, device="cuda")
    assert kernel in kernels(lib, f"mublis_{p}trsm", 0, mb.M_LOWER, 0, 0, m, n, 1.0, ptr(a), 1, m, ptr(b), 1, m)
