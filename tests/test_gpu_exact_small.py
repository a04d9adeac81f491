"""The one-launch kernels and the solves on integers (GPU): every sum is exact, so the
result must equal the integers it was made from, element by element, and a lost k
tail, block or update is a wrong integer.

* Products of gemm_direct.cu (operands in {-2 .. 2}) around its 32 and 64 tiles, its
  16- and 32-deep k-blocks and its k splits.
* Solves A X = alpha B with B made from X.  A is unit triangular with entries in
  {-1, 0, 1} from rows r % 16 in 0 .. 4 to 5 .. 10, from those to 11 .. 15, and from the
  first to the last: every 16 x 16 block has some, each step depends on solved rows, and
  the inverse stays below 2^11, so FP32 is exact in every method (substituted, inverted
  blocks, inverted leaves).
"""
import ctypes

import numpy as np
import pytest

import mublis_b200 as mb
from tests import test_gpu_large_kernels as large

pytestmark = pytest.mark.gpu
DT = large.DT
DIRECT = {"s": "direct_sgemm", "d": "direct_dgemm"}


@pytest.fixture(scope="module", autouse=True)
def plain_forms(lib):
    assert lib.mublis_b200_init() == 0, mb.last_error(lib)
    lib.mublis_b200_set_form(b"s", b"plain")
    lib.mublis_b200_set_form(b"d", b"plain")


@pytest.mark.parametrize("p", ["s", "d"])
@pytest.mark.parametrize("ta,tb", large.TRANS)
@pytest.mark.parametrize("pads", [(0, 0, 0), (1, 1, 1)])
@pytest.mark.parametrize("mnk", [(1, 1, 1), (31, 33, 17), (32, 64, 16), (65, 63, 33), (20, 24, 2049),
                                 (64, 64, 4097), (333, 40, 5), (515, 771, 261), (700, 400, 1031)])
def test_direct_gemm(lib, p, ta, tb, pads, mnk):
    large.gemm(lib, p, *mnk, ta, tb, pads, kernel=DIRECT)


@pytest.mark.parametrize("p", ["s", "d"])
@pytest.mark.parametrize("uplo", [mb.M_LOWER, mb.M_UPPER])
@pytest.mark.parametrize("trans", [False, True])
@pytest.mark.parametrize("routine,n,k,pad", [("syrk", 33, 300, 0), ("syrk", 129, 2049, 1),
                                             ("syr2k", 70, 17, 0), ("syr2k", 129, 1030, 0)])
def test_direct_rank(lib, p, uplo, trans, routine, n, k, pad):
    large.rank(lib, p, routine, n, k, uplo, trans, pad, kernel=DIRECT)


@pytest.mark.parametrize("p", ["s", "d"])
@pytest.mark.parametrize("right,uplo,trans", [(False, mb.M_LOWER, False), (False, mb.M_UPPER, True),
                                              (True, mb.M_LOWER, True), (True, mb.M_UPPER, False)])
@pytest.mark.parametrize("m,n,pad", [(1, 1, 0), (31, 65, 1), (130, 97, 0), (257, 260, 1)])
def test_direct_trmm(lib, p, right, uplo, trans, m, n, pad):
    large.trmm(lib, p, right, uplo, trans, m, n, pad, kernel=DIRECT)


def unit_triangle(order, lower, seed):
    rng = np.random.default_rng(seed)
    a = rng.integers(-1, 2, (order, order))
    step = np.array([0] * 5 + [1] * 6 + [2] * 5)[np.arange(order) % 16]
    at = np.arange(order)
    before = (at[None, :] < at[:, None]) if lower else (at[None, :] > at[:, None])
    return np.where(before & (step[None, :] < step[:, None]), a, 0)


SIZES = [(o, n) for o in (1, 15, 16, 17, 128, 129, 255, 256) for n in (1, 33)] + [
    (257, 7), (272, 9), (512, 33), (513, 15), (530, 1185), (1023, 8), (2049, 33), (2049, 513)]


@pytest.mark.parametrize("p", ["s", "d"])
@pytest.mark.parametrize("right,lower,trans", [(False, True, False), (False, False, True),
                                               (True, True, False), (True, False, False)])
@pytest.mark.parametrize("order,rhs", SIZES)
def test_solve(lib, p, right, lower, trans, order, rhs):
    import torch
    acts_lower = lower != trans
    t = unit_triangle(order, acts_lower, order + rhs)  # op(A) without its diagonal
    x = np.random.default_rng(rhs).integers(-2, 3, (rhs, order) if right else (order, rhs))
    b = -2 * (x + x @ t if right else x + t @ x)  # alpha = -1/2
    a = (t.T if trans else t).astype(DT[p])
    unread = ~(np.tri(order, k=-1, dtype=bool) if lower else np.tri(order, k=-1, dtype=bool).T)
    a[unread] = np.nan
    m, n = b.shape
    da, db = (torch.from_numpy(np.ascontiguousarray(v.T.astype(DT[p]))).cuda() for v in (a, b))
    torch.cuda.synchronize()
    assert getattr(lib, f"mublis_{p}trsm")(
        int(right), mb.M_LOWER if lower else mb.M_UPPER, int(trans), mb.M_UNIT, m, n, -0.5,
        ctypes.c_void_p(da.data_ptr()), 1, order, ctypes.c_void_p(db.data_ptr()), 1, m) == 0, \
        mb.last_error(lib)
    np.testing.assert_array_equal(db.cpu().numpy().T, x)


@pytest.mark.parametrize("p", ["s", "d"])
def test_grouped_solve(lib, p):
    import torch
    keep, probs, want = [], [], []
    for i, (order, rhs) in enumerate(s for s in SIZES if s[0] <= 256):
        lower = i % 3 != 0
        t = unit_triangle(order, lower, i)
        x = np.random.default_rng(i).integers(-2, 3, (order, rhs))
        keep.append([torch.from_numpy(np.ascontiguousarray(v.T.astype(DT[p]))).cuda()
                     for v in (t, -2 * (x + t @ x))])
        probs.append(mb.TrsmProblem(mb.M_LOWER if lower else mb.M_UPPER, 0, mb.M_UNIT, order, rhs, -0.5,
                                    keep[-1][0].data_ptr(), order, keep[-1][1].data_ptr(), order))
        want.append(x)
    torch.cuda.synchronize()
    arr = (mb.TrsmProblem * len(probs))(*probs)
    assert lib.mublis_b200_trsm_grouped(p.encode(), arr, len(probs)) == 0, mb.last_error(lib)
    for (_, b), x in zip(keep, want):
        np.testing.assert_array_equal(b.cpu().numpy().T, x)


def test_small_solve_rounds_alpha_b_minus_the_update_once(lib):
    """FP32, A = I with a one below the first block: x[16] = alpha b[16] - x[0]."""
    import torch
    order, rhs, alpha = 17, 512, np.float32(0.7)
    rng = np.random.default_rng(5)
    a = np.eye(order, dtype=np.float32)
    a[16, 0] = 1
    b = rng.uniform(0.5, 1, (order, rhs)).astype(np.float32)
    da, db = torch.from_numpy(a.T.copy()).cuda(), torch.from_numpy(b.T.copy()).cuda()
    torch.cuda.synchronize()
    assert lib.mublis_strsm(0, mb.M_LOWER, 0, mb.M_NON_UNIT, order, rhs, float(alpha),
                            ctypes.c_void_p(da.data_ptr()), 1, order,
                            ctypes.c_void_p(db.data_ptr()), 1, order) == 0, mb.last_error(lib)
    x = db.cpu().numpy().T
    np.testing.assert_array_equal(x[:16], alpha * b[:16])
    once = (np.float64(alpha) * b[16] - x[0].astype(np.float64)).astype(np.float32)
    np.testing.assert_array_equal(x[16], once)
