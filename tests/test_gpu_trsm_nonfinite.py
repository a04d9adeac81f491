"""Triangular solves with a non-finite right-hand side (GPU): an Inf or NaN in row j
of one column belongs to that column's rows from j on (in the order of the solve).
The rows before it, and every other column, keep the bits they have without it; NaN
fills the rest, and so does Inf or NaN for an Inf.  The one-launch kernel (single and
grouped, orders up to 256) substitutes, so there Inf and NaN fall as they do row by
row; the leaf kernel (larger orders) applies inverted 16 x 16 blocks."""
import ctypes

import numpy as np
import pytest

import mublis_b200 as mb
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
DT = {"s": np.float32, "d": np.float64}
RHS = 40


@pytest.fixture(scope="module", autouse=True)
def plain_forms(lib):
    assert lib.mublis_b200_init() == 0, mb.last_error(lib)
    lib.mublis_b200_set_form(b"s", b"plain")
    lib.mublis_b200_set_form(b"d", b"plain")


def solve(lib, p, grouped, uplo, a, b):
    """inv(A) B for column-major arrays, on the device."""
    import torch
    order, rhs = b.shape
    da, db = torch.from_numpy(a.T.copy()).cuda(), torch.from_numpy(b.T.copy()).cuda()
    torch.cuda.synchronize()
    if grouped:
        probs = (mb.TrsmProblem * 1)(mb.TrsmProblem(uplo, 0, mb.M_NON_UNIT, order, rhs, 1.0,
                                                    da.data_ptr(), order, db.data_ptr(), order))
        st = lib.mublis_b200_trsm_grouped(p.encode(), probs, 1)
    else:
        st = getattr(lib, f"mublis_{p}trsm")(0, uplo, 0, mb.M_NON_UNIT, order, rhs, 1.0,
                                             ctypes.c_void_p(da.data_ptr()), 1, order,
                                             ctypes.c_void_p(db.data_ptr()), 1, order)
    assert st == 0, mb.last_error(lib)
    return db.cpu().numpy().T


def by_rows(a, b, lower):
    """inv(A) b of one column, row by row."""
    x = b.astype(np.float64)
    n = len(x)
    for i in range(n) if lower else range(n - 1, -1, -1):
        for q in range(i) if lower else range(i + 1, n):
            x[i] -= a[i, q] * x[q]
        x[i] /= a[i, i]
    return x


@pytest.mark.parametrize("p", ["s", "d"])
@pytest.mark.parametrize("lower", [True, False], ids=["lower", "upper"])
@pytest.mark.parametrize("order,grouped", [(48, True), (48, False), (200, True), (200, False),
                                           (600, False)])
def test_nonfinite_rhs_reaches_only_later_rows(lib, p, lower, order, grouped):
    pytest.importorskip("torch")
    a = orc.trsm_matrix(order, DT[p], 31, 0)
    b = orc.fill(order, RHS, DT[p], 31, 1)
    uplo = mb.M_LOWER if lower else mb.M_UPPER
    clean = solve(lib, p, grouped, uplo, a, b)
    assert np.isfinite(clean).all()
    last = order - 1
    bad = [(3, 0, np.nan), (5, 7, np.inf), (15, 8, -np.inf), (16, 9, np.inf), (21, 33, np.nan),
           (last - 2, 39, np.inf), (last, 38, np.nan)]  # (row in the order of the solve, column)
    dirty = b.copy(order="F")
    for j, col, v in bad:
        dirty[j if lower else last - j, col] = v
    out = solve(lib, p, grouped, uplo, a, dirty)
    ran = out if lower else out[::-1]
    want = clean if lower else clean[::-1]
    spoilt = {col: j for j, col, _ in bad}
    for col in range(RHS):
        j = spoilt.get(col, order)
        np.testing.assert_array_equal(ran[:j, col], want[:j, col], err_msg=f"column {col}")
        assert not np.isfinite(ran[j:, col]).any(), col
    for j, col, v in bad:
        if np.isnan(v):
            assert np.isnan(ran[j:, col]).all(), col
        elif order <= 256:
            with np.errstate(invalid="ignore"):
                ref = by_rows(a.astype(np.float64), dirty[:, col], lower)
            np.testing.assert_array_equal(np.isnan(out[:, col]), np.isnan(ref))
