"""Small triangular solves are backward stable (GPU): every element of B - A X is within
2 (order + 4) u of |A| |X|, as for a substitution against the reciprocal diagonal
(order products and sums, the reciprocal's and its product's rounding; the factor 2 is
margin), whatever the triangle's condition.  Grouped calls and single ones up to the
one-launch kernel's order."""
import ctypes

import numpy as np
import pytest

import mublis_b200 as mb

pytestmark = pytest.mark.gpu
DT = {"s": np.float32, "d": np.float64}


def triangle(kind, n, rng):
    a = np.tril(rng.uniform(-1, 1, (n, n)), -1)
    if kind == "small diagonal":
        return a + np.diag(rng.uniform(0.05, 1, n))
    if kind == "unit":
        return a + np.eye(n)
    scale = np.logspace(0, -4, n)
    return (a + np.eye(n)) * (scale[:, None] if kind == "graded rows" else scale[None, :])


@pytest.mark.parametrize("p", ["s", "d"])
@pytest.mark.parametrize("kind", ["small diagonal", "unit", "graded rows", "graded columns"])
@pytest.mark.parametrize("n", [16, 30, 64, 128, 200])
@pytest.mark.parametrize("grouped", [True, False])
def test_small_solves_are_backward_stable(lib, p, kind, n, grouped):
    torch = pytest.importorskip("torch")
    assert lib.mublis_b200_init() == 0, mb.last_error(lib)
    lib.mublis_b200_set_form(p.encode(), b"plain")
    rng, dt, rhs = np.random.default_rng(n), DT[p], 50
    a = triangle(kind, n, rng).astype(dt)
    wide = a.astype(np.longdouble)
    b = (wide @ rng.uniform(-1, 1, (n, rhs))).astype(dt)
    da, db = torch.from_numpy(a.T.copy()).cuda(), torch.from_numpy(b.T.copy()).cuda()
    torch.cuda.synchronize()
    if grouped:
        probs = (mb.TrsmProblem * 1)(mb.TrsmProblem(mb.M_LOWER, 0, mb.M_NON_UNIT, n, rhs, 1.0,
                                                    da.data_ptr(), n, db.data_ptr(), n))
        st = lib.mublis_b200_trsm_grouped(p.encode(), probs, 1)
    else:
        st = getattr(lib, f"mublis_{p}trsm")(0, mb.M_LOWER, 0, mb.M_NON_UNIT, n, rhs, 1.0,
                                             ctypes.c_void_p(da.data_ptr()), 1, n,
                                             ctypes.c_void_p(db.data_ptr()), 1, n)
    assert st == 0, mb.last_error(lib)
    x = db.cpu().numpy().T.astype(np.longdouble)
    worst = float((np.abs(wide @ x - b) / (np.abs(wide) @ np.abs(x))).max())
    assert worst <= 2 * (n + 4) * np.finfo(dt).eps / 2, worst
