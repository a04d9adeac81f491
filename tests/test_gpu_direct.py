"""Small products in one launch (gemm_direct.cu) against the oracle, device
pointers (GPU): sizes around the 32 and 64 tiles, the 16- and 32-deep
k-blocks and the cluster's k split, aligned and odd leading dimensions (16-byte
and element copies), in-place TRMM, and operands that are blocks of the
output's own matrix.  Normwise error <= 4 k u."""
import ctypes
import itertools

import numpy as np
import pytest

import mublis_b200 as mb
from oracle import oracle as orc
from tests import cases as cs

pytestmark = pytest.mark.gpu
DT = {"s": np.float32, "d": np.float64}


@pytest.fixture(scope="module", autouse=True)
def plain_forms(lib):
    assert lib.mublis_b200_init() == 0, mb.last_error(lib)
    lib.mublis_b200_set_form(b"s", b"plain")
    lib.mublis_b200_set_form(b"d", b"plain")
    orc.set_threads(8)


def padded(x, pad):
    """x (column-major) as the leading rows of a taller matrix, and on the device."""
    torch = pytest.importorskip("torch")
    full = np.full((x.shape[0] + pad, x.shape[1]), np.nan, x.dtype, order="F")
    full[:x.shape[0]] = x
    return torch.from_numpy(full.T.copy()).cuda()


def ptr(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("p", ["s", "d"])
@pytest.mark.parametrize("ta,tb", list(itertools.product((0, 1), repeat=2)))
@pytest.mark.parametrize("pad", [0, 1, 4])
@pytest.mark.parametrize("mnk", [(1, 1, 1), (32, 64, 16), (31, 33, 17), (64, 64, 64), (65, 63, 33),
                                 (20, 24, 2049), (96, 100, 1000), (333, 40, 5), (516, 772, 260)])
def test_direct_gemm_sizes(lib, p, ta, tb, pad, mnk):
    m, n, k = mnk
    dt = DT[p]
    a = orc.fill(*((k, m) if ta else (m, k)), dt, 11, 0)
    b = orc.fill(*((n, k) if tb else (k, n)), dt, 11, 1)
    c0 = orc.fill(m, n, dt, 11, 2)
    da, db, dc = padded(a, pad), padded(b, pad), padded(c0, pad)
    import torch
    torch.cuda.synchronize()
    args = lambda x: (1, x)  # noqa: E731
    assert getattr(lib, f"mublis_{p}gemm")(
        ta, tb, m, n, k, 0.75, ptr(da), *args(a.shape[0] + pad), ptr(db), *args(b.shape[0] + pad),
        0.25, ptr(dc), *args(m + pad)) == 0, mb.last_error(lib)
    out = dc.cpu().numpy().T
    ref = c0.copy(order="F")
    assert getattr(orc.restated(), f"oracle_{p}gemm")(
        ta, tb, m, n, k, 0.75, a.ctypes.data, 1, a.shape[0], b.ctypes.data, 1, b.shape[0], 0.25,
        ref.ctypes.data, 1, m) == 0
    err = np.linalg.norm(out[:m].astype(np.float64) - ref) / (
        0.75 * np.linalg.norm(a) * np.linalg.norm(b) + 0.25 * np.linalg.norm(c0))
    assert err <= 4 * k * cs.EPS[np.dtype(dt)]
    assert np.isnan(out[m:]).all()  # the padding is untouched


@pytest.mark.parametrize("p", ["s", "d"])
@pytest.mark.parametrize("side,uplo,trans,diag", [(0, 1, 0, 0), (0, 2, 1, 1), (1, 1, 1, 0), (1, 2, 0, 1)])
@pytest.mark.parametrize("m,n", [(1, 5), (32, 33), (65, 130), (300, 97)])
def test_direct_trmm_in_place(lib, p, side, uplo, trans, diag, m, n):
    import torch
    dt = DT[p]
    ka = m if side == 0 else n
    a = orc.fill(ka, ka, dt, 12, 0)
    a[np.triu_indices(ka, 1) if uplo == 1 else np.tril_indices(ka, -1)] = np.nan
    if diag:
        np.fill_diagonal(a, np.nan)
    b0 = orc.fill(m, n, dt, 12, 1)
    da, db = padded(a, 0), padded(b0, 3)
    torch.cuda.synchronize()
    assert getattr(lib, f"mublis_{p}trmm")(side, uplo, trans, diag, m, n, 0.75, ptr(da), 1, ka,
                                           ptr(db), 1, m + 3) == 0, mb.last_error(lib)
    ref = b0.copy(order="F")
    assert getattr(orc.restated(), f"oracle_{p}trmm")(side, uplo, trans, diag, m, n, 0.75,
                                                      a.ctypes.data, 1, ka, ref.ctypes.data, 1, m) == 0
    out = db.cpu().numpy().T
    bound = 0.75 * np.linalg.norm(np.nan_to_num(a, nan=1.0)) * np.linalg.norm(b0)
    assert np.linalg.norm(out[:m].astype(np.float64) - ref) / bound <= 4 * ka * cs.EPS[np.dtype(dt)]
    assert np.isnan(out[m:]).all()


@pytest.mark.parametrize("p", ["s", "d"])
@pytest.mark.parametrize("shift", [0, 40])
def test_direct_gemm_on_blocks_of_one_matrix(lib, p, shift):
    """C -= A B with all three blocks of one matrix: row blocks below one
    another (read in place), and (shift) a C that covers rows of B, which must
    be computed from the values B had before the call."""
    import torch
    dt = DT[p]
    m, n, k, ld = 96, 80, 64, 256
    x0 = orc.fill(ld, 160, dt, 13, 0)
    dx = padded(x0, 0)
    torch.cuda.synchronize()
    elt = np.dtype(dt).itemsize
    at = lambda i, j: ctypes.c_void_p(dx.data_ptr() + elt * (i + ld * j))  # noqa: E731
    row_c = 64 - shift
    assert getattr(lib, f"mublis_{p}gemm")(0, 0, m, n, k, -1.0, at(160, 80), 1, ld, at(0, 0), 1, ld,
                                           1.0, at(row_c, 0), 1, ld) == 0, mb.last_error(lib)
    out = dx.cpu().numpy().T.astype(np.float64)
    ref = x0.astype(np.float64)
    prod = ref[160:160 + m, 80:80 + k] @ ref[:k, :n]
    ref[row_c:row_c + m, :n] -= prod
    scale = np.linalg.norm(x0[160:160 + m, 80:80 + k]) * np.linalg.norm(x0[:k, :n]) + np.linalg.norm(
        x0[row_c:row_c + m, :n])
    assert np.linalg.norm(out - ref) / scale <= 4 * k * cs.EPS[np.dtype(dt)]
