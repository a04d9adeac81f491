"""The plain products' sums are as short as split-K makes them (GPU).  Each call's
normwise error, on 48 rows and columns against exact values, is held against that of
the same entries added up on the host in runs of `chunk` products (one rounding per
multiply-add) and then run by run: the chunks into which these shapes' k was cut when
all of them ran on 128 x 128 tiles.  The margin of 1.15 covers the sample: the error
of 2304 entries has a standard deviation of about 1.5%."""
import ctypes

import numpy as np
import pytest

import mublis_b200 as mb
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
WIDE = {np.dtype(np.float32): np.float64, np.dtype(np.float64): np.longdouble}


def in_runs(a, b, chunk):
    """a b with sums of `chunk` products in a's precision."""
    dt, k = a.dtype, a.shape[1]
    wide = WIDE[dt]
    total = np.zeros((a.shape[0], b.shape[1]), dt)
    for k0 in range(0, k, chunk):
        run = np.zeros_like(total)
        for p in range(k0, min(k, k0 + chunk)):
            run = (run.astype(wide) + np.multiply.outer(a[:, p].astype(wide), b[p].astype(wide))).astype(dt)
        total = total + run
    return total


SMALL = [("s", 696, 389, 1855, 160), ("s", 1794, 151, 1863, 208), ("s", 677, 327, 3015, 192),
         ("s", 1236, 788, 1005, 256), ("d", 254, 1050, 1370, 176), ("d", 1180, 300, 1500, 304)]


LARGE = [("s", 2000, 2587, 1300, 336), ("s", 1660, 2849, 901, 240), ("s", 197, 4081, 1805, 464)]


@pytest.mark.parametrize("p,m,n,k,chunk", SMALL + LARGE)
def test_sums_are_as_short_as_split_k_made_them(lib, p, m, n, k, chunk):
    torch = pytest.importorskip("torch")
    assert lib.mublis_b200_init() == 0, mb.last_error(lib)
    lib.mublis_b200_set_form(p.encode(), b"plain")
    dt = np.float32 if p == "s" else np.float64
    a, b = orc.fill(m, k, dt, 41, 0), orc.fill(k, n, dt, 41, 1)
    da, db = torch.from_numpy(a.T.copy()).cuda(), torch.from_numpy(b.T.copy()).cuda()
    dc = torch.zeros(n, m, dtype=da.dtype, device="cuda")
    torch.cuda.synchronize()
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    assert getattr(lib, f"mublis_{p}gemm")(0, 0, m, n, k, 1.0, ptr(da), 1, m, ptr(db), 1, k, 0.0,
                                           ptr(dc), 1, m) == 0, mb.last_error(lib)
    rows, cols = np.linspace(0, m - 1, 48).astype(int), np.linspace(0, n - 1, 48).astype(int)
    x, y = a[rows], b[:, cols]
    exact = x.astype(np.longdouble) @ y.astype(np.longdouble)
    err = np.linalg.norm((dc.cpu().numpy().T[np.ix_(rows, cols)] - exact).astype(np.float64))
    ref = np.linalg.norm((in_runs(x, y, chunk) - exact).astype(np.float64))
    assert err <= 1.15 * ref, (err / ref)
