"""The large products' kernels (gemm_ffma.cu, gemm_dmma.cu) on integers (GPU):
operands in {-2 .. 2}, so every sum is exact in either precision and the result must
equal NumPy's, element by element -- a lost k tail, edge row, pair or tile is a wrong
integer, whatever the size.

* Shapes that the dispatch sends there: ragged, every transpose, leading dimensions
  on 16 bytes and odd (operands read in place, or packed, or one of each), both
  layouts of C, triangular outputs, SYR2K's pair end on and off a k-block, and tile
  lists that the launch's parameters do not hold.  The library's profile says which
  kernel ran.
* test_small_shapes_without_the_small_kernel runs this module's small shapes, and the
  ragged, strided, split-K and generic-driver tests of the other modules, in a process
  where MUBLIS_B200_SMALL=0 sends every product to these kernels.
"""
import ctypes
import itertools
import json
import os
import subprocess
import sys

import numpy as np
import pytest

import mublis_b200 as mb
from tests.conftest import ROOT

pytestmark = pytest.mark.gpu
DT = {"s": np.float32, "d": np.float64}
KERNEL = {"s": "ffma_sgemm", "d": "dmma_dgemm"}
FORCED = os.environ.get("MUBLIS_B200_SMALL") == "0"
ALPHA, BETA = 2.0, -1.0


@pytest.fixture(scope="module", autouse=True)
def plain_forms(lib):
    assert lib.mublis_b200_init() == 0, mb.last_error(lib)
    lib.mublis_b200_set_form(b"s", b"plain")
    lib.mublis_b200_set_form(b"d", b"plain")


class Matrix:
    """rows x cols integers on the device, in `order`, lines `pad` elements apart from
    a multiple of 4 (0: on 16 bytes; 1: odd) and starting `shift` elements in."""

    def __init__(self, p, rows, cols, seed, order="F", pad=0, shift=0):
        import torch
        rng = np.random.default_rng(seed)
        self.x = rng.integers(-2, 3, (rows, cols)).astype(DT[p])
        self.order, lines, width = order, *((cols, rows) if order == "F" else (rows, cols))
        self.ld = -(-width // 4) * 4 + pad
        self.at, self.width, self.lines = shift, width, lines
        host = np.full(shift + lines * self.ld, 9, DT[p])
        host[shift:].reshape(lines, self.ld)[:, :width] = self.x.T if order == "F" else self.x
        self.host, self.dev = host, torch.from_numpy(host).cuda()
        self.ptr = ctypes.c_void_p(self.dev.data_ptr() + shift * host.itemsize)
        self.strides = (1, self.ld) if order == "F" else (self.ld, 1)

    def result(self):
        """The matrix now; what lies between its lines must be as it was."""
        out = self.dev.cpu().numpy()
        body = out[self.at:].reshape(self.lines, self.ld)
        assert (out[:self.at] == 9).all() and (body[:, self.width:] == 9).all()
        return body[:, :self.width].T if self.order == "F" else body[:, :self.width]


def run(lib, call, *args, kernel):
    """Makes the call; the profile must name the kernel."""
    import torch
    buf = ctypes.create_string_buffer(1 << 16)
    torch.cuda.synchronize()
    lib.mublis_b200_profile_read(buf, len(buf))
    lib.mublis_b200_profile_enable(1)
    st = call(*args)
    lib.mublis_b200_profile_enable(0)
    lib.mublis_b200_profile_read(buf, len(buf))
    assert st == 0, mb.last_error(lib)
    ran = json.loads(buf.value.decode())
    assert kernel in ran, ran


def gemm(lib, p, m, n, k, ta, tb, pads, order="F", corder="F", shift=0,
         kernel=KERNEL):
    a = Matrix(p, *((k, m) if ta else (m, k)), 1, order, pads[0], shift)
    b = Matrix(p, *((n, k) if tb else (k, n)), 2, order, pads[1], shift)
    c = Matrix(p, m, n, 3, corder, pads[2])
    run(lib, getattr(lib, f"mublis_{p}gemm"), int(ta), int(tb), m, n, k, ALPHA, a.ptr, *a.strides,
        b.ptr, *b.strides, BETA, c.ptr, *c.strides, kernel=kernel[p])
    op = lambda x, t: x.x.T if t else x.x  # noqa: E731
    want = ALPHA * (op(a, ta).astype(np.float64) @ op(b, tb).astype(np.float64)) + BETA * c.x
    np.testing.assert_array_equal(c.result(), want)


TRANS = list(itertools.product((False, True), repeat=2))


@pytest.mark.parametrize("p", ["s", "d"])
@pytest.mark.parametrize("ta,tb", TRANS)
@pytest.mark.parametrize("pads", [(0, 0, 0), (1, 1, 1), (0, 1, 1), (1, 0, 0)])
def test_gemm(lib, p, ta, tb, pads):
    gemm(lib, p, 3001, 2847, 1333, ta, tb, pads)


@pytest.mark.parametrize("p", ["s", "d"])
@pytest.mark.parametrize("order,corder,shift", [("C", "C", 0), ("F", "C", 0), ("C", "F", 0), ("F", "F", 1)])
def test_gemm_layouts(lib, p, order, corder, shift):
    gemm(lib, p, 2700, 2531, 1285, False, True, (0, 0, 0), order, corder, shift)


def rank(lib, p, routine, n, k, uplo, trans, pad, kernel=KERNEL):
    shape = (k, n) if trans else (n, k)
    a, b = Matrix(p, *shape, 4, pad=pad), Matrix(p, *shape, 5, pad=pad)
    c = Matrix(p, n, n, 6, pad=pad)
    if routine == "syrk":
        run(lib, getattr(lib, f"mublis_{p}syrk"), uplo, int(trans), n, k, ALPHA, a.ptr, *a.strides,
            BETA, c.ptr, *c.strides, kernel=kernel[p])
    else:
        run(lib, getattr(lib, f"mublis_{p}syr2k"), uplo, int(trans), n, k, ALPHA, a.ptr, *a.strides,
            b.ptr, *b.strides, BETA, c.ptr, *c.strides, kernel=kernel[p])
    x, y = (a.x.T, b.x.T) if trans else (a.x, b.x)
    x, y = x.astype(np.float64), y.astype(np.float64)
    full = x @ x.T if routine == "syrk" else x @ y.T + y @ x.T
    keep = np.tri(n, dtype=bool) if uplo == mb.M_LOWER else np.tri(n, dtype=bool).T
    np.testing.assert_array_equal(c.result(), np.where(keep, ALPHA * full + BETA * c.x, c.x))


@pytest.mark.parametrize("p", ["s", "d"])
@pytest.mark.parametrize("uplo", [mb.M_LOWER, mb.M_UPPER])
@pytest.mark.parametrize("routine,k,trans,pad", [("syrk", 1333, False, 0), ("syrk", 1333, True, 1),
                                                 ("syr2k", 672, False, 0), ("syr2k", 672, True, 0),
                                                 ("syr2k", 667, False, 0), ("syr2k", 672, False, 1)])
def test_triangular_outputs(lib, p, uplo, routine, k, trans, pad):
    rank(lib, p, routine, 3601, k, uplo, trans, pad)


# More than 1024 tiles of the triangle: the list is uploaded.
@pytest.mark.parametrize("p", ["s", "d"])
@pytest.mark.parametrize("uplo", [mb.M_LOWER, mb.M_UPPER])
def test_uploaded_tile_list(lib, p, uplo):
    rank(lib, p, "syrk", 6001, 600, uplo, False, 0)


def trmm(lib, p, right, uplo, trans, m, n, pad, kernel=KERNEL):
    s = n if right else m
    a, b = Matrix(p, s, s, 7, pad=pad), Matrix(p, m, n, 8, pad=pad)
    run(lib, getattr(lib, f"mublis_{p}trmm"), int(right), uplo, int(trans), mb.M_NON_UNIT, m, n,
        ALPHA, a.ptr, *a.strides, b.ptr, *b.strides, kernel=kernel[p])
    t = (np.tril if uplo == mb.M_LOWER else np.triu)(a.x).astype(np.float64)
    t, x = t.T if trans else t, b.x.astype(np.float64)
    np.testing.assert_array_equal(b.result(), ALPHA * (x @ t if right else t @ x))


# Tile indexes past 255, which the launch's parameters cannot hold either.
@pytest.mark.parametrize("p", ["s", "d"])
@pytest.mark.parametrize("right", [False, True])
def test_wide_triangular_product(lib, p, right):
    m, n = (33000, 520) if right else (520, 33000)
    trmm(lib, p, right, mb.M_LOWER, False, m, n, 0)


# ---- small shapes, in a process without the small kernel ----------------------

def forced(test):
    test.__test__ = FORCED  # collected in that process only
    return test


@forced
@pytest.mark.parametrize("p", ["s", "d"])
@pytest.mark.parametrize("ta,tb", TRANS)
@pytest.mark.parametrize("pads", [(0, 0, 0), (1, 1, 1), (0, 1, 0), (1, 0, 1)])
@pytest.mark.parametrize("mnk", [(1, 1, 1), (127, 129, 255), (128, 128, 16), (130, 257, 33),
                                 (300, 200, 513), (129, 127, 2049), (3, 700, 15)])
def forced_gemm(lib, p, ta, tb, pads, mnk):
    gemm(lib, p, *mnk, ta, tb, pads)


@forced
@pytest.mark.parametrize("p", ["s", "d"])
@pytest.mark.parametrize("order,corder,shift", [("C", "C", 0), ("F", "C", 0), ("C", "F", 0),
                                                ("F", "F", 1), ("F", "F", 2)])
@pytest.mark.parametrize("ta,tb", TRANS)
def forced_layouts(lib, p, order, corder, shift, ta, tb):
    gemm(lib, p, 261, 135, 83, ta, tb, (0, 0, 0), order, corder, shift)


@forced
@pytest.mark.parametrize("p", ["s", "d"])
@pytest.mark.parametrize("uplo", [mb.M_LOWER, mb.M_UPPER])
@pytest.mark.parametrize("trans", [False, True])
@pytest.mark.parametrize("routine,n,k,pad", [("syrk", 1, 1, 0), ("syrk", 129, 2049, 0), ("syrk", 300, 40, 1),
                                             ("syr2k", 129, 16, 0), ("syr2k", 300, 17, 0),
                                             ("syr2k", 257, 1024, 0), ("syr2k", 257, 48, 1)])
def forced_rank(lib, p, uplo, trans, routine, n, k, pad):
    rank(lib, p, routine, n, k, uplo, trans, pad)


@forced
@pytest.mark.parametrize("p", ["s", "d"])
@pytest.mark.parametrize("right,uplo,trans", list(itertools.product((False, True), (mb.M_LOWER, mb.M_UPPER),
                                                                    (False, True))))
@pytest.mark.parametrize("m,n,pad", [(1, 1, 0), (130, 129, 0), (257, 40, 1), (400, 385, 0)])
def forced_trmm(lib, p, right, uplo, trans, m, n, pad):
    trmm(lib, p, right, uplo, trans, m, n, pad)


@pytest.mark.parametrize("direct", ["1", "0"], ids=["in_place", "packed"])
def test_small_shapes_without_the_small_kernel(direct):
    """direct 0: every operand packed as well."""
    here = ["tests/test_gpu_large_kernels.py", "-k", "forced"]
    others = ["tests/test_gpu_sched.py", "tests/test_gpu_parity.py", "-k",
              "split_k or direct_loads or ragged or midsize or beta_zero or strides or domains"]
    env = dict(os.environ, MUBLIS_B200_SMALL="0", MUBLIS_B200_DIRECT=direct)
    for args in (here, others) if direct == "1" else (here,):
        subprocess.run([sys.executable, "-m", "pytest", "-q", "-x", "-m", "gpu", "-p", "no:cacheprovider",
                        *args], check=True, cwd=ROOT, env=env, timeout=600)
