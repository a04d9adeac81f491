"""Triangular solves at the edges of their kernels (GPU), against the oracle: the
one-launch kernel's 16-row blocks, its two orders of CTA (128, 256) and its 32
columns; the leaf kernel's blocks, leaves (512) and column groups (8, 16, 32);
and the orders and counts of right-hand sides at which the leaves change.  Both
triangles, unit and non-unit, from the left and the right, both layouts, odd
leading dimensions, alpha != 1.  Relative forward error <= 4 * order * u."""
import numpy as np
import pytest

import mublis_b200 as mb
from oracle import oracle as orc
from tests import cases as cs

pytestmark = pytest.mark.gpu

SMALL = [(o, n) for o in (1, 15, 16, 17, 128, 129, 255, 256) for n in (1, 31, 32, 33)]
LEAF = [(257, 7), (272, 9), (500, 17), (512, 33), (513, 15), (1023, 8), (530, 1184), (530, 1185),
        (530, 1193), (2048, 512), (2049, 512), (2049, 513)]
FLAGS = [dict(right=False, lower=True, ta=False, unit=False, order="F"),
         dict(right=False, lower=False, ta=True, unit=True, order="C"),
         dict(right=True, lower=True, ta=False, unit=True, order="F"),
         dict(right=True, lower=False, ta=False, unit=False, order="C")]


@pytest.fixture(scope="module", autouse=True)
def plain_forms(lib):
    assert lib.mublis_b200_init() == 0, mb.last_error(lib)
    lib.mublis_b200_set_form(b"s", b"plain")
    lib.mublis_b200_set_form(b"d", b"plain")
    orc.set_threads(8)


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("flags", FLAGS, ids=["LLN", "LUTu", "RLNu", "RUN"])
@pytest.mark.parametrize("order,rhs", SMALL + LEAF)
def test_trsm_edges(lib, dtype, flags, order, rhs):
    m, n = (rhs, order) if flags["right"] else (order, rhs)
    case = dict(routine="trsm", dtype=dtype, m=m, n=n, k=0, alpha=-1.25, seed=order + rhs, **flags)
    a, b, c0 = cs.build(case)
    out, ref = c0.copy(order="K"), c0.copy(order="K")
    cs.cblas_call(lib, case, a, b, out)
    cs.oracle_call(case, a, b, ref)
    assert np.isfinite(out).all()
    assert cs.normwise_error(case, out, ref, a, b, c0) <= 4 * order * cs.EPS[np.dtype(dtype)]
