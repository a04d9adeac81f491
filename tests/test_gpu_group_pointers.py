"""Grouped calls check every operand's pointer though most lie in allocations they
have already met (GPU): one host pointer (pageable or pinned) anywhere among
device pointers of few or many allocations is refused and nothing is written;
without it the products are right (exact: small integers)."""
import numpy as np
import pytest

import mublis_b200 as mb

pytestmark = pytest.mark.gpu
N = 4  # order of every product


@pytest.mark.parametrize("p", ["s", "d"])
@pytest.mark.parametrize("own", [False, True], ids=["shared", "own"])
@pytest.mark.parametrize("count", [1, 3, 40, 100])
def test_group_pointer_checks(lib, p, own, count):
    torch = pytest.importorskip("torch")
    assert lib.mublis_b200_init() == 0, mb.last_error(lib)
    dt = torch.float32 if p == "s" else torch.float64
    # Allocations of their own: larger than the allocator's shared blocks.
    size = (12 << 20) // dt.itemsize if own else N * N
    keep = [torch.ones(size, dtype=dt, device="cuda") for _ in range(count if own else 1)]
    a = [keep[i] if own else keep[0] for i in range(count)]
    c = torch.full((count, N, N), 7.0, dtype=dt, device="cuda")

    def problems(bad=None, where="a"):
        out = []
        for i in range(count):
            q = dict(a=a[i].data_ptr(), b=a[-1 - i].data_ptr(), c=c[i].data_ptr())
            if i == bad[0] if bad else False:
                q[where] = bad[1]
            out.append(mb.GemmProblem(0, 0, N, N, N, 1.0, 0.0, q["a"], N, q["b"], N, q["c"], N))
        return (mb.GemmProblem * count)(*out)

    host = torch.ones(N * N, dtype=dt)
    pinned = torch.ones(N * N, dtype=dt).pin_memory()
    for where in "abc":
        for t in (host, pinned):
            for i in {0, count // 2, count - 1}:
                probs = problems((i, t.data_ptr()), where)
                assert lib.mublis_b200_gemm_grouped(p.encode(), probs, count) != 0
    torch.cuda.synchronize()
    assert (c == 7.0).all()
    assert lib.mublis_b200_gemm_grouped(p.encode(), problems(), count) == 0, mb.last_error(lib)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(c.cpu().numpy(), np.full((count, N, N), float(N)))
