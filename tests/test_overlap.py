"""The overlap test that decides whether a product may read its operands in
place (b200_views_overlap): against the element addresses themselves, for
blocks of one matrix in every orientation and for unrelated strides (CPU)."""
import ctypes
import random

import mublis_b200 as mb


def addresses(base, rs, cs, m, n, elt):
    return {base + elt * (i * rs + j * cs) for i in range(m) for j in range(n)}


def test_overlap_never_misses_a_shared_element():
    lib = mb.load()
    fn = lib.b200_views_overlap
    fn.argtypes = [ctypes.c_void_p] + [ctypes.c_long] * 4 + [ctypes.c_void_p] + [ctypes.c_long] * 5
    rng = random.Random(7)
    disjoint = exact = 0
    for trial in range(4000):
        elt = rng.choice([4, 8])
        ld = rng.randint(1, 9)
        base = 1 << 20

        def view(ld):
            width, lines = rng.randint(1, ld), rng.randint(1, 6)
            at = base + elt * (rng.randint(0, ld - 1) + ld * rng.randint(0, 8))
            if rng.random() < 0.1:
                at += rng.randint(1, elt - 1)
            if rng.random() < 0.5:
                return at, 1, ld, width, lines
            return at, ld, 1, lines, width

        c = view(ld)
        x = view(ld if rng.random() < 0.8 else rng.randint(1, 9))
        got = fn(*c, *x, elt)
        shared = any(abs(p - q) < elt for p in addresses(*c, elt) for q in addresses(*x, elt))
        assert got or not shared, (c, x, elt)
        if not shared:
            disjoint += 1
            exact += not got
    assert exact > disjoint / 2  # and it does tell disjoint blocks apart
    # Row blocks of one column-major matrix: interleaved intervals, no element shared.
    assert not fn(base, 1, 100, 50, 20, base + 50 * 8, 1, 100, 50, 20, 8)
    assert fn(base, 1, 100, 51, 20, base + 50 * 8, 1, 100, 50, 20, 8)
    assert fn(base, 1, -100, 50, 20, base + 50 * 8, 1, 100, 50, 20, 8)  # negative stride: assumed
