"""Performance cases of the library: Level-3 BLAS calls as its users make them.

``listed()`` names the calls that are timed, ``draw()`` gives further calls of
the same ranges, ``prepare()`` builds what a caller has in hand (operands,
problem tables, plans), ``run()`` makes the one public call, ``work()`` counts
the bytes and flops the call cannot do without and ``exact()`` evaluates it in
float64 with torch.

Sizes are those of this repository's benchmark and tests: the n = 4096 family,
the 1024^3 SGEMM, the 8192^3 precision forms, 4096 grouped SGEMMs of 16-512,
1024 grouped DTRSMs of order 32-256, and the ragged sizes of the parity suite.
Inputs are uniform[-1, 1); triangular operands have off-diagonals uniform/n
and a diagonal in [1, 2), which keeps solves well conditioned.
"""
from __future__ import annotations

import ctypes
import math

import torch

import mublis_b200 as mb

ALPHA, BETA = 0.75, 0.25
DTYPES = {"s": torch.float32, "d": torch.float64}

_stream = None


def _lib():
    """The library, with the calling thread's work on a torch stream."""
    global _stream
    lib = mb.load()
    if _stream is None:
        mb.check(lib.mublis_b200_init(), lib)
        _stream = torch.cuda.Stream()
        mb.check(lib.mublis_b200_set_stream(_stream.cuda_stream), lib)
    return lib


# ---- the cases ---------------------------------------------------------------

def _gemm(name, dtype, m, n, k, ta="n", tb="n", form="plain", order="col", pad=0, beta=BETA,
          host=False):
    return {"name": name, "kind": "gemm", "dtype": dtype, "form": form, "order": order, "m": m,
            "n": n, "k": k, "ta": ta, "tb": tb, "pad": pad, "beta": beta, "host": host}


def _tri(name, kind, dtype, m, n, side="left", uplo="lower", trans="n", diag="nonunit",
         order="col", pad=0):
    return {"name": name, "kind": kind, "dtype": dtype, "form": "plain", "order": order, "m": m,
            "n": n, "side": side, "uplo": uplo, "trans": trans, "diag": diag, "pad": pad}


def _rank(name, kind, dtype, n, k, uplo="lower", trans="n", order="col", pad=0):
    return {"name": name, "kind": kind, "dtype": dtype, "form": "plain", "order": order, "n": n,
            "k": k, "uplo": uplo, "trans": trans, "pad": pad, "beta": BETA}


def _symm(name, dtype, m, n, side="left", uplo="lower", order="col", pad=0):
    return {"name": name, "kind": "symm", "dtype": dtype, "form": "plain", "order": order, "m": m,
            "n": n, "side": side, "uplo": uplo, "pad": pad, "beta": BETA}


def _group(name, kind, dtype, count, lo, hi, form="plain", plan=True):
    return {"name": name, "kind": kind, "dtype": dtype, "form": form, "count": count, "lo": lo,
            "hi": hi, "plan": plan}


def listed():
    return [
        # The smallest calls: one block of a blocked algorithm; latency counts.
        _gemm("sgemm_64", "s", 64, 64, 64),
        # An odd-sized block in double, A transposed.
        _gemm("dgemm_ragged", "d", 301, 177, 211, ta="t"),
        # The ordinary single call of the reference's first configuration.
        _gemm("sgemm_1024", "s", 1024, 1024, 1024),
        # The headline family at n = 4096: FP32 and FP64 products ...
        _gemm("sgemm_4096_nt", "s", 4096, 4096, 4096, tb="t"),
        _gemm("dgemm_4096", "d", 4096, 4096, 4096),
        # ... a triangular output (Gram matrices), at a size of the served mix ...
        _rank("ssyrk_2048", "syrk", "s", 2048, 2048),
        # ... and the triangular solve.
        _tri("dtrsm_4096", "trsm", "d", 4096, 4096),
        # A solve from the right with a ragged transposed upper factor.
        _tri("strsm_ragged_right", "trsm", "s", 1500, 1001, side="right", uplo="upper",
             trans="t"),
        # Many small independent products, planned once and replayed.
        _group("grouped_sgemm_4096", "grouped_gemm", "s", 4096, 16, 512),
        # The large FP32-class product on the tensor cores.
        _gemm("sgemm_8192_fp16x3", "s", 8192, 8192, 8192, form="fp16x3"),
        # The FP64-class product emulated on the int8 tensor cores.
        _gemm("dgemm_4096_ozaki2", "d", 4096, 4096, 4096, form="ozaki2"),
        # A caller of the reference's API with its operands in (pinned) host memory.
        _gemm("dgemm_host_1500", "d", 1500, 1500, 1500, host=True),
    ]


def _log_int(rng, lo, hi):
    """An integer of [lo, hi], uniform over its logarithm."""
    return min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))


def draw(rng):
    order = rng.choice(["col", "col", "row"])
    pad = rng.choice([0, 0, 0, 4, 5])
    dtype = rng.choice(["s", "d"])
    what = rng.choice(["gemm"] * 5 + ["trsm"] * 2 + ["trmm", "symm", "syrk", "syr2k", "grouped_gemm",
                                                     "grouped_trsm", "form", "form", "host"])
    m, n, k = (_log_int(rng, 16, 4096) for _ in range(3))
    if what == "gemm":
        c = _gemm("", dtype, m, n, k, rng.choice("nt"), rng.choice("nt"), order=order, pad=pad,
                  beta=rng.choice([0.0, BETA]))
    elif what in ("trsm", "trmm"):
        c = _tri("", what, dtype, m, n, rng.choice(["left", "right"]),
                 rng.choice(["lower", "upper"]), rng.choice("nt"),
                 rng.choice(["nonunit", "nonunit", "unit"]), order, pad)
    elif what == "symm":
        c = _symm("", dtype, m, n, rng.choice(["left", "right"]), rng.choice(["lower", "upper"]),
                  order, pad)
    elif what in ("syrk", "syr2k"):
        c = _rank("", what, dtype, n, k, rng.choice(["lower", "upper"]), rng.choice("nt"), order,
                  pad)
    elif what == "grouped_gemm":
        c = _group("", what, dtype, _log_int(rng, 64, 4096), 16, rng.choice([64, 128, 256, 512]),
                   rng.choice(["plain", "plain", "fp16x3"]) if dtype == "s" else "plain",
                   rng.random() < 0.5)
    elif what == "grouped_trsm":
        c = _group("", what, dtype, _log_int(rng, 64, 2048), 32, 256, plan=rng.random() < 0.5)
    elif what == "form":
        if dtype == "s":
            m, n, k = (_log_int(rng, 512, 8192) for _ in range(3))
            c = _gemm("", "s", m, n, k, rng.choice("nt"), rng.choice("nt"),
                      rng.choice(["fp16x3", "bf16x6", "bf16x3", "auto"]), order, pad)
        else:
            m, n, k = (_log_int(rng, 512, 4096) for _ in range(3))
            c = _gemm("", "d", m, n, k, rng.choice("nt"), rng.choice("nt"),
                      rng.choice(["ozaki2", "ozaki2:14", "auto"]), order, pad)
    else:
        m, n, k = (_log_int(rng, 16, 2048) for _ in range(3))
        c = _gemm("", dtype, m, n, k, rng.choice("nt"), rng.choice("nt"), order=order, pad=pad,
                  host=True)
    del c["name"]
    return c


# ---- operands ----------------------------------------------------------------
#
# A matrix is a torch tensor of its memory: row-major (rows, ld), column-major
# (cols, ld); _view gives it as rows x cols.

class _Maker:
    def __init__(self, case, seed):
        self.case, self.dt = case, DTYPES[case["dtype"]]
        self.gen = torch.Generator(device="cuda").manual_seed(seed)

    def uniform(self, *shape):
        return torch.rand(*shape, dtype=self.dt, device="cuda", generator=self.gen) * 2 - 1

    def matrix(self, rows, cols):
        if self.case["order"] == "row":
            return self.uniform(rows, cols + self.case["pad"])
        return self.uniform(cols, rows + self.case["pad"])

    def triangular(self, n):
        t = self.matrix(n, n).div_(n)
        diag = torch.rand(n, dtype=self.dt, device="cuda", generator=self.gen) + 1
        t[:, :n].diagonal().copy_(diag)
        return t


def _view(t, case, rows, cols):
    return t[:, :cols] if case["order"] == "row" else t[:, :rows].T


def _stored(rows, cols, trans):
    return (cols, rows) if trans == "t" else (rows, cols)


def _group_sizes(case):
    """The group's sizes: log-uniform over [lo, hi], the same for every seed."""
    g = torch.Generator().manual_seed(1000003 * case["count"] + case["hi"])
    shape = (case["count"], 3)
    lo, hi = math.log(case["lo"]), math.log(case["hi"] + 1)
    dims = torch.exp(torch.rand(shape, generator=g, dtype=torch.float64) * (hi - lo) + lo)
    dims = dims.floor().clamp_(case["lo"], case["hi"]).long()
    if case["kind"] == "grouped_trsm":  # right-hand sides: 1 .. 128
        dims[:, 1] = torch.exp(torch.rand(case["count"], generator=g, dtype=torch.float64)
                               * math.log(129)).floor().clamp_(1, 128).long()
    scal = torch.rand((case["count"], 2), generator=g, dtype=torch.float64) + 0.5
    if case["kind"] == "grouped_gemm":
        scal[:, 1] -= 0.5  # beta in [0, 1)
    return dims.tolist(), scal.tolist()


class _Plan:
    """A plan handle that is given back with its owner."""

    def __init__(self, lib, handle):
        self.lib, self.handle = lib, handle

    def __del__(self):
        self.lib.mublis_b200_plan_destroy(self.handle)


def _group_operands(case, seed):
    """Flat buffers of the group's operands and each problem's offsets."""
    mk = _Maker(case, seed)
    dims, scal = _group_sizes(case)
    if case["kind"] == "grouped_gemm":
        lens = [(m * k, k * n, m * n) for m, n, k in dims]
    else:
        lens = [(m * m, m * n) for m, n, _ in dims]
    offs, total = [], [0] * len(lens[0])
    for ls in lens:
        offs.append(tuple(total))
        for i, x in enumerate(ls):  # every matrix starts on 16 bytes
            total[i] += -(-x // 4) * 4
    bufs = [mk.uniform(t) for t in total]
    if case["kind"] == "grouped_trsm":
        idx, val = [], []
        for (m, _, _), (oa, _) in zip(dims, offs):
            bufs[0][oa:oa + m * m].div_(m)
            idx.append(oa + torch.arange(m) * (m + 1))
        idx = torch.cat(idx).cuda()
        val = torch.rand(idx.numel(), dtype=mk.dt, device="cuda", generator=mk.gen) + 1
        bufs[0][idx] = val
    return dims, scal, offs, bufs


def _prepare_group(case, seed):
    lib = _lib()
    dims, scal, offs, bufs = _group_operands(case, seed)
    elt = bufs[0].element_size()
    ptr = [b.data_ptr() for b in bufs]
    state = {"bufs": bufs}
    if case["kind"] == "grouped_gemm":
        probs = [mb.GemmProblem(0, 0, m, n, k, al, be, ptr[0] + oa * elt, m, ptr[1] + ob * elt, k,
                                ptr[2] + oc * elt, m)
                 for (m, n, k), (al, be), (oa, ob, oc) in zip(dims, scal, offs)]
        arr = (mb.GemmProblem * len(probs))(*probs)
        make = lib.mublis_b200_plan_gemm_grouped
    else:
        state["b0"] = bufs[1].clone()
        probs = [mb.TrsmProblem(mb.M_LOWER, 0, mb.M_NON_UNIT, m, n, al, ptr[0] + oa * elt, m,
                                ptr[1] + ob * elt, m)
                 for (m, n, _), (al, _), (oa, ob) in zip(dims, scal, offs)]
        arr = (mb.TrsmProblem * len(probs))(*probs)
        make = lib.mublis_b200_plan_trsm_grouped
    torch.cuda.synchronize()  # the plan's trial runs read the operands
    state["problems"] = arr
    if case["plan"]:
        handle = ctypes.c_void_p()
        mb.check(make(case["dtype"].encode(), arr, len(probs), ctypes.byref(handle)), lib)
        state["plan"] = _Plan(lib, handle)
    return state


def _operands(case, seed):
    """The call's matrices, in its argument order, on the GPU."""
    mk, kind = _Maker(case, seed), case["kind"]
    if kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return [mk.matrix(*_stored(m, k, case["ta"])), mk.matrix(*_stored(k, n, case["tb"])),
                mk.matrix(m, n)]
    if kind in ("syrk", "syr2k"):
        n, k = case["n"], case["k"]
        ins = [mk.matrix(*_stored(n, k, case["trans"])) for _ in range(1 + (kind == "syr2k"))]
        return ins + [mk.matrix(n, n)]
    m, n = case["m"], case["n"]
    ka = m if case["side"] == "left" else n
    if kind == "symm":
        return [mk.matrix(ka, ka), mk.matrix(m, n), mk.matrix(m, n)]
    return [mk.triangular(ka), mk.matrix(m, n)]


def prepare(case, seed):
    lib = _lib()
    # A program chooses its precision forms once.
    mb.check(lib.mublis_b200_set_form(case["dtype"].encode(), case["form"].encode()), lib)
    if case["kind"].startswith("grouped"):
        state = _prepare_group(case, seed)
    else:
        ops = _operands(case, seed)
        if case.get("host"):
            ops = [x.cpu().pin_memory() for x in ops]
        state = {"ops": ops, "args": _arguments(case, ops)}
        if case["kind"] in ("trmm", "trsm"):
            state["b0"] = ops[1].clone()  # the right-hand sides, which the call overwrites
    state["case"] = case
    state["fn"] = getattr(lib, _entry(case))
    return state


# ---- the calls ---------------------------------------------------------------

def _entry(case):
    if case["kind"].startswith("grouped"):
        if case["plan"]:
            return "mublis_b200_plan_run"
        return "mublis_b200_gemm_grouped" if case["kind"] == "grouped_gemm" \
            else "mublis_b200_trsm_grouped"
    return f"cblas_{case['dtype']}{case['kind']}"


_CBLAS = {"row": mb.ROW, "col": mb.COL, "n": mb.NO_TRANS, "t": mb.TRANS, "upper": mb.UPPER,
          "lower": mb.LOWER, "nonunit": mb.NON_UNIT, "unit": mb.UNIT, "left": mb.LEFT,
          "right": mb.RIGHT}


def _arguments(case, ops):
    """The cblas call's arguments."""
    e, kind = (lambda key: _CBLAS[case[key]]), case["kind"]
    p = [v for x in ops for v in (x.data_ptr(), x.shape[1])]  # pointer, leading dimension
    if kind == "gemm":
        return (e("order"), e("ta"), e("tb"), case["m"], case["n"], case["k"], ALPHA, *p[:4],
                case["beta"], *p[4:])
    if kind == "symm":
        return (e("order"), e("side"), e("uplo"), case["m"], case["n"], ALPHA, *p[:4],
                case["beta"], *p[4:])
    if kind in ("syrk", "syr2k"):
        return (e("order"), e("uplo"), e("trans"), case["n"], case["k"], ALPHA, *p[:-2],
                case["beta"], *p[-2:])
    return (e("order"), e("side"), e("uplo"), e("trans"), e("diag"), case["m"], case["n"], ALPHA,
            *p)


def run(state):
    case = state["case"]
    if "b0" in state:  # new right-hand sides, on the stream the library works on
        with torch.cuda.stream(_stream):
            (state["ops"][1] if "ops" in state else state["bufs"][1]).copy_(state["b0"])
    if "ops" in state:
        state["fn"](*state["args"])
        return state["ops"][-1]
    if case["plan"]:
        mb.check(state["fn"](state["plan"].handle))
    else:
        mb.check(state["fn"](case["dtype"].encode(), state["problems"], len(state["problems"])))
    return state["bufs"][-1]


# ---- what a call cannot do without, and its value ---------------------------

def work(case):
    elt, kind = (4 if case["dtype"] == "s" else 8), case["kind"]
    if kind.startswith("grouped"):
        dims, scal = _group_sizes(case)
        if kind == "grouped_gemm":
            return {"bytes": elt * sum(m * k + k * n + 2 * m * n for m, n, k in dims),
                    "flops": sum(2.0 * m * n * k for m, n, k in dims)}
        return {"bytes": elt * sum(m * (m + 1) / 2 + 2 * m * n for m, n, _ in dims),
                "flops": sum(float(m) * m * n for m, n, _ in dims)}
    n = case["n"]
    if kind in ("syrk", "syr2k"):
        pairs, k = (1 if kind == "syrk" else 2), case["k"]
        return {"bytes": elt * (pairs * n * k + n * (n + 1)), "flops": pairs * float(n) * (n + 1) * k}
    m = case["m"]
    if kind == "gemm":
        k = case["k"]
        return {"bytes": elt * (m * k + k * n + m * n * (2 if case["beta"] else 1)),
                "flops": 2.0 * m * n * k}
    ka = m if case["side"] == "left" else n
    if kind == "symm":
        return {"bytes": elt * (ka * (ka + 1) / 2 + 3 * m * n), "flops": 2.0 * m * n * ka}
    return {"bytes": elt * (ka * (ka + 1) / 2 + 2 * m * n), "flops": float(m) * n * ka}


def _exact_group(case, seed):
    dims, scal, offs, bufs = _group_operands(case, seed)
    bufs = [b.double() for b in bufs]
    for (m, n, k), (al, be), off in zip(dims, scal, offs):
        if case["kind"] == "grouped_gemm":
            a = bufs[0][off[0]:off[0] + m * k].view(k, m).T
            b = bufs[1][off[1]:off[1] + k * n].view(n, k).T
            c = bufs[2][off[2]:off[2] + m * n].view(n, m).T
            c.mul_(be).add_(a @ b, alpha=al)
        else:
            a = bufs[0][off[0]:off[0] + m * m].view(m, m).T
            b = bufs[1][off[1]:off[1] + m * n].view(n, m).T
            b.copy_(torch.linalg.solve_triangular(a.tril(), b * al, upper=False))
    return bufs[-1]


def exact(case, seed):
    """The value of run()'s output, from the same inputs in float64."""
    if case["kind"].startswith("grouped"):
        return _exact_group(case, seed)
    ops, kind = [x.double() for x in _operands(case, seed)], case["kind"]
    op = lambda t, rows, cols, tr: (_view(t, case, cols, rows).T if tr == "t"  # noqa: E731
                                    else _view(t, case, rows, cols))
    n = case["n"]
    if kind == "gemm":
        m, k = case["m"], case["k"]
        c = _view(ops[2], case, m, n)
        c.copy_(ALPHA * (op(ops[0], m, k, case["ta"]) @ op(ops[1], k, n, case["tb"]))
                + case["beta"] * c)
        return ops[2].cpu() if case["host"] else ops[2]
    if kind in ("syrk", "syr2k"):
        a = op(ops[0], n, case["k"], case["trans"])
        b = op(ops[-2], n, case["k"], case["trans"])
        full = a @ b.T if kind == "syrk" else a @ b.T + b @ a.T
        c = _view(ops[-1], case, n, n)
        mask = torch.ones(n, n, dtype=torch.bool, device="cuda")
        mask = mask.tril() if case["uplo"] == "lower" else mask.triu()
        c.copy_(torch.where(mask, ALPHA * full + case["beta"] * c, c))
        return ops[-1]
    m, left = case["m"], case["side"] == "left"
    ka = m if left else n
    a, b = _view(ops[0], case, ka, ka), _view(ops[1], case, m, n)
    half = a.tril() if case["uplo"] == "lower" else a.triu()
    if kind == "symm":
        a = half + half.T - torch.diag(half.diagonal())
        c = _view(ops[2], case, m, n)
        c.copy_(ALPHA * (a @ b if left else b @ a) + case["beta"] * c)
        return ops[2]
    if case["diag"] == "unit":
        half = half - torch.diag(half.diagonal()) + torch.eye(ka, dtype=half.dtype, device="cuda")
    a = half.T if case["trans"] == "t" else half
    if kind == "trmm":
        b.copy_(ALPHA * (a @ b if left else b @ a))
    else:
        upper = (case["uplo"] == "upper") != (case["trans"] == "t")
        b.copy_(torch.linalg.solve_triangular(a, ALPHA * b, upper=upper, left=left))
    return ops[1]
