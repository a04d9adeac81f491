#!/usr/bin/env python
"""Benchmark of the B200 Level-3 BLAS (one JSON line on rank 0).

Workload (N = 1): the plain Level-3 family at n = 4096 in FP32 and FP64 --
GEMM in all four transA/transB combinations at m = n = k = 4096, SYMM
left/lower (lower triangle stored), SYRK and SYR2K lower (n = k = 4096),
TRMM left/lower/non-unit, TRSM left/lower/non-unit (A: off-diagonals
uniform[-1,1)/n, diagonal uniform[1,2)), B 4096 x 4096, alpha 0.75,
beta 0.25, column-major, seeded Philox uniform[-1,1) inputs.  One step is
those 18 calls through the cblas_* entry points.

* value: TFLOP/s of the whole step with operands resident in HBM (device
  pointers), timed with CUDA events on the library's stream (the caller's
  torch stream, set with mublis_b200_set_stream).  BLAS flop counts: GEMM
  2mnk, SYMM 2m^2n, SYRK n(n+1)k, SYR2K 2n(n+1)k, TRMM/TRSM m^2n.
* e2e: the same step through cblas_* with pinned HOST buffers, so every call
  stages its operands to the device and its result back inside the timed
  region.
* roofline: the dominant kernel's achieved rate from per-launch CUDA events
  (library profiler, recorded on the launching stream during the timed
  region) against its pipe's peak.
* cpu_baseline: the reference's own avx2 build (oracle/_ref) on the host
  cores: one step of the same n = 4096 family, every call cut into column
  panels that are separate reference calls, spread over all host threads
  (the library is single-threaded per call); plus the family at n = 2048
  on one thread.
* --impl reference: the reference's avx2 build timed the same way on the
  same n = 4096 family, --steps timed steps after --warmup untimed ones.

Multi-GPU: the path does not shard (one BLAS call per GPU); --gpus N runs N
independent replicas under torchrun, value = total flops / max-over-ranks
time, scaling "weak".
"""
from __future__ import annotations

import argparse
import ctypes
import json
import os
import re
import statistics
import subprocess
import sys
import time
from pathlib import Path

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

METRIC = "SGEMM/DGEMM/TRSM TFLOP/s (% of peak) at stated err; served p50/p99 vs plain"
ROUTINES = ["gemm_nn", "gemm_nt", "gemm_tn", "gemm_tt", "symm", "syrk", "syr2k", "trmm", "trsm"]
COL, NT, TR, UPPER, LOWER, NONUNIT, LEFT = 102, 111, 112, 121, 122, 131, 141
ALPHA, BETA = 0.75, 0.25
FP64_NOMINAL_TFLOPS = 148 * 64 * 2 * 1.965e9 / 1e12   # SMs x FP64 FMA lanes x 2 x max clock
FP32_NOMINAL_TFLOPS = 148 * 128 * 2 * 1.965e9 / 1e12  # SMs x FP32 FMA lanes x 2 x max clock


def flops(routine: str, n: int) -> float:
    if routine.startswith("gemm"):
        return 2.0 * n ** 3
    if routine == "symm":
        return 2.0 * n ** 3
    if routine == "syrk":
        return float(n) * (n + 1) * n
    if routine == "syr2k":
        return 2.0 * n * (n + 1) * n
    return float(n) ** 3


def family_flops(n: int) -> float:
    return 2 * sum(flops(r, n) for r in ROUTINES)


def kernel_flops(n: int) -> dict:
    """Algorithmic flops of one step attributed to the kernel that executes
    them: every routine but TRSM, whose leaves and whose smaller updates run in
    other kernels (a larger update that this kernel runs is not credited)."""
    gemm_part = sum(flops(r, n) for r in ROUTINES if r != "trsm")
    return {"ffma_sgemm": gemm_part, "simt_dgemm": gemm_part, "dmma_dgemm": gemm_part}


def max_over_ranks(dist, torch, ms: float, world: int, device: str = "cuda") -> float:
    """The slowest replica's time: every rank contributes its own and all get
    the maximum (a job of N replicas is as fast as its slowest one)."""
    if world <= 1:
        return ms
    t = torch.tensor([ms], device=device, dtype=torch.float64)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def whole_job_tflops(flops_per_rank: float, world: int, ms: float) -> float:
    """Whole-job throughput: every rank does flops_per_rank in ms (the max)."""
    return world * flops_per_rank / (ms * 1e-3) / 1e12


def measured_peaks() -> dict:
    p = ROOT / "MEASURED_PEAKS.json"
    if p.is_file():
        try:
            return json.loads(p.read_text())
        except ValueError:
            pass
    return {}


def profile_traffic(kernel: str):
    """DRAM bytes per launch of `kernel` from a committed ncu summary
    (profiles/<kernel>_*.txt, line 'dram_bytes_per_launch: N'), or None."""
    for f in sorted((ROOT / "profiles").glob(f"{kernel}_*.txt")):
        m = re.search(r"dram_bytes_per_launch:\s*([0-9.eE+]+)", f.read_text())
        if m:
            return float(m.group(1))
    return None


class ClockSampler:
    """nvidia-smi clock / throttle-reason sampling during the timed region."""

    FIELDS = ("clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index: int):
        self.proc = None
        self.out = []
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(gpu_index), f"--query-gpu={self.FIELDS}",
                 "--format=csv,noheader,nounits", "-lms", "200"],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
        except OSError:
            self.proc = None

    def stop(self) -> dict | None:
        if self.proc is None:
            return None
        self.proc.terminate()
        try:
            text, _ = self.proc.communicate(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
            text, _ = self.proc.communicate()
        sm, mx, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in text.strip().splitlines():
            parts = [x.strip() for x in line.split(",")]
            if len(parts) < 8:
                continue
            try:
                sm.append(float(parts[0]))
                mx.append(float(parts[1]))
            except ValueError:
                continue
            for name, val in zip(names, parts[4:8]):
                if val.lower() == "active":
                    reasons.add(name)
        if not sm:
            return None
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": max(mx),
                "samples": len(sm), "reasons": sorted(reasons)}


# ---------------------------------------------------------------- reference arm

def ref_bench(n: int, threads: int, reps: int, warmup: int, mode: str = "family",
              panel: int = 512) -> dict:
    """Times the reference's own avx2 build through oracle/lib/ref_bench.
    mode "family": every thread runs the whole 18-call family on its own
    operands; "family_par": one shared family of 18 calls, each cut into
    column panels of `panel` columns (separate reference cblas calls), spread
    over all threads, one pass per step."""
    from oracle import oracle as orc  # checker/baseline only
    lib = orc.ref_lib_path("avx2")
    if not lib.is_file() or not orc.REF_BENCH.is_file():
        raise FileNotFoundError("reference build missing (make -C oracle)")
    cmd = [str(orc.REF_BENCH), str(lib), mode, "x", str(n), str(n), str(n), str(threads),
           str(reps), str(warmup)]
    if mode == "family_par":
        cmd.append(str(panel))
    out = subprocess.run(cmd, check=True, capture_output=True, text=True).stdout
    return json.loads(out.strip().splitlines()[-1])


def host_threads() -> int:
    try:
        return len(os.sched_getaffinity(0))
    except AttributeError:  # pragma: no cover
        return os.cpu_count() or 1


def par_sample(n: int, threads: int, panel: int) -> str:
    return (f"per step: the 18-call family at m=n=k={n} (the benchmarked workload), every call "
            f"cut into column panels of {panel} columns issued as separate reference cblas "
            f"calls (SYRK/SYR2K: diagonal block + GEMMs below), largest first over {threads} "
            f"host threads (reference linux_avx2 build, 1 thread per call)")


def run_reference_arm(args, rank: int, world: int) -> None:
    if rank != 0:
        return
    n = args.n
    threads = host_threads()
    config = workload_config(n)
    try:
        r = ref_bench(n, threads, args.steps, args.warmup, mode="family_par", panel=512)
    except Exception as e:  # noqa: BLE001
        print(json.dumps({"impl": "reference", "unavailable": f"reference build not runnable: {e}"}))
        return
    ms = r["wall_s"] / args.steps * 1e3
    value = r["gflops_aggregate"] / 1e3
    print(json.dumps({
        "impl": "reference", "metric": METRIC, "value": value, "unit": "TFLOP/s",
        "n_gpus": world, "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32+f64",
        "data": "synthetic", "config": config,
        "cpu_baseline": {"value": value, "unit": "TFLOP/s", "cores": threads,
                         "kind": "reference", "sample": par_sample(n, threads, 512)},
        "e2e": {"value": value, "unit": "TFLOP/s", "h2d_bytes_per_step": 0,
                "d2h_bytes_per_step": 0}}))


def workload_config(n: int) -> dict:
    return {"workload": f"plain L3 family n={n}: FP32+FP64 GEMM NN/NT/TN/TT, SYMM L/lower, "
                        f"SYRK lower, SYR2K lower, TRMM L/lower/non-unit, TRSM L/lower/non-unit",
            "n": n, "calls_per_step": 18, "alpha": ALPHA, "beta": BETA,
            "layout": "column-major", "forms": {"s": "plain", "d": "plain"},
            "l2": "inputs larger than L2: every call owns its operands, 4.6 GB per step "
                  "vs 126 MB L2, so each call starts cold",
            "parallelism": "replicas"}


# ---------------------------------------------------------------- device arm

def tri_elements(n: int, block: int = 256) -> int:
    """Elements of an n x n triangle as the host path stages it: blocks of
    `block` columns, each from its first column's diagonal down."""
    return sum((n - j0) * min(block, n - j0) for j0 in range(0, n, block))


class Family:
    """The 18 calls of one step with their own operands."""

    def __init__(self, torch, lib, n: int, device: bool):
        self.torch, self.lib, self.n = torch, lib, n
        self.calls = []
        self.h2d = 0
        self.d2h = 0
        for p, dt in (("s", torch.float32), ("d", torch.float64)):
            fill = getattr(lib, f"mublis_b200_fill_{p}")
            elt = 4 if p == "s" else 8
            for r in ROUTINES:
                mid = len(self.calls) * 3

                def mat(i, kind=0):
                    t = torch.empty(n, n, dtype=dt, device="cuda")
                    assert fill(ctypes.c_void_p(t.data_ptr()), n, n, n, 0, mid + i, kind) == 0
                    return t
                a = mat(0)
                if r in ("trmm", "trsm"):
                    d = mat(0, 2)
                    a.div_(n)
                    a.diagonal().copy_(d.diagonal())
                    del d
                b = mat(1)
                c = mat(2) if r not in ("trmm", "trsm") else None
                ops = [a, b] + ([c] if c is not None else [])
                if not device:
                    ops = [x.cpu().pin_memory() for x in ops]
                self.calls.append((p, r, ops))
                # Bytes the host path moves: triangular / symmetric A cross
                # PCIe as their triangle only, in blocks of 256 columns; the
                # SYRK / SYR2K C (both ways) in the lower-triangle pipeline's
                # blocks of 128 columns.
                n2, t2 = n * n * elt, tri_elements(n) * elt
                piped = n >= 2048 and n * n * elt // 2 >= 32 << 20
                c2 = tri_elements(n, 128 if piped else 256) * elt
                if r in ("trmm", "trsm"):
                    self.h2d += t2 + n2
                    self.d2h += n2
                elif r == "symm":
                    self.h2d += t2 + 2 * n2
                    self.d2h += n2
                elif r == "syrk":
                    self.h2d += n2 + c2
                    self.d2h += c2
                elif r == "syr2k":
                    self.h2d += 2 * n2 + c2
                    self.d2h += c2
                else:
                    self.h2d += 3 * n2
                    self.d2h += n2
        torch.cuda.synchronize()

    def step(self):
        lib, n = self.lib, self.n
        for p, r, ops in self.calls:
            ptr = [ctypes.c_void_p(x.data_ptr()) for x in ops]
            if r.startswith("gemm"):
                ta = TR if r[5] == "t" else NT
                tb = TR if r[6] == "t" else NT
                getattr(lib, f"cblas_{p}gemm")(COL, ta, tb, n, n, n, ALPHA, ptr[0], n, ptr[1], n,
                                               BETA, ptr[2], n)
            elif r == "symm":
                getattr(lib, f"cblas_{p}symm")(COL, LEFT, LOWER, n, n, ALPHA, ptr[0], n, ptr[1],
                                               n, BETA, ptr[2], n)
            elif r == "syrk":
                getattr(lib, f"cblas_{p}syrk")(COL, LOWER, NT, n, n, ALPHA, ptr[0], n, BETA,
                                               ptr[2], n)
            elif r == "syr2k":
                getattr(lib, f"cblas_{p}syr2k")(COL, LOWER, NT, n, n, ALPHA, ptr[0], n, ptr[1],
                                                n, BETA, ptr[2], n)
            else:
                getattr(lib, f"cblas_{p}{r}")(COL, LEFT, LOWER, NT, NONUNIT, n, n, ALPHA, ptr[0],
                                              n, ptr[1], n)


def verify_step(torch, fam, ncheck: int = 16, seed: int = 7) -> dict:
    """Checks one more step of the family, outside the timed region: on
    `ncheck` seeded columns of every call's output, the normwise error against
    a float64 evaluation of the same columns on the device (torch; TRSM by a
    float64 triangular solve, relative forward error), divided by the stated
    bound 4*k*u.  SYRK/SYR2K's upper triangle must come back unchanged."""
    n = fam.n
    g = torch.Generator().manual_seed(seed)
    cols = torch.randperm(n, generator=g)[:ncheck].sort().values.cuda()
    norm = torch.linalg.norm
    before = []
    for p, r, ops in fam.calls:
        out = ops[1] if r in ("trmm", "trsm") else ops[2]
        before.append(out.t()[:, cols].to(torch.float64))
    fam.step()
    torch.cuda.synchronize()
    worst, untouched, per_call = 0.0, True, {}
    rows = torch.arange(n, device="cuda").unsqueeze(1)
    lower = rows >= cols.unsqueeze(0)
    for (p, r, ops), c0 in zip(fam.calls, before):
        u = 2.0 ** -24 if p == "s" else 2.0 ** -53
        A = ops[0].t().to(torch.float64)
        k = 2 * n if r == "syr2k" else n
        if r in ("trmm", "trsm"):
            L = torch.tril(A)
            got = ops[1].t()[:, cols].to(torch.float64)
            if r == "trmm":
                ref = ALPHA * (L @ c0)
                err = norm(got - ref) / (ALPHA * norm(L) * norm(c0))
            else:
                ref = torch.linalg.solve_triangular(L, ALPHA * c0, upper=False)
                err = norm(got - ref) / norm(ref)
        else:
            B = ops[1].t().to(torch.float64)
            got = ops[2].t()[:, cols].to(torch.float64)
            if r.startswith("gemm"):
                opa = A.t() if r[5] == "t" else A
                opb = (B.t() if r[6] == "t" else B)[:, cols]
                prod, fa = opa @ opb, norm(opa) * norm(opb)
            elif r == "symm":
                sym = torch.tril(A) + torch.tril(A, -1).t()
                prod, fa = sym @ B[:, cols], norm(sym) * norm(B[:, cols])
            elif r == "syrk":
                prod, fa = A @ A[cols, :].t(), norm(A) * norm(A[cols, :])
            else:
                prod = A @ B[cols, :].t() + B @ A[cols, :].t()
                fa = norm(A) * norm(B[cols, :]) + norm(B) * norm(A[cols, :])
            ref = ALPHA * prod + BETA * c0
            if r in ("syrk", "syr2k"):
                untouched = untouched and bool(torch.equal(got[~lower], c0[~lower]))
                got, ref, c0 = got * lower, ref * lower, c0 * lower
            err = norm(got - ref) / (ALPHA * fa + BETA * norm(c0))
        ratio = float(err) / (4 * k * u)
        per_call[f"{p}{r}"] = round(ratio, 6)
        worst = max(worst, ratio)
    return {"calls": len(fam.calls), "columns_per_call": ncheck,
            "max_err_over_bound": round(worst, 6), "bound": "4*k*u normwise (TRSM: relative "
            "forward error 4*n*u)", "upper_triangle_untouched": untouched,
            "err_over_bound": per_call}


def timed(torch, fn, steps: int):
    s = torch.cuda.current_stream()
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    e0.record(s)
    for _ in range(steps):
        fn()
    e1.record(s)
    torch.cuda.synchronize()
    return e0.elapsed_time(e1) / steps


FORM_CALLS = 10  # timed calls per form in the 8192 study (mean of one event pair)


def forms_study(torch, lib, n: int = 8192) -> dict:
    """Precision forms at m = n = k = n (8192 by default): one warm-up call,
    then FORM_CALLS back-to-back calls timed by one CUDA-event pair."""
    import mublis_b200 as mb
    out = {}
    for p, dt, forms in (("s", torch.float32, ["plain", "bf16x3", "bf16x6", "fp16x3", "ozaki2"]),
                         ("d", torch.float64, ["plain", "ozaki:7", "ozaki:8", "ozaki2:14", "ozaki2"])):
        fill = getattr(lib, f"mublis_b200_fill_{p}")
        a, b, c = (torch.empty(n, n, dtype=dt, device="cuda") for _ in range(3))
        for i, x in enumerate((a, b, c)):
            fill(ctypes.c_void_p(x.data_ptr()), n, n, n, 0, i, 0)
        fn = getattr(lib, f"cblas_{p}gemm")
        if p == "d":
            # The modulus-count autotuner at two error targets: its choice
            # (measured on the leading 256 x 256 block) and the form's speed.
            for target in (1e-15, 1e-17):
                nm, err = ctypes.c_int(), ctypes.c_double()
                mb.check(lib.mublis_b200_ozaki2_autotune(
                    b"d", 0, 0, n, n, n, ctypes.c_void_p(a.data_ptr()), 1, n,
                    ctypes.c_void_p(b.data_ptr()), 1, n, target, ctypes.byref(nm),
                    ctypes.byref(err)), lib)
                out[f"dgemm_{n}_ozaki2@{target:g}_moduli"] = nm.value
                out[f"dgemm_{n}_ozaki2@{target:g}_calibration_err"] = float(f"{err.value:.3g}")
                forms = forms + [f"ozaki2@{target:g}"]
        for f in forms:
            lib.mublis_b200_set_form(p.encode(), f.encode())
            call = lambda: fn(COL, NT, NT, n, n, n, 1.0, ctypes.c_void_p(a.data_ptr()), n,  # noqa: E731
                              ctypes.c_void_p(b.data_ptr()), n, 0.5,
                              ctypes.c_void_p(c.data_ptr()), n)
            call()
            ms = timed(torch, call, FORM_CALLS)
            out[f"{p}gemm_{n}_{f}"] = round(2.0 * n ** 3 / ms / 1e9, 2)
        lib.mublis_b200_set_form(p.encode(), b"plain")
        del a, b, c
        torch.cuda.empty_cache()
    # DTRSM of order n with n right-hand sides: FP64 diagonal blocks, updates
    # plain or emulated (left, lower, non-unit; A = U[-1,1)/n off the
    # diagonal, U[1,2) on it).
    a = torch.empty(n, n, dtype=torch.float64, device="cuda")
    dg = torch.empty(n, n, dtype=torch.float64, device="cuda")
    b = torch.empty(n, n, dtype=torch.float64, device="cuda")
    lib.mublis_b200_fill_d(ctypes.c_void_p(a.data_ptr()), n, n, n, 0, 0, 0)
    lib.mublis_b200_fill_d(ctypes.c_void_p(dg.data_ptr()), n, n, n, 0, 9, 2)
    lib.mublis_b200_fill_d(ctypes.c_void_p(b.data_ptr()), n, n, n, 0, 1, 0)
    a.div_(n)
    a.diagonal().copy_(dg.diagonal())
    del dg
    b0 = b.clone()
    for f in ("plain", "ozaki2"):
        lib.mublis_b200_set_form(b"d", f.encode())
        call = lambda: lib.cblas_dtrsm(COL, LEFT, LOWER, NT, NONUNIT, n, n, 1.0,  # noqa: E731
                                       ctypes.c_void_p(a.data_ptr()), n,
                                       ctypes.c_void_p(b.data_ptr()), n)
        call()
        b.copy_(b0)
        ms = timed(torch, call, FORM_CALLS)
        b.copy_(b0)
        out[f"dtrsm_{n}_{f}"] = round(float(n) ** 3 / ms / 1e9, 2)
    lib.mublis_b200_set_form(b"d", b"plain")
    del a, b, b0
    torch.cuda.empty_cache()
    return out


def sides_study(torch, lib, n: int = 4096) -> dict:
    """TRSM and TRMM for every side x uplo x transpose at m = n (device
    operands, alpha 1, non-unit, A = U[0,1)/n + 1.5 I), TF/s credited with
    m^2 n; mean of 2 event-timed calls after a warm-up."""
    out = {}
    for p, dt in (("s", torch.float32), ("d", torch.float64)):
        a = torch.rand(n, n, dtype=dt, device="cuda") / n
        a.diagonal().add_(1.5)
        b0 = torch.rand(n, n, dtype=dt, device="cuda")
        b = b0.clone()
        for r in ("trsm", "trmm"):
            fn = getattr(lib, f"cblas_{p}{r}")
            for side, sname in ((LEFT, "left"), (LEFT + 1, "right")):
                for uplo, uname in ((LOWER, "lower"), (UPPER, "upper")):
                    for tr, tname in ((NT, "N"), (TR, "T")):
                        call = lambda: fn(COL, side, uplo, tr, NONUNIT, n, n, 1.0,  # noqa: E731
                                          ctypes.c_void_p(a.data_ptr()), n,
                                          ctypes.c_void_p(b.data_ptr()), n)
                        b.copy_(b0)
                        call()
                        ms = 0.0
                        for _ in range(2):
                            b.copy_(b0)
                            ms += timed(torch, call, 1)
                        out[f"{p}{r} {sname} {uname} {tname}"] = round(float(n) ** 3 / (ms / 2) / 1e9, 1)
        del a, b, b0
        torch.cuda.empty_cache()
    return out


def _log_uniform_int(rng, lo, hi, size):
    import numpy as np
    return np.floor(np.exp(rng.uniform(np.log(lo), np.log(hi + 1), size))).astype(int)


def _grouped_sgemms(torch, rng):
    """The grouped study's 4096 SGEMMs on the device: (problems, operand tensors, ctypes array)."""
    import mublis_b200 as mb
    torch.manual_seed(1)
    mnk = _log_uniform_int(rng, 16, 512, (4096, 3))
    ab = rng.uniform(0.5, 1.5, (4096, 2))
    probs, keep = [], []
    for q in range(4096):
        m, n, k = (int(x) for x in mnk[q])
        a = torch.rand(k, m, device="cuda") * 2 - 1
        b = torch.rand(n, k, device="cuda") * 2 - 1
        c = torch.rand(n, m, device="cuda") * 2 - 1
        probs.append(mb.GemmProblem(0, 0, m, n, k, ab[q, 0], ab[q, 1], a.data_ptr(), m,
                                    b.data_ptr(), k, c.data_ptr(), m))
        keep.append((a, b, c))
    return probs, keep, (mb.GemmProblem * len(probs))(*probs)


def grouped_direct(torch, lib, form: str = "plain") -> dict:
    """The grouped study's SGEMMs as direct grouped calls (no plan, no autotuning) in
    the given FP32 form: one warm-up call, then five timed (plain: three
    kernel launches per call, one per tile class; fp16x3: a pack and one
    tensor-core launch).  For profiler captures of the grouped kernels."""
    import numpy as np
    import mublis_b200 as mb
    probs, keep, arr = _grouped_sgemms(torch, np.random.default_rng(1))
    gflop = sum(2.0 * p.m * p.n * p.k for p in probs)
    mb.check(lib.mublis_b200_set_form(b"s", form.encode()), lib)
    mb.check(lib.mublis_b200_gemm_grouped(b"s", arr, len(probs)), lib)
    ms = timed(torch, lambda: lib.mublis_b200_gemm_grouped(b"s", arr, len(probs)), 5)
    lib.mublis_b200_set_form(b"s", b"plain")
    del keep
    return {"form": form, "gflop": round(gflop / 1e9, 2), "ms": round(ms, 3),
            "tflops": round(gflop / ms / 1e9, 2)}


def grouped_study(torch, lib) -> dict:
    """Grouped study: 4096 independent SGEMMs with m, n, k log-uniform over [16, 512]
    (seed 1), column-major, lda = m, per-problem alpha, beta uniform[0.5, 1.5);
    and 1024 DTRSMs (left, lower, non-unit) with order log-uniform in [32, 256],
    right-hand sides log-uniform in [1, 128], A off-diagonal uniform/n and
    diagonal in [1, 2).  One persistent grouped launch per plan (tiles
    autotuned, CUDA-graph replay) against one library call per problem."""
    import numpy as np
    import mublis_b200 as mb
    rng = np.random.default_rng(1)
    probs, keep, arr = _grouped_sgemms(torch, rng)
    gflop = sum(2.0 * p.m * p.n * p.k for p in probs)
    plan = ctypes.c_void_p()
    mb.check(lib.mublis_b200_plan_gemm_grouped(b"s", arr, len(probs), ctypes.byref(plan)), lib)
    ms_plan = timed(torch, lambda: lib.mublis_b200_plan_run(plan), 10)
    lib.mublis_b200_plan_destroy(plan)
    # The same group on the tensor cores (FP32 form fp16x3: tc_grouped.cu).
    lib.mublis_b200_set_form(b"s", b"fp16x3")
    plan = ctypes.c_void_p()
    mb.check(lib.mublis_b200_plan_gemm_grouped(b"s", arr, len(probs), ctypes.byref(plan)), lib)
    ms_tc = timed(torch, lambda: lib.mublis_b200_plan_run(plan), 10)
    lib.mublis_b200_set_form(b"s", b"plain")

    def loop():
        for p in probs:
            lib.mublis_sgemm(0, 0, p.m, p.n, p.k, p.alpha, p.a, 1, p.lda, p.b, 1, p.ldb, p.beta,
                             p.c, 1, p.ldc)
    ms_loop = timed(torch, loop, 2)
    lib.mublis_b200_plan_destroy(plan)
    del keep
    orders = _log_uniform_int(rng, 32, 256, 1024)
    nrhs = _log_uniform_int(rng, 1, 128, 1024)
    tp, tk = [], []
    for q in range(1024):
        m, n = int(orders[q]), int(nrhs[q])
        a = (torch.rand(m, m, dtype=torch.float64, device="cuda") * 2 - 1) / m
        a.diagonal().copy_(torch.rand(m, dtype=torch.float64, device="cuda") + 1)
        b = torch.rand(n, m, dtype=torch.float64, device="cuda") * 2 - 1
        tp.append(mb.TrsmProblem(mb.M_LOWER, 0, mb.M_NON_UNIT, m, n, 1.0, a.data_ptr(), m,
                                 b.data_ptr(), m))
        tk.append((a, b))
    tflop = sum(float(p.m) ** 2 * p.n for p in tp)
    tarr = (mb.TrsmProblem * len(tp))(*tp)
    tplan = ctypes.c_void_p()
    mb.check(lib.mublis_b200_plan_trsm_grouped(b"d", tarr, len(tp), ctypes.byref(tplan)), lib)
    ms_tplan = timed(torch, lambda: lib.mublis_b200_plan_run(tplan), 10)

    def tloop():
        for p in tp:
            lib.mublis_dtrsm(0, p.uplo, 0, 0, p.m, p.n, 1.0, p.a, 1, p.lda, p.b, 1, p.ldb)
    ms_tloop = timed(torch, tloop, 2)
    lib.mublis_b200_plan_destroy(tplan)
    del tk
    torch.cuda.empty_cache()
    return {"sgemm_x4096": {"gflop": round(gflop / 1e9, 2), "grouped_ms": round(ms_plan, 3),
                            "grouped_tflops": round(gflop / ms_plan / 1e9, 2),
                            "grouped_fp16x3_ms": round(ms_tc, 3),
                            "grouped_fp16x3_tflops": round(gflop / ms_tc / 1e9, 2),
                            "one_call_per_launch_ms": round(ms_loop, 2),
                            "speedup": round(ms_loop / ms_plan, 1)},
            "dtrsm_x1024": {"gflop": round(tflop / 1e9, 3), "grouped_ms": round(ms_tplan, 3),
                            "one_call_per_launch_ms": round(ms_tloop, 2),
                            "speedup": round(ms_tloop / ms_tplan, 1)}}


def served_study(torch, lib, nreq: int = 4000, ring: int = 8) -> dict:
    """Served study: 16 host threads issue cblas calls with Poisson arrivals
    (aggregate 20k calls/s, seed 2); mix 60% SGEMM, 20% DGEMM, 10% SSYRK, 10%
    DTRSM; 80% of sizes log-uniform in [32, 256], 20% from {1024, 2048, 4096,
    8192}; operands device-resident in server handles under a 64 GiB HBM
    budget.  `nreq` requests (the large ones carry ~99% of the flops, so the
    run is throughput-bound for several seconds).

    Three runs of the same requests at the same arrival times: serialized
    plain calls (one at a time, no server), the request server with plain
    forms (the batching / overlap gain alone), and the server with "auto"
    forms (adding the tensor-core precision forms).  Latency = completion -
    scheduled arrival.

    Operands: every small request owns its handles; the large requests of one
    (kind, size) share their read-only operands and take their output (C, or
    B for TRSM) from a ring of `ring` handles, so that 4000 requests fit the
    64 GiB budget.  Outputs of large requests may therefore be overwritten by
    a later request of the same class while both are in flight: this study
    measures throughput and latency only; that each result is the same alone
    and in the mix is tests/test_gpu_serve.py's."""
    import threading
    import numpy as np
    import mublis_b200 as mb
    rng = np.random.default_rng(2)
    arrivals = np.cumsum(rng.exponential(1 / 20000.0, nreq))
    kinds = rng.choice(["sgemm", "dgemm", "ssyrk", "dtrsm"], p=[0.6, 0.2, 0.1, 0.1], size=nreq)
    cfg = mb.ServerConfig(hbm_budget_bytes=64 << 30, streams=4, batch_window_us=100,
                          small_max_dim=512, max_batch=4096, sform=None, dform=None)
    srv = ctypes.c_void_p()
    mb.check(lib.mublis_b200_server_create(ctypes.byref(cfg), ctypes.byref(srv)), lib)
    reqs, extra, pools = [], [], {}
    try:
        def handle(rows, cols, elt, p, seed, mid, kind=0):
            d = ctypes.c_void_p()
            mb.check(lib.mublis_b200_server_alloc(srv, rows * cols * elt, ctypes.byref(d)), lib)
            mb.check(getattr(lib, f"mublis_b200_fill_{p}")(d, rows, cols, rows, seed, mid, kind), lib)
            return d.value

        def trsm_operand(m, seed):  # well-conditioned triangle
            a = torch.empty(m, m, dtype=torch.float64, device="cuda")
            dg = torch.empty(m, m, dtype=torch.float64, device="cuda")
            lib.mublis_b200_fill_d(ctypes.c_void_p(a.data_ptr()), m, m, m, seed, 0, 0)
            lib.mublis_b200_fill_d(ctypes.c_void_p(dg.data_ptr()), m, m, m, seed, 9, 2)
            a.div_(m)
            a.diagonal().copy_(dg.diagonal())
            extra.append(a)
            return a.data_ptr()

        for q in range(nreq):
            large = rng.random() >= 0.8
            if large:
                m = n = k = int(rng.choice([1024, 2048, 4096, 8192]))
            else:
                m, n, k = (int(x) for x in np.floor(np.exp(rng.uniform(np.log(32), np.log(257), 3))))
            kind = kinds[q]
            p = kind[0]
            elt = 4 if p == "s" else 8
            if kind.endswith("gemm"):
                shapes, fl = [(m, k), (k, n), (m, n)], 2.0 * m * n * k
            elif kind == "ssyrk":
                m = n
                shapes, fl = [(n, k), (n, n)], float(n) * (n + 1) * k
            else:
                shapes, fl = [(m, m), (m, n)], float(m) * m * n
            if large:
                key = (kind, m)
                if key not in pools:
                    ins = [handle(r, c, elt, p, 1000 + len(pools), i) for i, (r, c) in
                           enumerate(shapes[:-1])]
                    if kind == "dtrsm":
                        ins[0] = trsm_operand(m, 1000 + len(pools))
                    r, c = shapes[-1]
                    outs = [handle(r, c, elt, p, 2000 + len(pools), t) for t in range(ring)]
                    pools[key] = (ins, outs, [0])
                ins, outs, nxt = pools[key]
                ptrs = ins + [outs[nxt[0] % ring]]
                nxt[0] += 1
            else:
                ptrs = [handle(r, c, elt, p, q, i) for i, (r, c) in enumerate(shapes)]
                if kind == "dtrsm":
                    ptrs[0] = trsm_operand(m, q)
            reqs.append(dict(kind=kind, m=m, n=n, k=k, p=ptrs, fl=fl, at=float(arrivals[q])))
        torch.cuda.synchronize()
        P = ctypes.c_void_p

        def issue(r):
            k_, m, n, p = r["kind"], r["m"], r["n"], r["p"]
            if k_ == "sgemm":
                lib.cblas_sgemm(COL, NT, NT, m, n, r["k"], 0.75, P(p[0]), m, P(p[1]), r["k"], 0.25,
                                P(p[2]), m)
            elif k_ == "dgemm":
                lib.cblas_dgemm(COL, NT, NT, m, n, r["k"], 0.75, P(p[0]), m, P(p[1]), r["k"], 0.25,
                                P(p[2]), m)
            elif k_ == "ssyrk":
                lib.cblas_ssyrk(COL, LOWER, NT, n, r["k"], 0.75, P(p[0]), n, 0.25, P(p[1]), n)
            else:
                lib.cblas_dtrsm(COL, LEFT, LOWER, NT, NONUNIT, m, n, 0.75, P(p[0]), m, P(p[1]), m)

        def set_forms(form):
            for pp in (b"s", b"d"):
                lib.mublis_b200_set_form(pp, form)

        def serial(count):
            set_forms(b"plain")
            lat = [0.0] * count
            t0 = time.perf_counter()
            for q in range(count):
                target = t0 + reqs[q]["at"]
                while time.perf_counter() < target:
                    pass
                issue(reqs[q])
                lat[q] = time.perf_counter() - target
            return lat, time.perf_counter() - t0

        def served(count, form):
            set_forms(form)
            lib.mublis_b200_server_attach(srv)
            lib.mublis_b200_server_reset_stats(srv)
            lat = [0.0] * count
            t0 = time.perf_counter() + 0.05

            def worker(t):
                for q in range(t, count, 16):
                    target = t0 + reqs[q]["at"]
                    while time.perf_counter() < target:
                        pass
                    issue(reqs[q])
                    lat[q] = time.perf_counter() - target
            ths = [threading.Thread(target=worker, args=(t,)) for t in range(16)]
            for th in ths:
                th.start()
            for th in ths:
                th.join()
            span = time.perf_counter() - t0
            lib.mublis_b200_server_attach(None)
            st = mb.ServerStats()
            lib.mublis_b200_server_stats(srv, ctypes.byref(st))
            return lat, span, st

        # Warm-up of every path on the first 400 requests (module loads,
        # tuned tiles, pools), then the timed runs over all of them.
        warm = min(400, nreq)
        serial(warm)
        served(warm, b"plain")
        served(warm, b"auto")
        lat_s, span_s = serial(nreq)
        lat_p, span_p, st_p = served(nreq, b"plain")
        lat_v, span_v, st_v = served(nreq, b"auto")
        tot = sum(r["fl"] for r in reqs)
        pct = lambda l, q: round(float(np.percentile(l, q)) * 1e3, 2)  # noqa: E731

        def run(lat, span, st=None, forms=None):
            d = {"tflops": round(tot / span / 1e12, 2), "span_s": round(span, 3),
                 "p50_ms": pct(lat, 50), "p99_ms": pct(lat, 99)}
            if st is not None:
                d.update(batches=int(st.batches), batched_requests=int(st.batched_requests),
                         forms=forms)
            return d
        return {"requests": nreq, "arrival_span_s": round(float(arrivals[-1]), 3),
                "tflop": round(tot / 1e12, 2),
                "serialized_plain": run(lat_s, span_s),
                "served_plain": run(lat_p, span_p, st_p, "plain"),
                "served": run(lat_v, span_v, st_v,
                              "auto (fp16x3 / bf16x6 / ozaki2 above crossover, else plain)"),
                "batching_ratio_plain": round(span_s / span_p, 2),
                "throughput_ratio": round(span_s / span_v, 2)}
    finally:
        lib.mublis_b200_server_attach(None)
        lib.mublis_b200_server_destroy(srv)
        for pp in (b"s", b"d"):
            lib.mublis_b200_set_form(pp, b"plain")
        del extra
        torch.cuda.empty_cache()


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="mublis", choices=["mublis", "reference"])
    ap.add_argument("--n", type=int, default=4096)
    ap.add_argument("--no-forms", action="store_true", help="skip the 8192 precision-form study")
    ap.add_argument("--no-cpu", action="store_true", help="skip the CPU baseline")
    ap.add_argument("--no-studies", action="store_true",
                    help="skip the grouped (4096 small GEMMs) and served (4000-request mix) studies")
    ap.add_argument("--only-forms", action="store_true",
                    help="run only the precision-form study (for profiler captures)")
    ap.add_argument("--forms-n", type=int, default=8192)
    ap.add_argument("--only-sides", action="store_true",
                    help="run only the TRSM/TRMM side x uplo x transpose study")
    ap.add_argument("--only-grouped", action="store_true",
                    help="run only the grouped study's SGEMMs as direct grouped calls (profiler captures)")
    ap.add_argument("--grouped-form", default="plain", choices=["plain", "fp16x3"],
                    help="FP32 form of --only-grouped")
    ap.add_argument("--only-trsm", default=None, choices=["s", "d"],
                    help="run only two TRSMs of order --n with --n right-hand sides "
                         "(left, lower, non-unit; profiler captures of the TRSM kernels)")
    ap.add_argument("--only-timed", action="store_true",
                    help="warm-up + timed steps only (for profiler launch lists)")
    args = ap.parse_args()
    args.warmup = max(args.warmup, 3)

    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if args.impl == "reference":
        run_reference_arm(args, rank, world)
        return

    import torch
    import torch.distributed as dist

    import mublis_b200 as mb

    torch.cuda.set_device(local)
    if world > 1:
        import datetime
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120),
                                device_id=torch.device("cuda", local))
    lib = mb.load()
    mb.check(lib.mublis_b200_init(), lib)
    for p in (b"s", b"d"):
        lib.mublis_b200_set_form(p, b"plain")
    stream = torch.cuda.current_stream()
    mb.check(lib.mublis_b200_set_stream(ctypes.c_void_p(stream.cuda_stream)), lib)

    if args.only_sides:
        if rank == 0:
            print(json.dumps({"sides_tflops": sides_study(torch, lib, args.n), "n": args.n}))
        return

    if args.only_trsm:
        if rank == 0:
            p = args.only_trsm
            dt = torch.float32 if p == "s" else torch.float64
            n = args.n
            a = torch.empty(n, n, dtype=dt, device="cuda")
            getattr(lib, f"mublis_b200_fill_{p}")(ctypes.c_void_p(a.data_ptr()), n, n, n, 0, 0, 0)
            a.div_(n)
            a.diagonal().add_(1.5)
            b = torch.rand(n, n, dtype=dt, device="cuda")
            fn = getattr(lib, f"mublis_{p}trsm")
            for _ in range(2):
                mb.check(fn(0, 1, 0, 0, n, n, 1.0, a.data_ptr(), 1, n, b.data_ptr(), 1, n), lib)
            torch.cuda.synchronize()
            print(json.dumps({"trsm": p, "n": n, "ok": True}))
        return

    if args.only_grouped:
        if rank == 0:
            print(json.dumps({"grouped_direct": grouped_direct(torch, lib, args.grouped_form)}))
        return

    if args.only_forms:
        if rank == 0:
            print(json.dumps({"forms_tflops": forms_study(torch, lib, args.forms_n),
                              "n": args.forms_n}))
        return

    n = args.n
    fam = Family(torch, lib, n, device=True)
    for _ in range(args.warmup):
        fam.step()
    torch.cuda.synchronize()

    gpu_index = int(os.environ.get("CUDA_VISIBLE_DEVICES", str(local)).split(",")[0]) \
        if os.environ.get("CUDA_VISIBLE_DEVICES", "").split(",")[0].isdigit() else local
    sampler = ClockSampler(gpu_index)
    time.sleep(0.3)
    if world > 1:
        dist.barrier()
    launches0 = lib.mublis_b200_launch_count()
    lib.mublis_b200_profile_enable(1)
    ms = timed(torch, fam.step, args.steps)
    lib.mublis_b200_profile_enable(0)
    launches = lib.mublis_b200_launch_count() - launches0
    if world > 1:
        dist.barrier()
    clocks = sampler.stop()
    buf = ctypes.create_string_buffer(1 << 16)
    lib.mublis_b200_profile_read(buf, len(buf))
    kstats = json.loads(buf.value.decode() or "{}")

    ms = max_over_ranks(dist, torch, ms, world)
    value = whole_job_tflops(family_flops(n), world, ms)

    # per-routine breakdown (untimed by the headline; one pass, event per call)
    if args.only_timed:
        args.no_forms = args.no_cpu = args.no_studies = True
    breakdown = {}
    if rank == 0 and not args.only_timed:
        for (p, r, ops), _ in zip(fam.calls, range(len(fam.calls))):
            single = Family.__new__(Family)
            single.lib, single.n, single.calls = lib, n, [(p, r, ops)]
            t1 = timed(torch, single.step, 1)
            breakdown[f"{p}{r}"] = round(flops(r, n) / (t1 * 1e-3) / 1e12, 2)

    verified = None
    if rank == 0 and not args.only_timed:
        verified = verify_step(torch, fam)

    # roofline of the dominant kernel
    roof = None
    if kstats and rank == 0:
        dom = max(kstats, key=lambda k: kstats[k][1])
        launches_k, total_ms = kstats[dom]
        kf = kernel_flops(n).get(dom)
        peaks = measured_peaks()
        if kf is not None:
            per_launch = kf * args.steps / launches_k
            avg_ms = total_ms / launches_k
            achieved = per_launch / (avg_ms * 1e-3) / 1e12
            is64 = dom.endswith("d") or "dgemm" in dom
            tensor = dom.startswith("dmma")
            peak = FP64_NOMINAL_TFLOPS if is64 else FP32_NOMINAL_TFLOPS
            traffic = profile_traffic(dom)
            if tensor:
                bound = "tensor"
                source = ("nominal FP64 tensor pipe (MEASURED_PEAKS.json has no FP64 figure): "
                          "148 SMs x 64 FP64 FMA/clk x 2 x 1965 MHz; a register-only "
                          "mma.sync m16n8k4 .f64 loop reaches 37.0 TF/s on this B200")
            else:
                bound = "fp64_fma_pipe" if is64 else "fp32_fma_pipe"
                source = ("nominal (no FMA-pipe peak in MEASURED_PEAKS.json): 148 SMs x "
                          + ("64 FP64" if is64 else "128 FP32") + " FMA lanes x 2 x 1965 MHz")
            roof = {"kernel": dom, "bound": bound,
                    "achieved": round(achieved, 3), "peak": round(peak, 2), "unit": "TFLOP/s",
                    "frac": round(achieved / peak, 4),
                    "peak_source": source,
                    "traffic": traffic, "launches_per_step": launches_k / args.steps,
                    "share_of_step": round(total_ms / args.steps / ms, 4),
                    "bf16_tflops_measured": peaks.get("bf16_tflops"),
                    "hbm_gbs_measured": peaks.get("hbm_gbs")}

    # end to end through cblas_* with pinned host buffers
    e2e = None
    if not args.only_timed:
        del fam
        torch.cuda.empty_cache()
        hfam = Family(torch, lib, n, device=False)
        hfam.step()
        e2e_ms = max_over_ranks(dist, torch, timed(torch, hfam.step, max(2, min(args.steps, 3))),
                                world)
        e2e = {"value": round(whole_job_tflops(family_flops(n), world, e2e_ms), 3),
               "unit": "TFLOP/s",
               "ms_per_step": round(e2e_ms, 3), "h2d_bytes_per_step": hfam.h2d,
               "d2h_bytes_per_step": hfam.d2h, "api": "cblas_* with pinned host buffers"}
        if rank == 0:
            per = {}
            for call in hfam.calls:
                single = Family.__new__(Family)
                single.lib, single.n, single.calls = lib, n, [call]
                per[f"{call[0]}{call[1]}"] = round(timed(torch, single.step, 1), 3)
            e2e["ms_per_call"] = per
        del hfam

    forms = None
    if rank == 0 and world == 1 and not args.no_forms:
        fsampler = ClockSampler(gpu_index)
        forms = forms_study(torch, lib, args.forms_n)
        forms["clocks"] = fsampler.stop()
    grouped = served = None
    if rank == 0 and world == 1 and not args.no_studies:
        grouped = grouped_study(torch, lib)
        served = served_study(torch, lib)

    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu:
        try:
            threads = host_threads()
            r = ref_bench(n, threads, 1, 0, mode="family_par", panel=512)
            r1 = ref_bench(2048, 1, 1, 0)  # one call at a time on one core
            cpu = {"value": round(r["gflops_aggregate"] / 1e3, 4), "unit": "TFLOP/s",
                   "cores": threads, "kind": "reference",
                   "sample": par_sample(n, threads, 512) + f"; one step, wall {r['wall_s']:.1f} s",
                   "one_thread": {"value": round(r1["gflops_aggregate"] / 1e3, 4),
                                  "unit": "TFLOP/s", "cores": 1,
                                  "sample": f"the 18-call family at m=n=k=2048, one pass on one "
                                            f"thread, wall {r1['wall_s']:.1f} s"}}
        except Exception as e:  # noqa: BLE001
            cpu = {"value": None, "unavailable": str(e)}

    if rank == 0:
        line = {"metric": METRIC, "value": round(value, 3), "unit": "TFLOP/s", "n_gpus": world,
                "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(ms, 3),
                "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
                "dtype": "f32+f64", "data": "synthetic: seeded Philox uniform[-1,1); TRSM/TRMM "
                "A off-diagonal uniform/n, diagonal uniform[1,2)",
                "config": workload_config(n), "e2e": e2e, "roofline": roof, "cpu_baseline": cpu,
                "clocks": clocks, "gpu_launches": int(launches), "breakdown_tflops": breakdown,
                "verified": verified,
                "stated_err": "normwise relative error <= 4*k*u against the oracle "
                              "(tests/test_gpu_family_n4096.py checks this workload's 18 calls); "
                              "measured plain SGEMM ~1.9e-8, DGEMM ~3.4e-17 at 8192",
                "forms_8192_tflops": forms, "grouped_study": grouped, "served_study": served,
                "kernels_ms_per_step": {k: round(v[1] / args.steps, 4) for k, v in kstats.items()}}
        print(json.dumps(line))
    if world > 1:
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
