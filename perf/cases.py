"""The calls this framework's performance is measured on, and how to make them.

Each case is one call through a public entry point, C += A * B with operands already where the
caller keeps them:

  gemm    runtime.fmm_gemm / runtime.plain_gemm: one FP64 problem on device tensors, any
          algorithm of the generator and the three pack types (abc, ab, naive)
  split   runtime.split_gemm: FP32 operands, FP64 C, products on the bf16 tensor cores
  batch   runtime.Batch.run: independent FP64 problems planned once, run again and again
  submit  runtime.batch_submit: a batch formed, run and released in one call (request loops)
  host    runtime.fmm_gemm_host / runtime.bl_dgemm_host: the drop-in form, host matrices in and
          out, pinned

Sizes come from the sweep families (square 240 .. 12000, rank-k 14400 x 14400 x k), the
benchmark's workloads (2048^3, 16384^3, 14400 x 14400 x 480, split 8192^3, 512 problems with
dimensions log-uniform in [256, 4096]) and ragged sizes like those of the parity tests.
C keeps accumulating when a case runs again on the same state, as in a caller's loop.
"""
import math
import random

import numpy as np
import torch

from fmm_gen_b200 import algebra, ops, runtime as rt

DEV = "cuda"
BATCH_DIMS = (256, 4096)     # dimension range of the batch and request workloads
BATCH_FMM_MIN = 1200         # batch problems at least this large in every dimension take 222-1


def listed():
    return [
        # the first size of the square sweep: one small call, launch latency and few work units
        {"name": "strassen_240", "kind": "gemm", "alg": "222-1", "pack": "abc", "m": 240, "n": 240, "k": 240},
        # the classical comparator at a small odd size (odd leading dimensions)
        {"name": "plain_odd_701", "kind": "gemm", "alg": "classical", "pack": "abc", "m": 701, "n": 503, "k": 615},
        # an ordinary call whose dimensions leave every fringe
        {"name": "strassen_ragged_1501", "kind": "gemm", "alg": "222-1", "pack": "abc", "m": 1501, "n": 1203, "k": 999},
        # one-level Strassen at the benchmark's small square size
        {"name": "strassen_2048", "kind": "gemm", "alg": "222-1", "pack": "abc", "m": 2048, "n": 2048, "k": 2048},
        # the ab pack type (products kept in a workspace), two levels, a rectangular problem
        {"name": "two_level_ab_4200", "kind": "gemm", "alg": "222-2", "pack": "ab", "m": 3600, "n": 4200, "k": 2900},
        # the two-level hybrid on a rank-k update: little k per product, C traffic
        {"name": "hybrid_rankk_14400", "kind": "gemm", "alg": "222-1_333-1", "pack": "abc", "m": 14400, "n": 14400,
         "k": 480},
        # the two-level hybrid at the benchmark's largest square size
        {"name": "hybrid_16384", "kind": "gemm", "alg": "222-1_333-1", "pack": "abc", "m": 16384, "n": 16384,
         "k": 16384},
        # a mid-size ragged FP32 request
        {"name": "split_ragged_3007", "kind": "split", "alg": "222-1", "m": 1021, "n": 3007, "k": 1530},
        # the benchmark's FP32 problem
        {"name": "split_8192", "kind": "split", "alg": "222-2", "m": 8192, "n": 8192, "k": 8192},
        # the 512-problem batch, planned once
        {"name": "batch_512", "kind": "batch", "count": 512, "shapes": 0},
        # one step of a request loop: a fresh batch of two dozen mixed requests
        {"name": "submit_24", "kind": "submit", "count": 24, "shapes": 1},
        # a host program calling the drop-in form
        {"name": "host_2880", "kind": "host", "alg": "222-1", "pack": "abc", "m": 2400, "n": 2880, "k": 1920},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dims(rng, lo, hi):
    """(m, n, k): square, rank-k like or unrelated dimensions; half of them ragged, the others
    whole multiples of 8 or of the sweep's step of 48 (240 = 5 * 48)."""
    unit = rng.choice((1, 1, 8, 48))

    def size(a, b):
        return max(unit, _log_int(rng, a, b) // unit * unit)

    shape = rng.choice(("square", "rankk", "any"))
    if shape == "square":
        s = size(lo, hi)
        return s, s, s
    if shape == "rankk":
        s = size(2 * lo, hi)
        return s, s, size(max(64, lo // 4), min(1024, hi))
    return size(lo, hi), size(lo, hi), size(lo, hi)


def draw(rng):
    kind = rng.choices(("gemm", "split", "batch", "submit", "host"), (10, 4, 2, 2, 2))[0]
    if kind == "gemm":
        alg = rng.choice(("classical", "222-1", "222-1", "232-1", "333-1", "222-2", "222-1_333-1"))
        pack = "abc" if alg == "classical" else rng.choice(("abc", "abc", "abc", "ab", "naive"))
        m, n, k = _dims(rng, 240, 12000)
        return {"kind": kind, "alg": alg, "pack": pack, "m": m, "n": n, "k": k}
    if kind == "split":
        m, n, k = _dims(rng, 256, 8192)
        return {"kind": kind, "alg": rng.choice(("classical", "222-1", "222-2")), "m": m, "n": n, "k": k}
    if kind == "host":
        m, n, k = _dims(rng, 240, 4096)
        return {"kind": kind, "alg": rng.choice(("classical", "222-1", "222-2")), "pack": "abc", "m": m, "n": n, "k": k}
    return {"kind": kind, "count": _log_int(rng, *((16, 512) if kind == "batch" else (2, 64))),
            "shapes": rng.randrange(2, 1 << 30)}


def _plan(alg):
    return None if alg == "classical" else ops.plan_for(alg)


def _problems(case):
    """[(algorithm, m, n, k)] of a batch or submit case."""
    r = random.Random(case["shapes"])
    out = []
    for _ in range(case["count"]):
        m, n, k = (_log_int(r, *BATCH_DIMS) for _ in range(3))
        out.append(("222-1" if min(m, n, k) >= BATCH_FMM_MIN else "classical", m, n, k))
    return out


def _arena(shapes, gen):
    """Column-major FP64 matrices, U(-1, 1), in one allocation; each starts on 256 bytes."""
    offs, total = [], 0
    for r, c in shapes:
        offs.append(total)
        total += (r * c + 31) // 32 * 32
    flat = torch.empty(total, dtype=torch.float64, device=DEV).uniform_(-1, 1, generator=gen)
    return flat, [flat[o:o + r * c].view(c, r).t() for o, (r, c) in zip(offs, shapes)]


def _operands(case, seed):
    """Device operands of any case, from the seed alone: A, B, C (lists for batches, plus the
    flat allocation that holds every C)."""
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    if case["kind"] in ("batch", "submit"):
        shapes = _problems(case)
        _, As = _arena([(m, k) for _, m, _, k in shapes], gen)
        _, Bs = _arena([(k, n) for _, _, n, k in shapes], gen)
        flat, Cs = _arena([(m, n) for _, m, n, _ in shapes], gen)
        return As, Bs, Cs, flat
    m, n, k = case["m"], case["n"], case["k"]
    if case["kind"] == "split":
        A = rt.colmajor(m, k, dtype=torch.float32, device=DEV).normal_(generator=gen)
        B = rt.colmajor(k, n, dtype=torch.float32, device=DEV).normal_(generator=gen)
    else:
        A = rt.colmajor(m, k, device=DEV).uniform_(-1, 1, generator=gen)
        B = rt.colmajor(k, n, device=DEV).uniform_(-1, 1, generator=gen)
    C = rt.colmajor(m, n, device=DEV).uniform_(-1, 1, generator=gen)
    return A, B, C, None


def _pinned(x):
    """A pinned host copy of a column-major device matrix, as a Fortran-ordered array."""
    host = torch.empty((x.shape[1], x.shape[0]), dtype=x.dtype, pin_memory=True)
    host.copy_(x.t())
    return host.numpy().T, host


def prepare(case, seed):
    A, B, C, flat = _operands(case, seed)
    s = {"case": case}
    if case["kind"] in ("batch", "submit"):
        shapes = _problems(case)
        s["plans"] = [_plan(alg) for alg, _, _, _ in shapes]
        s.update(A=A, B=B, C=C, flat=flat)
        if case["kind"] == "batch":
            s["batch"] = rt.Batch([p[1:] for p in shapes], s["plans"])
        return s
    s["plan"] = _plan(case["alg"])
    if case["kind"] == "host":
        (s["A"], a), (s["B"], b), (s["C"], c) = _pinned(A), _pinned(B), _pinned(C)
        s["keep"] = (a, b, c)
        return s
    s.update(A=A, B=B, C=C)
    return s


def run(state):
    kind, A, B, C = state["case"]["kind"], state["A"], state["B"], state["C"]
    if kind == "batch":
        state["batch"].run(A, B, C)
        return state["flat"]
    if kind == "submit":
        rt.batch_submit(state["plans"], A, B, C)
        return state["flat"]
    plan = state["plan"]
    if kind == "split":
        rt.split_gemm(plan, A, B, C)
    elif kind == "host":
        if plan is None:
            rt.bl_dgemm_host(A, B, C)
        else:
            rt.fmm_gemm_host(plan, A, B, C, state["case"]["pack"])
    elif plan is None:
        rt.plain_gemm(A, B, C)
    else:
        rt.fmm_gemm(plan, A, B, C, state["case"]["pack"])
    return C


_MULTS = {}


def _mult_flops(alg, m, n, k):
    """Multiply-add flops of the algorithm: its R products on the core, classical fringes."""
    if alg == "classical":
        return 2.0 * m * n * k
    if alg not in _MULTS:
        p = algebra.make_plan(*ops.parse_levels(alg))
        _MULTS[alg] = (p.dims, p.rank)
    (dm, dk, dn), rank = _MULTS[alg]
    md, kd, nd = m - m % (8 * dm), k - k % dk, n - n % (4 * dn)
    core = float(md) * nd * kd
    return 2.0 * (core * rank / (dm * dk * dn) + float(m) * n * k - core)


def work(case):
    if case["kind"] in ("batch", "submit"):
        ps = _problems(case)
        return {"bytes": sum(8.0 * (m * k + k * n + 2 * m * n) for _, m, n, k in ps),
                "flops": sum(_mult_flops(a, m, n, k) for a, m, n, k in ps)}
    m, n, k = case["m"], case["n"], case["k"]
    split = case["kind"] == "split"  # FP32 operands, six bf16 plane products per product
    return {"bytes": (4.0 if split else 8.0) * (m * k + k * n) + 16.0 * m * n,
            "flops": (6.0 if split else 1.0) * _mult_flops(case["alg"], m, n, k)}


def exact(case, seed):
    A, B, C, flat = _operands(case, seed)
    if case["kind"] in ("batch", "submit"):
        for a, b, c in zip(A, B, C):
            c.add_(a @ b)
        return flat
    C.add_(A.double() @ B.double())
    return C.cpu().numpy() if case["kind"] == "host" else C
