"""The work that users of the library have it do, as cases that can be timed.

A case is a dict of plain values; its "kind" names the public entry point:

  commit    CommitPlan.run + results: the circle LDE of a device-resident trace, the
            row-leaf Merkle tree with the gamma combination, the committed fold chain
  lde       circle_lde_noalloc: one circle low-degree extension between caller-owned
            device buffers
  fft       circle_fft / circle_ifft on host arrays (the reference's GPU entry points)
  prove     prove: one proof from wire bytes on the host (SeededFib, the AND-table lookup
            AIR, stacked Rescue, the linear layer)
  batch     prove_batch: independent proofs of mixed AIRs and sizes over several streams
  columns   commit_columns: the prover's per-column commitment alone
  binius    binius_prove_combination: a combination sum-check over GF(2^8) or GF(2^128)

Every output is a whole number or a byte, so no case has a value in floating point.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "zig-stark_b200"))

from zs_b200 import native, wire  # noqa: E402
from zs_b200 import workload as wl  # noqa: E402

P = 2**31 - 1
# The sum-check instance: t0 t1 t2 + 2 t0 over three tables.
TERMS = [([0, 1, 2], 1), ([0], 2)]
AIRS = {"fib": wl.AIR_SEEDED_FIB, "and_table": wl.AIR_AND_TABLE, "rescue": wl.AIR_RESCUE_STACKED,
        "ml_linear": wl.AIR_ML_LINEAR}
QUERIES, REMAINDER_LOG = 16, 3


def listed():
    return [
        # the smallest commits (a few columns, every launch short): latency and launches
        {"name": "commit 8x2^10", "kind": "commit", "columns": 8, "log_rows": 10, "log_blowup": 2, "folds": 6},
        # an ordinary trace with a ragged column count and the larger blowup
        {"name": "commit 37x2^15 b8", "kind": "commit", "columns": 37, "log_rows": 15, "log_blowup": 3, "folds": 12},
        # the headline workload: 64 columns of 2^20 rows, blowup 4, 16 folds
        {"name": "commit 64x2^20", "kind": "commit", "columns": 64, "log_rows": 20, "log_blowup": 2, "folds": 16},
        # a plugin's in-place extension of a few columns in its own device buffers
        {"name": "lde 5x2^16", "kind": "lde", "columns": 5, "log_rows": 16, "log_blowup": 2},
        # interpolation of one batch of columns from host arrays
        {"name": "ifft 12x2^16", "kind": "fft", "inverse": True, "columns": 12, "log_n": 16},
        # the smallest proof served: a 2^12-row Fibonacci trace, bound by latency
        {"name": "prove fib 2^12", "kind": "prove", "air": "fib", "log_rows": 12, "log_blowup": 2},
        # a lookup AIR (preprocessed and LogUp columns) at an ordinary size and blowup 8
        {"name": "prove and_table 2^14 b8", "kind": "prove", "air": "and_table", "log_rows": 14, "log_blowup": 3},
        # a large proof: 2^15 stacked Rescue permutations
        {"name": "prove rescue 2^18", "kind": "prove", "air": "rescue", "log_rows": 18, "log_blowup": 2},
        # a wide proof: the 128 x 128 linear layer, 387 committed columns
        {"name": "prove ml_linear 2^15", "kind": "prove", "air": "ml_linear", "log_rows": 15, "log_blowup": 2},
        # a prover node working through a queue of mixed requests
        {"name": "batch 24 of 2^10..2^17", "kind": "batch", "jobs": 24, "log_min": 10, "log_max": 17, "workers": 8},
        # the sum-check provers: bytes over many rows, 128-bit elements over fewer
        {"name": "binius gf8 2^22", "kind": "binius", "bits": 8, "log_rows": 22},
        {"name": "binius gf128 2^16", "kind": "binius", "bits": 128, "log_rows": 16},
    ]


def draw(rng):
    kind = rng.choice(["commit"] * 3 + ["prove"] * 4 + ["lde", "fft", "batch", "columns", "binius"])
    if kind == "commit":
        log_rows, log_blowup = rng.randint(8, 19), rng.randint(1, 3)
        top = min(100, max(1, (1 << 26) >> (log_rows + log_blowup)))
        columns = max(1, min(top, round(math.exp(rng.uniform(0, math.log(top + 0.49))))))
        return {"kind": kind, "columns": columns, "log_rows": log_rows, "log_blowup": log_blowup,
                "folds": rng.randint(4, min(16, log_rows + log_blowup))}
    if kind == "lde":
        log_rows, log_blowup = rng.randint(8, 17), rng.randint(1, 3)
        n, big = 1 << log_rows, 1 << (log_rows + log_blowup)
        top = max(1, min(64, ((1 << 22) - 2 * n - 2 * big) // (n + big)))
        return {"kind": kind, "columns": rng.randint(1, top), "log_rows": log_rows, "log_blowup": log_blowup} \
            if 2 * n + 2 * big + n + big <= 1 << 22 else draw(rng)
    if kind == "fft":
        log_n = rng.randint(6, 18)
        return {"kind": kind, "inverse": rng.random() < 0.5, "log_n": log_n,
                "columns": rng.randint(1, min(48, (1 << 22) >> log_n))}
    if kind == "prove":
        air = rng.choice(["fib", "fib", "and_table", "rescue", "rescue", "ml_linear"])
        low, high = {"fib": (10, 19), "and_table": (8, 15), "rescue": (8, 18), "ml_linear": (8, 13)}[air]
        return {"kind": kind, "air": air, "log_rows": rng.randint(low, high),
                "log_blowup": 2 if air == "ml_linear" else rng.choice([2, 2, 3])}
    if kind == "batch":
        log_min = rng.randint(8, 12)
        return {"kind": kind, "jobs": rng.randint(3, 24), "log_min": log_min, "log_max": rng.randint(log_min + 1, 16),
                "workers": rng.choice([4, 8, 16])}
    if kind == "columns":
        log_rows = rng.randint(8, 17)
        return {"kind": kind, "columns": rng.randint(1, min(24, (1 << 20) >> log_rows)), "log_rows": log_rows,
                "log_blowup": rng.randint(1, 3)}
    bits = rng.choice([8, 128])
    return {"kind": kind, "bits": bits, "log_rows": rng.randint(8, 22 if bits == 8 else 18)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _uniform(rng, *shape):
    return rng.integers(0, P, shape, dtype=np.uint32)


def _job(air, log_rows, log_blowup, seed):
    """(air id, params, public inputs, trace, preprocessed, separator) as wire bytes."""
    pre = b""
    if air == "fib":
        tr, pi = wl.seeded_fib(log_rows, seed)
    elif air == "rescue":
        tr, pi = wl.rescue_stacked(log_rows, seed)
    elif air == "and_table":
        tr, pre_cols = wl.and_table_trace(1 << log_rows)
        pi, pre = b"", wire.columns(pre_cols)
    else:
        tr, pre_cols, pi = wl.ml_linear(log_rows, seed)
        pre = wire.columns(pre_cols)
    params = wire.StarkParams(log_rows, log_blowup, QUERIES, REMAINDER_LOG).encode()
    return AIRS[air], params, pi, wire.columns(tr), pre, b"zs-perf:%d" % seed


def _batch_shapes(case):
    """The batch's AIRs and sizes, the same for every seed."""
    rng = np.random.default_rng([case["jobs"], case["log_min"], case["log_max"]])
    return [("fib" if rng.random() < 0.5 else "rescue", int(rng.integers(case["log_min"], case["log_max"] + 1)))
            for _ in range(case["jobs"])]


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    if kind == "commit":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        trace = torch.randint(0, P, (case["columns"], 1 << case["log_rows"]), generator=gen, device="cuda",
                              dtype=torch.int32)
        plan = native.CommitPlan(case["columns"], case["log_rows"], case["log_blowup"], case["folds"])
        plan.set_challenges(_uniform(rng, case["columns"], 4), _uniform(rng, case["folds"], 4))
        torch.cuda.synchronize()  # the plan runs on its caller's stream, the trace was made on torch's
        return case, plan, trace
    if kind == "lde":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        n = 1 << case["log_rows"]
        trace = torch.randint(0, P, (case["columns"], n), generator=gen, device="cuda", dtype=torch.int32)
        out = torch.zeros((case["columns"], n << case["log_blowup"]), device="cuda", dtype=torch.int32)
        return case, trace, out
    if kind == "fft":
        return case, _uniform(rng, case["columns"], 1 << case["log_n"])
    if kind == "prove":
        return case, _job(case["air"], case["log_rows"], case["log_blowup"], seed)
    if kind == "batch":
        return case, [_job(air, lg, 2, seed + 1000 * i) for i, (air, lg) in enumerate(_batch_shapes(case))]
    if kind == "columns":
        cols = _uniform(rng, case["columns"], 1 << case["log_rows"], 4)
        return case, wire.columns(list(cols))
    size = 3 * (1 << case["log_rows"]) * (case["bits"] // 8)
    tables = torch.from_numpy(rng.integers(0, 256, size, dtype=np.uint8)).pin_memory()
    return case, tables


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def _bytes(b):
    return np.frombuffer(b, dtype=np.uint8)


def run(state):
    case, kind = state[0], state[0]["kind"]
    if kind == "commit":
        _, plan, trace = state
        plan.run(trace.data_ptr())
        r = plan.results()
        return {"root": _bytes(r["lde_root"]), "layer_roots": r["layer_roots"], "final_layer": r["final_layer"]}
    if kind == "lde":
        _, trace, out = state
        native.check(native.circle_lde_noalloc(trace.data_ptr(), out.data_ptr(), case["columns"], case["log_rows"],
                                               case["log_blowup"], torch.cuda.current_stream().cuda_stream), "lde")
        return out
    if kind == "fft":
        return (native.circle_ifft if case["inverse"] else native.circle_fft)(state[1])
    if kind == "prove":
        return _bytes(native.prove(*state[1]))
    if kind == "batch":
        return [_bytes(p) for p in native.prove_batch(state[1], concurrency=case["workers"])]
    if kind == "columns":
        return [_bytes(r) for r in native.commit_columns(state[1], case["log_rows"], case["log_blowup"])]
    claimed, rounds = native.binius_prove_combination(case["bits"], state[1], case["log_rows"], 3, TERMS)
    return [_bytes(claimed), _bytes(rounds)]


def exact(case, seed):
    """Field elements, hashes and proof bytes: whole numbers, compared bit by bit."""
    return None


# ---------------------------------------------------------------------------
# the work a pass cannot do without
# ---------------------------------------------------------------------------

COMPRESS = 7 * 8 * 14  # one Blake3 compression: 7 rounds of 8 G of 6 adds, 4 xors, 4 rotations
BUTTERFLY = 3          # a field product, a sum and a difference
CM31 = 3               # field products of a CM31 product


def _tree(n, leaf):
    return n * leaf * COMPRESS + 2 * (n - 1) * COMPRESS


def _prove_work(air, log_rows, log_blowup):
    n, big = 1 << log_rows, 1 << (log_rows + log_blowup)
    pre, main, acc = {"fib": (0, 2, 0), "and_table": (2, 3, 1), "rescue": (0, 12, 0), "ml_linear": (128, 258, 1)}[air]
    m = pre + main + acc
    ntt = 2 * CM31 * BUTTERFLY * (n * log_rows // 2 + big * log_rows // 2)
    fri = sum(_tree(big >> i, 1) + (big >> i) * 40 for i in range(log_rows + log_blowup - REMAINDER_LOG))
    paths = QUERIES * (32 * (log_rows + log_blowup) * (2 * m + 1) + 16 * (2 * m + 1))
    return {"bytes": 4 * n * (pre + main) + paths, "flops": m * (ntt + _tree(big, 1)) + _tree(big, 1) + fri}


def work(case):
    kind = case["kind"]
    if kind in ("commit", "lde"):
        c, lr, lb = case["columns"], case["log_rows"], case["log_blowup"]
        n, big = 1 << lr, 1 << (lr + lb)
        flops = c * BUTTERFLY * (n * lr // 2 + big * lr // 2)
        if kind == "lde":
            return {"bytes": 4 * c * (n + big), "flops": flops}
        flops += _tree(big, (4 * c + 63) // 64) + 8 * c * big
        byts = 4 * c * (n + big) + 64 * big
        for i in range(case["folds"]):
            flops += _tree(big >> i, 1) + (big >> i) * 40
            byts += (16 + 64) * (big >> i)
        return {"bytes": byts, "flops": flops}
    if kind == "fft":
        n = 1 << case["log_n"]
        return {"bytes": 8 * case["columns"] * n, "flops": case["columns"] * BUTTERFLY * n * case["log_n"] // 2}
    if kind == "prove":
        return _prove_work(case["air"], case["log_rows"], case["log_blowup"])
    if kind == "batch":
        each = [_prove_work(air, lg, 2) for air, lg in _batch_shapes(case)]
        return {"bytes": sum(w["bytes"] for w in each), "flops": sum(w["flops"] for w in each)}
    if kind == "columns":
        c, lr, lb = case["columns"], case["log_rows"], case["log_blowup"]
        n, big = 1 << lr, 1 << (lr + lb)
        ntt = 2 * CM31 * BUTTERFLY * (n * lr // 2 + big * lr // 2)
        return {"bytes": 16 * c * n + 32 * c, "flops": c * (ntt + _tree(big, 1))}
    rows, es = 1 << case["log_rows"], case["bits"] // 8
    # per row pair and point: two tower products and the sums; the fold: one product a table
    mul = 1 if es == 1 else 121
    return {"bytes": 3 * rows * es, "flops": rows * (4 * 2 * (mul + 3) // 2 + 3 * (mul + 1))}
