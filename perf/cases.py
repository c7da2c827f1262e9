"""The calls this library is timed on: what each stands for, its inputs, one pass, its work, its value.

Every case goes through the public Python binding (sgemm.cu_b200/sgemm_b200.py),
as a user's program calls it: one GEMM on device matrices (plain FFMA path or a
split-precision tensor-core path), a grouped launch, or one GEMM on host
matrices.  Values are uniform on [-1, 1), the benchmark's distribution.

A case is a dict: "op" (gemm, grouped, grouped_split, host), "path" (plain,
bf16x6, tf32x3), the sizes m, n, k (or "count", "mix" and "table" for a grouped
launch), alpha and beta.
"""
import math
import os
import random
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "sgemm.cu_b200"))
import sgemm_b200 as sg  # noqa: E402


def _gemm(path, m, n, k, alpha, beta, op="gemm", **more):
    return dict(more, op=op, path=path, m=m, n=n, k=k, alpha=alpha, beta=beta)


def listed():
    return [
        # the low end of the square test sweep: launch and latency
        _gemm("plain", 256, 256, 256, 1.0, 0.0, name="plain_256"),
        # the smallest benchmarked size, alpha = 1 and beta = 0
        _gemm("plain", 1024, 1024, 1024, 1.0, 0.0, name="plain_1024"),
        # an odd size of the square sweep: rows that are not 16-byte aligned
        _gemm("plain", 3001, 3001, 3001, 1.5, 0.5, name="plain_3001"),
        # the headline size
        _gemm("plain", 8192, 8192, 8192, 1.5, 0.5, name="plain_8192"),
        # a few rows against a 4096 x 4096 weight: the serving mix's common request
        _gemm("plain", 24, 4096, 4096, 1.0, 0.0, name="plain_rows24"),
        # the same on the tensor cores, a larger and ragged row count
        _gemm("bf16x6", 136, 4096, 4096, 1.0, 0.0, name="bf16x6_rows136"),
        # mid-size, tile edges in both directions, C read
        _gemm("bf16x6", 1000, 1000, 1000, 1.5, 0.5, name="bf16x6_1000"),
        _gemm("tf32x3", 2048, 2048, 2048, 1.0, 0.0, name="tf32x3_2048"),
        # the split-precision headline size
        _gemm("bf16x6", 8192, 8192, 8192, 1.5, 0.5, name="bf16x6_8192"),
        # a server's batch: 60% few-row requests, 40% cubes, through a kept plan
        {"name": "grouped_serving32", "op": "grouped", "path": "plain", "mix": "serving",
         "count": 32, "table": 1, "alpha": 1.0, "beta": 0.0},
        # a table of uneven problems, m, n, k log-uniform on [64, 4096]
        {"name": "grouped_split_64", "op": "grouped_split", "path": "bf16x6", "mix": "uneven",
         "count": 64, "table": 2, "alpha": 1.0, "beta": 0.0},
        # host matrices in and out: the copies overlap the kernels
        _gemm("plain", 4096, 4096, 4096, 1.5, 0.5, op="host", name="host_4096"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi):
    """Log-uniform, every second one a multiple of 8."""
    v = _log_int(rng, lo, hi)
    return min(hi, max(lo, v if rng.random() < 0.5 else (v + 4) // 8 * 8))


def draw(rng):
    alpha, beta = rng.choice([(1.0, 0.0), (1.5, 0.5)])
    kind = rng.choice(["square", "square", "rows", "rows", "rect", "rect", "grouped", "host"])
    if kind == "square":
        path = rng.choice(["plain", "plain", "bf16x6", "tf32x3"])
        s = _size(rng, 200, 6144)
        return _gemm(path, s, s, s, alpha, beta)
    if kind == "rows":
        path = rng.choice(["plain", "bf16x6", "tf32x3"])
        return _gemm(path, rng.randint(16, 256), 4096, 4096, alpha, beta)
    if kind == "rect":
        path = rng.choice(["plain", "bf16x6", "tf32x3"])
        return _gemm(path, _size(rng, 64, 4096), _size(rng, 64, 4096), _size(rng, 64, 4096),
                     alpha, beta)
    if kind == "grouped":
        op, path = rng.choice([("grouped", "plain"), ("grouped_split", "bf16x6"),
                               ("grouped_split", "tf32x3")])
        return {"op": op, "path": path, "mix": rng.choice(["serving", "uneven"]),
                "count": rng.randint(8, 48), "table": rng.randint(3, 1 << 30), "alpha": alpha,
                "beta": beta}
    s = _size(rng, 512, 4096)
    return _gemm("plain", s, s, s, alpha, beta, op="host")


def _shapes(case):
    """(m, n, k) of each problem of the case."""
    if "m" in case:
        return [(case["m"], case["n"], case["k"])]
    rng = random.Random(case["table"])
    shapes = []
    for _ in range(case["count"]):
        if case["mix"] == "serving" and rng.random() < 0.6:
            shapes.append((rng.randint(16, 256), 4096, 4096))
        elif case["mix"] == "serving":
            s = max(512, _log_int(rng, 512, 4096) // 8 * 8)
            shapes.append((s, s, s))
        else:
            shapes.append(tuple(max(64, _log_int(rng, 64, 4096) // 8 * 8) for _ in range(3)))
    return shapes


def _inputs(case, seed):
    """A, B and C of each problem, made on the GPU from the seed."""
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def mat(r, c):
        return torch.rand(r, c, generator=gen, device="cuda").mul_(2.0).sub_(1.0)

    return [(mat(m, k), mat(k, n), mat(m, n)) for m, n, k in _shapes(case)]


def prepare(case, seed):
    ops = _inputs(case, seed)
    state = {"case": case, "ops": ops}
    specs = [(A, B, C, case["alpha"], case["beta"]) for A, B, C in ops]
    if case["op"] == "grouped":
        state["plan"] = sg.GroupedPlan(specs)
    elif case["op"] == "grouped_split":
        state["problems"] = sg.make_problems(specs)
    elif case["op"] == "host":
        state["ops"] = [tuple(x.cpu().pin_memory() for x in ops[0])]
    return state


def run(state):
    case = state["case"]
    if case["op"] == "grouped":
        state["plan"].launch()
    elif case["op"] == "grouped_split":
        sg.grouped_split(case["path"], state["problems"])
    elif case["op"] == "host":
        A, B, C = state["ops"][0]
        sg.sgemm_host(A, B, C, case["alpha"], case["beta"], case["path"])
        torch.cuda.synchronize()  # the call is stream-ordered: C is the host's after it
    elif case["path"] == "plain":
        A, B, C = state["ops"][0]
        sg.sgemm(A, B, C, case["alpha"], case["beta"])
    else:
        A, B, C = state["ops"][0]
        sg.gemm(case["path"], A, B, C, case["alpha"], case["beta"])
    return [C for _, _, C in state["ops"]]


def work(case):
    flops = sum(2.0 * m * n * k for m, n, k in _shapes(case))
    reads_c = 2 if case["beta"] != 0.0 else 1
    return {"bytes": sum(4.0 * (m * k + k * n + reads_c * m * n) for m, n, k in _shapes(case)),
            "flops": flops}


def exact(case, seed):
    return [case["alpha"] * (A.double() @ B.double()) + case["beta"] * C.double()
            for A, B, C in _inputs(case, seed)]
