"""The work that users of this framework have it do, as timed cases.

A case is one pass through a public entry point: a single array on a plan
(`Plan.run`), a batch of arrays in one launch (`Plan.run_segmented`), a
consumer of the answers (`stock_span`, `cartesian_parents`, ...), int64
positions (`Plan.run64`), or a whole stream of requests (`PoolServer.serve`).
The plan, the output buffer and the workspace are what a program keeps
between calls; keys come from the seed alone.

Key distributions: `uniform` (random keys), `walk` (a random walk: prices,
sensor readings), `down` / `up` (sorted data with a rare key out of place),
`dup` (few distinct values).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from apsep_gb300 import Plan, consumers
from apsep_gb300.serve import PoolServer, Request

DTYPES = {"int32": torch.int32, "float32": torch.float32, "int64": torch.int64, "float64": torch.float64}
CONSUMERS = ("prev_greater", "next_smaller", "stock_span", "cartesian_parents")


def listed():
    return [
        # one short array: latency and launches
        {"name": "run_small", "kind": "run", "dtype": "int32", "n": 1000, "dist": "uniform", "le": False},
        # a series of about a million readings
        {"name": "run_walk_2p20", "kind": "run", "dtype": "float32", "n": (1 << 20) + 77, "dist": "walk", "le": True},
        # the single-array benchmark's size and its four kinds of keys
        {"name": "run_uniform_2p25", "kind": "run", "dtype": "int32", "n": 1 << 25, "dist": "uniform", "le": False},
        {"name": "run_down_2p25", "kind": "run", "dtype": "int32", "n": 1 << 25, "dist": "down", "le": False},
        {"name": "run_up_f32", "kind": "run", "dtype": "float32", "n": 30_000_001, "dist": "up", "le": False},
        {"name": "run_dup_le_2p25", "kind": "run", "dtype": "int32", "n": 1 << 25, "dist": "dup", "le": True},
        # 8-byte keys
        {"name": "run_int64", "kind": "run", "dtype": "int64", "n": (1 << 24) + 5, "dist": "uniform", "le": False},
        # thousands of arrays of every length in one launch (random keys, descending runs, sawtooth)
        {"name": "batch_1024", "kind": "batch", "dtype": "int32", "segments": 1024, "lo": 32, "hi": 1 << 20},
        # span of every price of a long series
        {"name": "stock_span_2p24", "kind": "stock_span", "dtype": "float32", "n": 1 << 24, "dist": "walk", "le": False},
        # the tree behind range-minimum queries, an odd length
        {"name": "cartesian_5m", "kind": "cartesian_parents", "dtype": "int32", "n": 5_000_003, "dist": "uniform",
         "le": False},
        # int64 positions: an array in pieces of its plan's capacity
        {"name": "run64_pieces", "kind": "run64", "dtype": "int32", "n": (1 << 28) + 999, "piece": 1 << 27,
         "dist": "uniform", "le": False},
        # a saturated request stream, int32 and float32 arrays, keys and answers in device memory
        {"name": "serve_96", "kind": "serve", "requests": 96, "lo": 1 << 10, "hi": 1 << 22},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run"] * 6 + ["batch"] * 2 + ["consumer"] * 2 + ["run64", "serve"])
    if kind == "batch":
        return {"kind": "batch", "dtype": rng.choice(["int32", "float32"]), "segments": _log_int(rng, 8, 1024),
                "lo": 32, "hi": _log_int(rng, 1 << 10, 1 << 20)}
    if kind == "serve":
        return {"kind": "serve", "requests": rng.randint(16, 128), "lo": 1 << 10, "hi": _log_int(rng, 1 << 14, 1 << 22)}
    case = {"dtype": rng.choice(["int32", "int32", "float32", "float32", "int64", "float64"]),
            "dist": rng.choice(["uniform", "uniform", "walk", "down", "up", "dup"]), "le": rng.random() < 0.4}
    if kind == "run":
        return dict(case, kind="run", n=_log_int(rng, 1 << 8, 1 << 26))
    if kind == "run64":
        n = _log_int(rng, 1 << 22, 1 << 27)
        return dict(case, kind="run64", n=n, piece=max(1 << 20, n // rng.randint(1, 6)))
    return dict(case, kind=rng.choice(CONSUMERS), n=_log_int(rng, 1 << 10, 1 << 25))


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _keys(n, dtype, dist, g):
    dev = "cuda"
    if dist == "uniform":
        if dtype in (torch.float32, torch.float64):
            return torch.randn(n, generator=g, device=dev, dtype=dtype)
        hi = (1 << 31) - 1 if dtype == torch.int32 else 1 << 62
        return torch.randint(-hi if dtype == torch.int64 else 0, hi, (n,), generator=g, device=dev, dtype=dtype)
    if dist == "dup":
        return torch.randint(0, 16, (n,), generator=g, device=dev, dtype=torch.int32).to(dtype)
    if dist == "walk":  # steps of up to +-1000 ticks
        steps = torch.randint(-1000, 1001, (n,), generator=g, device=dev, dtype=torch.int32)
        x = torch.cumsum(steps, 0, dtype=torch.int64)
        return (x.to(torch.float64) * 0.01).to(dtype) if dtype in (torch.float32, torch.float64) else x.to(dtype)
    x = torch.arange(n, device=dev, dtype=torch.int32)
    if dist == "down":
        x = n - 1 - x
    # one key in 50,000 is out of place
    step = min(n, 50_000)
    at = torch.arange(n // step, device=dev) * step + torch.randint(0, step, (n // step,), generator=g, device=dev)
    x[at] = torch.randint(0, n, (n // step,), generator=g, device=dev, dtype=torch.int32)
    return x.to(dtype)


def _lengths(count, lo, hi):
    rng = np.random.default_rng(count)  # the case's own: other keys come in the same arrays
    return np.round(np.exp(rng.uniform(math.log(lo), math.log(hi), count))).astype(np.int64)


def _batch(case, seed):
    """Keys and offsets: uniform keys, descending runs of up to 4096 keys and a
    sawtooth, one of the three per array in turn."""
    g = _generator(seed)
    offs = np.zeros(case["segments"] + 1, dtype=np.int64)
    offs[1:] = np.cumsum(_lengths(case["segments"], case["lo"], case["hi"]))
    n = int(offs[-1])
    d_offs = torch.from_numpy(offs).cuda()
    pos = torch.arange(n, device="cuda", dtype=torch.int32)
    seg = torch.bucketize(pos.to(torch.int64), d_offs[1:], right=True).to(torch.int32)
    x = torch.randint(0, (1 << 31) - 1, (n,), generator=g, device="cuda", dtype=torch.int32)
    ends = torch.cumsum(torch.randint(1, 4097, (n // 1024 + 8,), generator=g, device="cuda"), 0)
    run = torch.bucketize(pos, ends.to(torch.int32), right=True, out_int32=True)
    top = torch.randint(4096, 1 << 30, (run.max().item() + 1,), generator=g, device="cuda", dtype=torch.int32)
    first = torch.cat([ends.new_zeros(1), ends])[run].to(torch.int32)
    x = torch.where(seg % 3 == 1, top[run] - (pos - first), x)
    x = torch.where(seg % 3 == 2, (pos - d_offs[seg].to(torch.int32)) % 257, x)
    return x.to(DTYPES[case["dtype"]]), d_offs


def prepare(case, seed):
    kind = case["kind"]
    if kind == "serve":
        n = _lengths(case["requests"], case["lo"], case["hi"])
        g = _generator(seed)
        out = torch.empty(int(n.sum()), dtype=torch.int32, device="cuda")
        reqs, at = [], 0
        for i, m in enumerate(n):
            m = int(m)
            keys = _keys(m, torch.int32 if i % 2 else torch.float32, "uniform", g)
            reqs.append(Request(rid=i, keys=keys, out=out[at:at + m]))
            at += m
        server = PoolServer(budget_bytes=2 << 30, max_batch_keys=1 << 25)
        return {"kind": kind, "server": server, "requests": reqs, "out": out}
    if kind == "batch":
        x, offs = _batch(case, seed)
        return {"kind": kind, "x": x, "offs": offs, "plan": Plan(x.numel(), x.dtype),
                "out": torch.empty(x.numel(), dtype=torch.int32, device="cuda")}
    n, dtype = case["n"], DTYPES[case["dtype"]]
    x = _keys(n, dtype, case["dist"], _generator(seed))
    state = {"kind": kind, "x": x, "le": case["le"]}
    if kind == "run":
        state["plan"] = Plan(n, dtype, inclusive=case["le"])
        state["out"] = torch.empty(n, dtype=torch.int32, device="cuda")
    elif kind == "run64":
        state["plan"] = plan = Plan(case["piece"], dtype, inclusive=case["le"])
        state["out"] = torch.empty(n, dtype=torch.int64, device="cuda")
        state["work"] = torch.empty(max(plan.workspace64_bytes(n), 16), dtype=torch.uint8, device="cuda")
    else:
        state["plan"] = Plan(n, dtype)
        state["work"] = torch.empty(consumers.workspace_bytes(n), dtype=torch.uint8, device="cuda")
    return state


def run(state):
    kind = state["kind"]
    if kind == "run":
        return state["plan"].run(state["x"], out=state["out"])
    if kind == "batch":
        return state["plan"].run_segmented(state["x"], state["offs"], out=state["out"])
    if kind == "run64":
        return state["plan"].run64(state["x"], out=state["out"], work=state["work"])
    if kind == "serve":
        state["server"].serve(state["requests"], realtime=False)
        return state["out"]
    if kind == "stock_span":
        return consumers.stock_span(state["x"], plan=state["plan"], work=state["work"])
    if kind == "cartesian_parents":
        return consumers.cartesian_parents(state["x"], plan=state["plan"], work=state["work"])
    fn = {"prev_greater": consumers.prev_greater, "next_smaller": consumers.next_smaller}[kind]
    return fn(state["x"], inclusive=state["le"], plan=state["plan"], work=state["work"])


def work(case):
    """Every key read once, every answer written once."""
    kind = case["kind"]
    if kind == "serve" or kind == "batch":
        count = case["requests"] if kind == "serve" else case["segments"]
        return {"bytes": 8 * int(_lengths(count, case["lo"], case["hi"]).sum()), "flops": 0}
    key = 8 if case["dtype"] in ("int64", "float64") else 4
    return {"bytes": (key + (8 if kind == "run64" else 4)) * case["n"], "flops": 0}


def _previous(a, qualifies):
    """For each key the nearest earlier one that `qualifies(earlier, key)`, by a stack."""
    out, stack = [], []
    for i, k in enumerate(a):
        while stack and not qualifies(a[stack[-1]], k):
            stack.pop()
        out.append(stack[-1] if stack else -1)
        stack.append(i)
    return out


def exact(case, seed):
    """The positions a sequential stack gives, for arrays short enough for one."""
    kind = case["kind"]
    if kind in ("serve", "batch") or case["n"] > 200_000:
        return None
    n = case["n"]
    a = _keys(n, DTYPES[case["dtype"]], case["dist"], _generator(seed)).tolist()
    le = case["le"]
    if kind in ("run", "run64"):
        got = _previous(a, (lambda u, v: u <= v) if le else (lambda u, v: u < v))
    elif kind == "prev_greater":
        got = _previous(a, (lambda u, v: u >= v) if le else (lambda u, v: u > v))
    elif kind == "next_smaller":
        got = _previous(a[::-1], (lambda u, v: u <= v) if le else (lambda u, v: u < v))
        got = [n - 1 - j if j >= 0 else -1 for j in got[::-1]]
    elif kind == "stock_span":
        got = [i - j for i, j in enumerate(_previous(a, lambda u, v: u > v))]
    else:  # Cartesian tree: the larger of previous smaller-or-equal and next smaller, the next one on a tie
        prev = _previous(a, lambda u, v: u <= v)
        nxt = [n - 1 - j if j >= 0 else -1 for j in _previous(a[::-1], lambda u, v: u < v)[::-1]]
        got = [p if r < 0 else r if p < 0 or a[r] >= a[p] else p for p, r in zip(prev, nxt)]
    return torch.tensor(got, dtype=torch.int64 if kind == "run64" else torch.int32)
