"""Performance cases of the counting library: the calls that its users make, over the range they make them in.

Every case goes through the public Python entry points (``n_queens_b200`` and ``n_queens_b200.learned``).  Inputs come
from the seed: random partial boards, random samples of a board's prefix tasks, random queue orders, random weights.

Kinds:

* ``board``     completions of one partial board (``n_queens``): one small call, where latency counts;
* ``tasks``     counts of a host task list (``count_tasks``), with per-task counts and, for cost labels, DFS nodes;
* ``device``    counts of tasks that lie in device memory already (``count_tasks_device``), total or per task;
* ``whole``     a whole board, or one machine's share of it: prefixes in a shuffled queue order of which the first part is
  counted (``count`` and ``count_dihedral`` with ``order`` and ``queue_len``);
* ``batch``     replays of a plan of many uneven partial boards (``BatchPlan.run``);
* ``grad``      forward and backward pass of the cost model (``CostModel.grad``), a minibatch or a larger set;
* ``predict``   predictions of the cost model for host tasks (``CostModel.predict``);
* ``schedule``  longest-first order of device-resident tasks (``nq_schedule_device``): tensor-core forward and sort.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import n_queens_b200 as nq
from n_queens_b200 import learned
from n_queens_b200.workloads import SplitMix64, random_board, random_boards

# DFS nodes of the half-board search (placements into rows k..N-2; for N >= 16 the repository's own figures).
NODES = {8: 431, 9: 2.7e3, 10: 1.45e4, 11: 7.6e4, 12: 4.1e5, 13: 2.28e6, 14: 1.35e7, 15: 8.4e7, 16: 5.63e8, 17: 3.96e9,
         18: 2.93e10, 19: 2.28e11, 20: 1.87e12, 21: 1.59e13}
OPS_PER_NODE = 22    # integer operations of one DFS node (the repository's cost model)
MOST_NODES = 1.28e12  # a pass of the largest listed case
EXACT_NODES = 1.5e7  # the plain count of `exact` takes a few seconds for this many


def listed():
    return [
        # One interactive query: how many ways a 14x14 board with three queens set can be completed.
        dict(name="one board N=14", kind="board", N=14, placed=3),
        # A service that counts a short host list of partial boards, each by itself.
        dict(name="host tasks N=13", kind="tasks", N=13, rows=4, n=1501, per_task=True, nodes=False),
        # An ordinary device-resident list: sum only, tasks of some thousand nodes.
        dict(name="device tasks N=16", kind="device", N=16, rows=5, n=60001, per_task=False),
        # A large device-resident list with a count per task.
        dict(name="device tasks N=18", kind="device", N=18, rows=6, n=1100003, per_task=True),
        # Solver-logged labels for the cost model: counts and DFS nodes of a sample of prefixes.
        dict(name="labels N=17", kind="tasks", N=17, rows=6, n=300007, per_task=True, nodes=True),
        # Nearly a whole board, tasks built on the device.
        dict(name="whole N=19", kind="whole", N=19, rows=6, share=0.97, device_expand=True, dihedral=False),
        # One of a dozen machines' share of the benchmark board (tasks built on the host).
        dict(name="share of N=21", kind="whole", N=21, rows=6, share=0.08, device_expand=False, dihedral=False),
        # Nearly a whole board through the 8-fold decomposition.
        dict(name="dihedral N=19", kind="whole", N=19, rows=6, share=0.97, device_expand=False, dihedral=True),
        # A replayed plan of 512 uneven boards (the autotuner's batch).
        dict(name="batch of 512", kind="batch", n=512, n_lo=12, n_hi=17),
        # One training minibatch.
        dict(name="gradient of 4096", kind="grad", N=18, rows=6, n=4096),
        # Hold-out predictions after a model build.
        dict(name="predict 200k", kind="predict", N=21, rows=6, n=200000),
        # Queue order of a whole N=19 board.
        dict(name="schedule 1.9M", kind="schedule", N=19, rows=6, n=1900001),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


@functools.lru_cache(None)
def _prefixes(N, rows):
    return int(nq.expand(N, rows)[0].size)


def draw(rng):
    kind = rng.choice(("board", "tasks", "device", "whole", "whole", "batch", "grad", "predict", "schedule"))
    if kind == "board":
        return dict(kind=kind, N=rng.randint(12, 17), placed=rng.randint(2, 3))
    if kind == "tasks":
        N = rng.randint(11, 18)
        rows = 4 if N < 14 else rng.randint(5, 6)
        return dict(kind=kind, N=N, rows=rows, n=_log_uniform(rng, 300, 0.9 * _prefixes(N, rows)), per_task=True,
                    nodes=rng.random() < 0.5)
    if kind == "device":
        N = rng.randint(14, 19)
        rows = rng.randint(5, 6)
        return dict(kind=kind, N=N, rows=rows, n=_log_uniform(rng, 5000, 0.9 * _prefixes(N, rows)),
                    per_task=rng.random() < 0.5)
    if kind == "whole":
        N = rng.randint(15, 21)
        most = min(0.97, 0.9 * MOST_NODES / NODES[N])
        return dict(kind=kind, N=N, rows=5 if N < 17 else 6, share=round(rng.uniform(0.3 * most, most), 4),
                    device_expand=rng.random() < 0.5, dihedral=rng.random() < 0.35)
    if kind == "batch":
        lo = rng.randint(8, 13)
        return dict(kind=kind, n=_log_uniform(rng, 17, 1500), n_lo=lo, n_hi=lo + rng.randint(2, 4))
    N = rng.randint(16, 21)
    n = {"grad": (1000, 200000), "predict": (2000, 400000), "schedule": (20000, 0.97 * _prefixes(N, 6))}[kind]
    return dict(kind=kind, N=N, rows=6, n=_log_uniform(rng, *n))


# ---------------------------------------------------------------------------- inputs
def _sample(case, seed):
    """A random sample, in random order, of the prefix tasks of (N, rows)."""
    c, l, r = nq.expand(case["N"], case["rows"])
    at = np.random.default_rng(seed).permutation(c.size)[:min(case["n"], c.size)]
    return c[at], l[at], r[at]


def _boards(case, seed):
    return random_boards(case["n"], seed, case["n_lo"], case["n_hi"], 0, 4)


def _weights(seed):
    """Weights of the size that training gives, output bias near the mean label."""
    p = np.random.default_rng(seed).uniform(-0.12, 0.12, learned.NUM_PARAMS).astype(np.float32)
    p[-1] = 12.0
    return p


def _labels(n, seed):
    return np.random.default_rng(seed + 1).normal(12.0, 1.5, n).astype(np.float32)


def _model(seed):
    m = learned.CostModel(seed=0)
    m.set_params(_weights(seed))
    return m


def _on_gpu(a):
    return torch.from_numpy(a.view(np.int32)).cuda()


def prepare(case, seed):
    kind, s = case["kind"], dict(case)
    if kind == "board":
        s["board"] = random_board(SplitMix64(seed), case["N"], case["placed"])
    elif kind == "tasks":
        s["tasks"] = _sample(case, seed)
    elif kind == "device":
        s["tasks"] = [_on_gpu(a) for a in _sample(case, seed)]
        n = s["tasks"][0].numel()
        s["sum"] = torch.zeros(2, dtype=torch.int64, device="cuda")
        s["out"] = torch.zeros(n, dtype=torch.int64, device="cuda") if case["per_task"] else None
        # the stack depth of (N, rows) prefixes, as the library states it
        s["config"] = dict(stack_levels=nq.stack_levels(case["N"], case["rows"]))
    elif kind == "whole":
        n = nq.dihedral_expand(case["N"], case["rows"])[0].size if case["dihedral"] else _prefixes(case["N"], case["rows"])
        s["order"] = np.random.default_rng(seed).permutation(n).astype(np.uint32)
        s["config"] = dict(order_kind=nq.NQ_ORDER_GIVEN, order=s["order"].ctypes.data,
                           queue_len=max(1, int(case["share"] * n)),
                           device_expand=int(case["device_expand"] and not case["dihedral"]))
    elif kind == "batch":
        s["plan"] = nq.BatchPlan(_boards(case, seed))
    else:
        s["model"] = _model(seed)
        s["tasks"] = _sample(case, seed)
        n = s["tasks"][0].size
        if kind == "grad":
            s["task_n"] = np.full(n, case["N"], np.uint8)
            s["target"] = _labels(n, seed)
        elif kind == "schedule":
            s["tasks"] = [_on_gpu(a) for a in s["tasks"]]
            s["order"] = torch.empty(n, dtype=torch.int32, device="cuda")
            s["pred"] = torch.empty(n, dtype=torch.float32, device="cuda")
    return s


# ---------------------------------------------------------------------------- one pass
def run(s):
    kind, N = s["kind"], s.get("N")
    if kind == "board":
        return nq.n_queens(N, *s["board"])
    if kind == "tasks":
        got = nq.count_tasks(N, *s["tasks"], per_task=s["per_task"], nodes=s["nodes"])
        return {"sum": got["sum"], "per_task": got["per_task"].view(np.int64),
                "nodes": got["nodes"].view(np.int64) if s["nodes"] else None}
    if kind == "device":
        nq.count_tasks_device(N, *s["tasks"], s["sum"], per_task=s["out"], config=s["config"],
                              stream=torch.cuda.current_stream())
        return {"sum": s["sum"], "per_task": s["out"]}
    if kind == "whole":
        count = nq.count_dihedral if s["dihedral"] else nq.count
        return count(N, s["rows"], config=s["config"]).total
    if kind == "batch":
        return s["plan"].run().view(np.int64)
    m = s["model"]
    if kind == "grad":
        gradient, loss = m.grad(s["task_n"], *s["tasks"], s["target"])
        return {"gradient": gradient, "loss": loss}
    if kind == "predict":
        return m.predict(N, *s["tasks"])
    rc = learned.lib.nq_schedule_device(m._m, N, *(t.data_ptr() for t in s["tasks"]), s["order"].numel(),
                                        s["order"].data_ptr(), s["pred"].data_ptr(),
                                        torch.cuda.current_stream().cuda_stream)
    if rc != nq.NQ_OK:
        raise nq.NQError(rc, "nq_schedule_device", nq.last_error())
    return {"order": s["order"], "pred": s["pred"]}


# ---------------------------------------------------------------------------- work of one pass
def _nodes(case):
    """DFS nodes of a pass, estimated from the whole board's."""
    kind = case["kind"]
    if kind == "board":
        return 2 * NODES[case["N"]] / (2 * _prefixes(case["N"], case["placed"]))
    if kind == "batch":
        sizes = range(case["n_lo"], case["n_hi"] + 1)
        return case["n"] / len(sizes) / 5 * sum(2 * NODES[N] * sum(1 / max(1, 2 * _prefixes(N, m)) for m in range(1, 5))
                                                for N in sizes)
    if kind == "whole":
        return NODES[case["N"]] * case["share"] / (1.75 if case["dihedral"] else 1)
    return NODES[case["N"]] * min(1.0, case["n"] / _prefixes(case["N"], case["rows"]))


def work(case):
    kind, n = case["kind"], case.get("n", 1)
    if kind in ("grad", "predict", "schedule"):
        weights = 96 * 128 + 128 * 128 + 128
        flops = {"grad": 6, "predict": 2, "schedule": 2}[kind] * weights * n
        moved = {"grad": 17 * n + 3 * 4 * weights, "predict": 16 * n + 2 * weights, "schedule": 20 * n + 2 * weights}[kind]
        return {"bytes": moved, "flops": flops}
    if kind == "whole":
        n = int(case["share"] * _prefixes(case["N"], case["rows"]))
    moved = 12 * n + (8 * n if case.get("per_task") else 0) + (8 * n if case.get("nodes") else 0) + 16
    return {"bytes": moved, "flops": OPS_PER_NODE * _nodes(case)}


# ---------------------------------------------------------------------------- the same in plain 64-bit arithmetic
def _completions(N, cols, ld, rd):
    """Completions of each partial board and its placements into rows before the last, level by level."""
    full = (1 << N) - 1
    c, l, r = (np.asarray(a, np.int64) & full for a in (cols, ld, rd))
    owner = np.arange(c.size)
    counts, nodes = np.zeros(c.size, np.int64), np.zeros(c.size, np.int64)
    while c.size:
        parts = []
        free = full & ~(c | l | r)
        for b in range(N):
            at = np.flatnonzero(free >> b & 1)
            p = 1 << b
            parts.append((c[at] | p, ((l[at] | p) << 1) & full, (r[at] | p) >> 1, owner[at]))
        c, l, r, owner = (np.concatenate([q[i] for q in parts]) for i in range(4))
        done = c == full
        counts += np.bincount(owner[done], minlength=counts.size)
        c, l, r, owner = c[~done], l[~done], r[~done], owner[~done]
        nodes += np.bincount(owner, minlength=counts.size)
    return counts, nodes


def _bits(N, tasks):
    m = np.stack([np.asarray(a, np.int64) & ((1 << N) - 1) for a in tasks])
    return torch.from_numpy((m[:, None, :] >> np.arange(32)[None, :, None] & 1).reshape(96, -1).T.copy()).double()


def _bf16(t):
    return t.float().bfloat16().double()


def _split(seed):
    p = torch.from_numpy(_weights(seed)).double()
    w1, b1, w2, b2, w3, b3 = torch.split(p, (128 * 96, 128, 128 * 128, 128, 128, 1))
    return _bf16(w1).view(128, 96), b1, _bf16(w2).view(128, 128), b2, _bf16(w3), b3


def _forward(N, tasks, seed, round_h1=False):
    w1, b1, w2, b2, w3, b3 = _split(seed)
    x = _bits(N, tasks)
    h1 = torch.relu(x @ w1.T + b1)
    if round_h1:  # the tensor-core forward rounds the layer-1 outputs to BF16
        h1 = _bf16(h1)
    h2 = torch.relu(h1 @ w2.T + b2)
    return x, h1, h2, h2 @ w3 + b3


def exact(case, seed):
    kind, N = case["kind"], case.get("N")
    if kind == "predict":
        return _forward(N, _sample(case, seed), seed)[3].numpy()
    if kind == "schedule":
        return {"order": None, "pred": _forward(N, _sample(case, seed), seed, round_h1=True)[3].numpy()}
    if kind == "grad":
        tasks = _sample(case, seed)
        n = tasks[0].size
        _, _, w2, _, w3, _ = _split(seed)
        x, h1, h2, out = _forward(N, tasks, seed)
        e = out - torch.from_numpy(_labels(n, seed)).double()
        d = 2.0 / n * e
        d2 = torch.outer(d, w3) * (h2 > 0)
        d1 = (d2 @ w2) * (h1 > 0)
        parts = (d1.T @ x, d1.sum(0), d2.T @ h1, d2.sum(0), h2.T @ d, d.sum())
        return {"gradient": torch.cat([g.reshape(-1) for g in parts]).numpy(), "loss": float((e * e).mean())}
    # Counts are whole numbers: compared bit for bit, and counted plainly where that is quick.
    if _nodes(case) > EXACT_NODES or kind in ("batch", "whole"):
        return None
    if kind == "board":
        return int(_completions(N, *([v] for v in random_board(SplitMix64(seed), N, case["placed"])))[0][0])
    counts, nodes = _completions(N, *_sample(case, seed))
    if kind == "device":
        return {"sum": np.array([counts.sum(), 0]), "per_task": counts if case["per_task"] else None}
    return {"sum": int(counts.sum()), "per_task": counts, "nodes": nodes if case["nodes"] else None}
