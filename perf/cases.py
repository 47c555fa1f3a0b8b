"""The work a user of this library has it do, as cases to time and compare.

Every case is a call or a short sequence of calls through the package's public
entry points. A board is contracted from the empty boundary, which has no
input besides its size, so the cases with a whole board also count the
completions of a partly placed board of the same size (two of a small one),
drawn from the seed: the check of a branch that goes with a board's total.

The program keeps one context (and one server) for all its calls, as the
package's default context does.
"""
from __future__ import annotations

import importlib
import random

import numpy as np
import torch

qp = importlib.import_module("quantum-harness-peps-naive_gb300")

KNOWN = (1, 1, 0, 0, 2, 10, 4, 40, 92, 352, 724, 2680, 14200, 73712, 365596, 2279184, 14772512, 95815104, 666090624,
         4968057848, 39029188884)  # OEIS A000170

# Boundary entries over all rows of a whole board with first-row reflection
# orbits, (read, written), from size 4; each further size has 6.2 to 6.8 times
# the entries of the one before.
ENTRIES = {4: (8, 8), 5: (25, 28), 6: (70, 71), 7: (275, 288), 8: (909, 939), 9: (4140, 4253), 10: (15958, 16182),
           11: (80788, 81556), 12: (370406, 373150), 13: (2103611, 2114574), 14: (10944059, 10984292),
           15: (68791796, 68951403), 16: (397600652, 398228827), 17: (2684482261, 2686800583),
           18: (16.68e9, 16.7e9)}

_kept: dict = {}


def _context(kind: str):
    """The program's context; "tuned" is the one that repeats a large board
    with the shipped tuning."""
    if kind not in _kept:
        c = qp.Context(0)
        if kind == "tuned":
            c.load_tuning(18, qp.LIBRARY_PATH.parent / "tuning_gb300.json")
        _kept[kind] = c
    return _kept[kind]


def _server():
    if "server" not in _kept:
        # Answers are computed, not looked up: the same requests come again.
        _kept["server"] = qp.Server(0, use_cache=0, batch_budget_bytes=16 << 30, large_budget_bytes=32 << 30)
    return _kept["server"]


def listed():
    return [
        # The smallest call: a partly placed small board, where latency is all.
        {"name": "prefix small", "kind": "prefix", "n": 9, "k": 3},
        # One small whole board, as `qpeps solve 8`.
        {"name": "board 8", "kind": "board", "n": 8},
        # Ordinary boards, up to the published range of the reference.
        {"name": "board 12", "kind": "board", "n": 12},
        {"name": "board 14", "kind": "board", "n": 14},
        {"name": "board 16", "kind": "board", "n": 16},
        # The largest board of one device batch.
        {"name": "board 17", "kind": "board", "n": 17},
        # The benchmark's repeated large board: shipped tuning, several device
        # batches, replayed as a CUDA graph.
        {"name": "board 18 replayed", "kind": "replay", "n": 18},
        # A request for the completions of a large partly placed board.
        {"name": "prefix large", "kind": "prefix", "n": 19, "k": 3},
        # A board beyond 64-bit keys.
        {"name": "prefix wide keys", "kind": "prefix", "n": 24, "k": 9},
        # Requests of mixed sizes and prefixes through the continuous-batching server.
        {"name": "serve mixed", "kind": "serve", "n_lo": 10, "n_hi": 14, "requests": 48},
        # The plain form of the contraction: the explicit tensor, one launch per site.
        {"name": "sites 11", "kind": "sites", "n": 11},
        # The explicit tensor's site frontier in diamond order.
        {"name": "diamond 11", "kind": "explicit", "n": 11, "order": 1},
    ]


def draw(rng: random.Random):
    kind = rng.choice(["prefix", "board", "prefix", "board", "wide", "serve", "sites", "explicit"])
    if kind == "prefix":
        # Any board up to 20, placed so far that a pass stays short.
        n = rng.randint(8, 20)
        lo = max(1, n - 16)
        return {"kind": "prefix", "n": n, "k": rng.randint(lo, lo + 3), "boards": rng.randint(1, 16)}
    if kind == "wide":
        n = rng.randint(22, 28)
        return {"kind": "prefix", "n": n, "k": n - rng.randint(13, 15), "boards": rng.randint(1, 16)}
    if kind == "serve":
        lo = rng.randint(8, 12)
        return {"kind": "serve", "n_lo": lo, "n_hi": lo + rng.randint(0, 3), "requests": rng.randint(5, 120)}
    if kind == "board":
        case = {"kind": "board", "n": rng.randint(8, 17), "symmetry": rng.choice([1, 1, 1, 0])}
    elif kind == "sites":
        case = {"kind": "sites", "n": rng.randint(8, 13)}
    else:
        case = {"kind": "explicit", "n": rng.randint(8, 12), "order": rng.randint(0, 1)}
    # The branches counted beside the board: how many, and the rows placed on each.
    case["branches"] = rng.randint(1, 6)
    case["rows"] = rng.randint(2, case["n"] // 2)
    return case


def _prefix_rows(case: dict) -> int:
    """Rows placed on the board counted beside a whole one."""
    return case.get("rows", max(2, case["n"] // 3))


def _branches(case: dict) -> int:
    """Boards counted beside a whole one."""
    return case.get("branches", 2 if case["n"] < 12 else 1)


def _draws(case: dict, seed: int) -> list:
    """The partly placed boards of a case: (size, columns)."""
    rng = random.Random(f"{seed}/{sorted(case.items(), key=lambda kv: kv[0])}")
    if case["kind"] == "prefix":
        # One call each, as they come.
        return [(case["n"], qp.random_prefix(rng, case["n"], case["k"])) for _ in range(case.get("boards", 4))]
    if case["kind"] == "serve":
        out = []
        for _ in range(case["requests"]):
            n = rng.randint(case["n_lo"], case["n_hi"])
            out.append((n, qp.random_prefix(rng, n, rng.randint(0, 3))))
        return out
    n = case["n"]
    return [(n, qp.random_prefix(rng, n, _prefix_rows(case))) for _ in range(_branches(case))]


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    state = {"case": case, "boards": _draws(case, seed)}
    if kind == "serve":
        state["server"] = _server()
    else:
        state["ctx"] = _context("tuned" if kind == "replay" else "plain")
    return state


def _layers(r) -> np.ndarray:
    """Per-row metrics, one line a row."""
    return np.array([[l.row, l.input_states, l.row_operator_candidates, l.row_operator_matched, l.completed_row_terms,
                      l.output_states, l.output_weight] for l in r.layers], dtype=np.int64)


def _counts(ctx, boards) -> np.ndarray:
    """Completions, largest boundary and examined and matched row terms of each board."""
    out = []
    for n, prefix in boards:
        count, r = ctx.count_with_stats(n, prefix)
        out.append([count, r.peak_states, r.row_operator_candidates, r.row_operator_matched])
    return np.array(out, dtype=np.int64)


def run(state: dict):
    case, boards = state["case"], state["boards"]
    kind = case["kind"]
    if kind == "serve":
        server = state["server"]
        for tag, (n, prefix) in enumerate(boards):
            server.submit(n, prefix, tag)
        counts = np.zeros(len(boards), dtype=np.int64)
        left = len(boards)
        while left:
            for done in server.poll(max_items=len(boards), wait_ms=1000):
                counts[done["tag"]] = done["count"] if done["status"] == 0 else -1
                left -= 1
        return {"counts": counts}
    ctx = state["ctx"]
    if kind == "prefix":
        return {"counts": _counts(ctx, boards)}
    n = case["n"]
    if kind == "explicit":
        e = ctx.explicit_frontier(n, case["order"], 1 << 40)
        out = {"board": np.array([e["count"], e["peak_states"], e["peak_open_bonds"], e["tensor_entries_examined"],
                                  e["tensor_entries_accepted"], e["contracted_sites"]], dtype=np.int64)}
    else:
        if kind == "sites":
            r = ctx.contract_rows(n, granularity=qp.GRAIN_SITE)
        elif kind == "replay":
            r = ctx.contract_rows(n, use_graph=1)
        else:
            r = ctx.contract_rows(n, symmetry=case.get("symmetry", 1))
        out = {"count": r.count, "peak": r.peak_states, "layers": _layers(r)}
    out["branches"] = _counts(ctx, boards)
    return out


def _entries(n: int) -> tuple:
    if n in ENTRIES:
        return ENTRIES[n]
    if n < 4:
        return (2 * n, 2 * n)
    up = 6.6 ** (n - 18)
    return (ENTRIES[18][0] * up, ENTRIES[18][1] * up)


def _prefix_entries(n: int, k: int) -> float:
    """About the entries read and written below a k-row prefix: each placed
    row divides a whole board's by the choices it had."""
    e = float(sum(_entries(n)))
    for i in range(k):
        e *= 2.0 / n if i == 0 else 1.0 / max(6.0, n - 3.0 * i)
    return max(e, 2.0 * (n - k))


def work(case: dict) -> dict:
    """The boundary entries a contraction reads and writes: a 64-bit key (128
    above 22 columns) and a 64-bit weight each."""
    kind = case["kind"]
    if kind == "prefix":
        size = 16 if case["n"] <= 22 else 24
        return {"bytes": case.get("boards", 4) * size * _prefix_entries(case["n"], case["k"]), "flops": 0}
    if kind == "serve":
        ns = range(case["n_lo"], case["n_hi"] + 1)
        one = sum(_prefix_entries(n, k) for n in ns for k in range(4)) / (4 * len(ns))
        return {"bytes": 16 * case["requests"] * one, "flops": 0}
    n = case["n"]
    board = float(sum(_entries(n)))
    if kind == "board" and not case.get("symmetry", 1):
        board *= 2
    if kind == "sites":
        board *= n  # one boundary a site
    if kind == "explicit":
        board *= n * 1.5  # 24-byte entries, one boundary a site
    return {"bytes": 16 * (board + _branches(case) * _prefix_entries(n, _prefix_rows(case))), "flops": 0}


# ---- the same numbers in plain torch -----------------------------------------


def _contract(n: int, prefix, symmetry: bool):
    """Rows of the contraction with whole 64-bit weights: the layers, the
    count and the largest boundary."""
    mask = (1 << n) - 1
    dev = "cuda" if torch.cuda.is_available() else "cpu"

    def after(cols, dr, dl, bit):
        return cols | bit, ((dr | bit) << 1) & mask, (dl | bit) >> 1

    cols = dr = dl = 0
    for c in prefix:
        if (cols | dr | dl) >> c & 1:
            return [], 0, 1
        cols, dr, dl = after(cols, dr, dl, 1 << c)
    state = [torch.tensor([v], dtype=torch.int64, device=dev) for v in (cols, dr, dl)]
    weight = torch.ones(1, dtype=torch.int64, device=dev)
    layers, peak = [], 1
    for row in range(len(prefix), n):
        keys, weights, matched = [], [], 0
        read = weight.numel()
        for c in range(n):
            bit = 1 << c
            free = (state[0] | state[1] | state[2]) & bit == 0
            matched += int(free.sum())
            w = weight[free]
            if row == 0 and symmetry:
                if 2 * c > n - 1:
                    continue
                w = w * (2 if 2 * c < n - 1 else 1)
            a, b, d = after(state[0][free], state[1][free], state[2][free], bit)
            keys.append(a | b << n | d << 2 * n)
            weights.append(w)
        key, w = torch.cat(keys), torch.cat(weights)
        done = key.numel()
        key, where = torch.unique(key, return_inverse=True)
        weight = torch.zeros(key.numel(), dtype=torch.int64, device=dev).index_add_(0, where, w)
        state = [key & mask, key >> n & mask, key >> 2 * n & mask]
        layers.append([row, read, n * read, matched, done, key.numel(), int(weight.sum())])
        peak = max(peak, key.numel())
    return layers, int(weight[state[0] == mask].sum()), peak


def _exact_counts(boards) -> np.ndarray:
    out = []
    for n, prefix in boards:
        layers, count, peak = _contract(n, prefix, False)
        out.append([count, peak, sum(l[2] for l in layers), sum(l[3] for l in layers)])
    return np.array(out, dtype=np.int64)


def exact(case: dict, seed: int):
    kind = case["kind"]
    boards = _draws(case, seed)
    if kind == "serve":
        one = {}
        for n, prefix in boards:
            if (n, tuple(prefix)) not in one:
                one[n, tuple(prefix)] = _contract(n, prefix, False)[1] if prefix else KNOWN[n]
        return {"counts": np.array([one[n, tuple(p)] for n, p in boards], dtype=np.int64)}
    if kind == "prefix":
        if case["n"] > 21 or _prefix_entries(case["n"], case["k"]) > 4e8:
            return None
        return {"counts": _exact_counts(boards)}
    n = case["n"]
    branches = _exact_counts(boards)
    if kind == "explicit":
        return {"board": None, "branches": branches}
    layers, count, peak = None, KNOWN[n], None
    if kind == "board" and n <= 15:
        layers, count, peak = _contract(n, [], bool(case.get("symmetry", 1)))
        layers = np.array(layers, dtype=np.int64)
    return {"count": count, "peak": peak, "layers": layers, "branches": branches}
