"""What a user of the engine has it do, as cases to time: single pairs from a
read against its window up to 2^20 x 2^20, batches of reads and of longer
strings, the host entry points, braid products and substring queries.

Sizes and contents are those of the benchmark workloads (slcs/workloads.py)
and of the cost model's sweep: sides from 64 to 262144, alphabets of 2, 4, 20
and 256 symbols, uniform strings or mutated copies.  Every output is a whole
number (strand ids, permutation entries, LCS lengths).
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "platform-independent-lcs_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import slcs  # noqa: E402
from slcs import workloads as W  # noqa: E402

SIGMAS = (2, 4, 20, 256)


def listed():
    return [
        # One read against its window: the smallest call, where latency counts.
        {"name": "pair_read", "kind": "pair", "m": 152, "n": 187, "sigma": 4, "mutated": True},
        # The benchmark's plain pair.
        {"name": "pair_4096", "kind": "pair", "m": 4096, "n": 4096, "sigma": 4, "mutated": False},
        # Two protein-like sequences of odd lengths.
        {"name": "pair_20011", "kind": "pair", "m": 20011, "n": 9973, "sigma": 20, "mutated": False},
        # A query against a long text: few rows, many columns.
        {"name": "pair_wide", "kind": "pair", "m": 1003, "n": 250007, "sigma": 4, "mutated": False},
        # The benchmark's two related sequences (10 % substitutions, indels).
        {"name": "pair_131072", "kind": "pair", "m": 131072, "n": 131072, "sigma": 4, "mutated": True},
        # The benchmark's long pair, the largest call.
        {"name": "pair_1048576", "kind": "pair", "m": 1 << 20, "n": 1 << 20, "sigma": 4, "mutated": False},
        # The benchmark's batch of 20,000 reads, inputs and strands on the device.
        {"name": "reads_20000", "kind": "reads", "pairs": 20000, "host": False, "graph": False},
        # The same end to end from pinned host buffers, strands as int16.
        {"name": "reads_20000_host", "kind": "reads", "pairs": 20000, "host": True, "graph": False},
        # A small batch of longer, uneven strings (sweep shapes), replayed as a graph.
        {"name": "batch_uneven", "kind": "batch", "pairs": 96, "m": 2900, "n": 3300, "sigma": 20, "graph": True},
        # A program of the reference's interface: Word symbols in host arrays.
        {"name": "words_host", "kind": "words", "m": 5003, "n": 7001, "sigma": 100},
        # Gluing two separately combed column strips of one pair.
        {"name": "braid_32768", "kind": "braid", "k": 32768, "p": 20000, "q": 30001, "row_glue": False},
        # Semi-local answers from one comb's strands.
        {"name": "queries", "kind": "queries", "m": 6000, "n": 50001, "queries": 20000},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pair", "pair", "pair", "pair", "reads", "reads", "batch", "batch", "words", "braid", "queries"])
    if kind == "pair":
        return {"kind": kind, "m": _log_uniform(rng, 64, 262144), "n": _log_uniform(rng, 64, 262144),
                "sigma": rng.choice(SIGMAS), "mutated": rng.random() < 0.5}
    if kind == "reads":
        host = rng.random() < 0.5
        return {"kind": kind, "pairs": _log_uniform(rng, 64, 20000), "host": host,
                "graph": not host and rng.random() < 0.5}
    if kind == "batch":
        m, n = _log_uniform(rng, 64, 16384), _log_uniform(rng, 64, 16384)
        pairs = min(_log_uniform(rng, 1, 4096), max(1, 2_000_000_000 // (m * n)))
        return {"kind": kind, "pairs": pairs, "m": m, "n": n, "sigma": rng.choice(SIGMAS),
                "graph": rng.random() < 0.5}
    if kind == "words":
        return {"kind": kind, "m": _log_uniform(rng, 64, 65536), "n": _log_uniform(rng, 64, 65536),
                "sigma": rng.choice(SIGMAS)}
    if kind == "braid":
        return {"kind": kind, "k": _log_uniform(rng, 512, 262144), "p": _log_uniform(rng, 512, 65536),
                "q": _log_uniform(rng, 512, 65536), "row_glue": rng.random() < 0.5}
    return {"kind": kind, "m": _log_uniform(rng, 64, 65536), "n": _log_uniform(rng, 1024, 262144),
            "queries": _log_uniform(rng, 64, 100000)}


def _strings(rng, m, n, sigma, mutated):
    a = W.uniform(rng, m, sigma)
    if mutated:
        b = W.fit_length(rng, W.mutate(rng, a, 0.10, 0.01, 0.01, sigma), n, sigma)
    else:
        b = W.uniform(rng, n, sigma)
    return a, b


def _padded_offsets(lens):
    off = np.zeros(len(lens) + 1, np.int64)
    np.cumsum((lens + 15) // 16 * 16, out=off[1:])
    return off


def _spread(off, lens):
    """Index of every symbol of strings that start at `off` and have `lens` symbols."""
    first = np.cumsum(lens) - lens
    return np.repeat(off - first, lens) + np.arange(int(lens.sum()))


def _reads(rng, pairs):
    """Reads against windows: W.reads_20000's lengths and error rates, whole arrays at a time.
    Lengths and indels follow from the batch size, symbols and substitutions from rng."""
    shape = np.random.default_rng(pairs)
    sd = math.sqrt(math.log(1.0 + 60.0 ** 2 / 150.0 ** 2))
    read = np.clip(np.round(shape.lognormal(math.log(150.0) - sd * sd / 2, sd, pairs)), 50, 1000).astype(np.int64)
    win = np.round(read * shape.uniform(1.0, 1.5, pairs)).astype(np.int64)
    b_off = _padded_offsets(win)
    b = rng.integers(0, 4, int(b_off[-1]) + 16, dtype=np.uint8)
    start = (rng.random(pairs) * (win - read + 1)).astype(np.int64)
    sym = b[_spread(b_off[:-1] + start, read)]
    sub = rng.random(len(sym)) < 0.05
    sym[sub] = (sym[sub] + rng.integers(1, 4, int(sub.sum()), dtype=np.uint8)) % 4
    u = shape.random(len(sym))
    times = np.where(u < 0.005, 0, np.where(u < 0.01, 1 + shape.geometric(1 / 3.0, len(sym)), 1))
    ends = np.cumsum(read)
    ms = np.add.reduceat(times, ends - read)
    sym = np.repeat(sym, times)
    a_off = _padded_offsets(ms)
    a = np.zeros(int(a_off[-1]) + 16, np.uint8)
    a[_spread(a_off[:-1], ms)] = sym
    return W.Batch(a, b, a_off[:-1], b_off[:-1], ms.astype(np.int32), win.astype(np.int32))


def _uneven(rng, pairs, m, n, sigma):
    """Pairs of uneven sides: between half of m and m rows, half of n and n columns
    (the same sides for every rng)."""
    shape = np.random.default_rng(pairs)
    ms = shape.integers((m + 1) // 2, m + 1, pairs)
    ns = shape.integers((n + 1) // 2, n + 1, pairs)
    a_off, b_off = _padded_offsets(ms), _padded_offsets(ns)
    a = rng.integers(0, sigma, int(a_off[-1]) + 16, dtype=np.uint8)
    b = rng.integers(0, sigma, int(b_off[-1]) + 16, dtype=np.uint8)
    return W.Batch(a, b, a_off[:-1], b_off[:-1], ms.astype(np.int32), ns.astype(np.int32))


def _pinned(x):
    return torch.from_numpy(x).pin_memory().numpy()


def _permutation(a, b):
    return slcs.strands_to_permutation(*slcs.comb_pair(a, b))[0]


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "pair":
        a, b = _strings(rng, case["m"], case["n"], case["sigma"], case["mutated"])
        return kind, torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    if kind in ("reads", "batch"):
        if kind == "reads":
            batch = _reads(rng, case["pairs"])
        else:
            batch = _uneven(rng, case["pairs"], case["m"], case["n"], case["sigma"])
        _, total = batch.strand_offsets()
        plan = slcs.BatchPlan(slcs.pair_descs(batch), slcs.Config.make(use_graph=1 if case["graph"] else 0))
        if kind == "reads" and case["host"]:
            out = torch.empty(total, dtype=torch.int16, pin_memory=True).numpy()
            return "host", plan, _pinned(batch.a_blob), _pinned(batch.b_blob), out
        out = torch.empty(total, dtype=torch.int32, device="cuda")
        return kind, plan, torch.from_numpy(batch.a_blob).cuda(), torch.from_numpy(batch.b_blob).cuda(), out
    if kind == "words":
        a, b = _strings(rng, case["m"], case["n"], case["sigma"], False)
        words = rng.permutation(1 << 20)[:case["sigma"]].astype(np.int32)
        return kind, words[a], words[b]
    if kind == "braid":
        shared = torch.from_numpy(W.uniform(rng, case["k"])).cuda()
        x, y = (torch.from_numpy(W.uniform(rng, case[s])).cuda() for s in ("p", "q"))
        if case["row_glue"]:
            p, q = _permutation(x, shared), _permutation(y, shared)
        else:
            p, q = _permutation(shared, x), _permutation(shared, y)
        return kind, p, q, case["k"], case["row_glue"]
    a, b = _strings(rng, case["m"], case["n"], 4, False)
    _, v = slcs.comb_pair(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda())
    ends = np.sort(rng.integers(0, case["n"] + 1, (case["queries"], 2)), axis=1).astype(np.int32)
    begin, end = (torch.from_numpy(np.ascontiguousarray(ends[:, i])).cuda() for i in (0, 1))
    return "queries", v.clone(), case["m"], begin, end


def run(state):
    kind = state[0]
    if kind == "pair":
        return slcs.comb_pair(state[1], state[2])
    if kind in ("reads", "batch"):
        _, plan, a, b, out = state
        plan.run(a, b, out)
        return out
    if kind == "host":
        _, plan, a, b, out = state
        plan.run_host16(a, b, out)
        return out
    if kind == "words":
        return slcs.comb_pair_words_host(state[1], state[2])
    if kind == "braid":
        _, p, q, k, row_glue = state
        return slcs.braid_multiply(p, q, k, row_glue)
    _, v, m, begin, end = state
    return slcs.substring_llcs(v, m, begin, end)


def work(case):
    """Bytes in and out once; operations: 5 per cell of a comb (a compare, a
    min, a max and two selects), one per permutation entry or strand read."""
    kind = case["kind"]
    if kind == "pair":
        m, n = case["m"], case["n"]
        return {"bytes": 5 * (m + n), "flops": 5 * m * n}
    if kind == "reads":  # 151 rows and 187 columns on average
        pairs, out = case["pairs"], 2 if case["host"] else 4
        return {"bytes": pairs * (1 + out) * 338, "flops": pairs * 5 * 32800}
    if kind == "batch":
        pairs, m, n = case["pairs"], 0.75 * case["m"], 0.75 * case["n"]
        return {"bytes": pairs * 5 * (m + n), "flops": pairs * 5 * m * n}
    if kind == "words":
        m, n = case["m"], case["n"]
        return {"bytes": 8 * (m + n), "flops": 5 * m * n}
    if kind == "braid":
        k, p, q = case["k"], case["p"], case["q"]
        return {"bytes": 4 * (3 * k + 2 * p + 2 * q), "flops": 2 * k + p + q}
    return {"bytes": 4 * case["n"] + 12 * case["queries"], "flops": case["queries"] * case["n"] / 3}
