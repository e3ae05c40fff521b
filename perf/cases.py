"""Measured workloads: what a program has this package do, each through its public entry points.

A case names an input family, its sizes and the call.  ``prepare`` makes the
input from the seed (on the GPU, then in the form the call takes: host arrays
for the miners, CUDA tensors for the kernel functions, a file for the text
reader), ``run`` makes one whole call from that input to the patterns.  The
miners load their input on every call, as the classes do for their users.
"""

from __future__ import annotations

import math
import tempfile
from pathlib import Path

import numpy as np
import torch

from cupami_b200 import cuApriori, cuEclat, cuPFApriori, cuPFEclat
from cupami_b200.datasets import TemporalCSR, TransactionCSR
from cupami_b200.frequentPattern import _bitsets

_MINERS = {"eclat": cuEclat, "apriori": cuApriori}
_PERIODIC = {"pfeclat": cuPFEclat, "pfapriori": cuPFApriori}


def listed():
    return [
        # The quickstart shape: a few thousand baskets of a small shop.  Latency and launches.
        {"name": "eclat-uniform-10k", "call": "eclat", "data": "uniform", "n": 10_000, "items": 50, "mean": 6.0,
         "minsup": 0.01},
        # Market baskets with planted patterns, the ordinary single database, by both miners.
        {"name": "eclat-planted-100k", "call": "eclat", "data": "planted", "n": 100_000, "items": 1_000, "mean": 10.0,
         "minsup": 0.005},
        {"name": "apriori-planted-100k", "call": "apriori", "data": "planted", "n": 100_000, "items": 1_000,
         "mean": 10.0, "minsup": 0.005},
        # Few items held by most transactions: a deep lattice of dense tidsets.
        {"name": "eclat-dense-64k", "call": "eclat", "data": "dense", "n": 65_536, "items": 128, "minsup": 0.6},
        # Large sparse logs, an ordinary one of odd size and the largest.
        {"name": "eclat-sparse-250k", "call": "eclat", "data": "sparse", "n": 250_007, "items": 20_000, "mean": 40.0,
         "minsup": 0.002},
        {"name": "eclat-sparse-1m", "call": "eclat", "data": "sparse", "n": 1_000_000, "items": 20_000, "mean": 40.0,
         "minsup": 0.001},
        # Very long tidsets over few items (a year of receipts over product groups).
        {"name": "eclat-long-2m", "call": "eclat", "data": "zipf", "n": 2_000_003, "items": 400, "mean": 8.0,
         "minsup": 0.004},
        # Many independent databases in one call (one per store), sizes from 1,000 to 200,000.
        {"name": "batch-512", "call": "batch", "data": "zipf", "databases": 512, "low": 1_000, "high": 200_000,
         "items": 200, "mean": 8.0, "minsup": 0.01},
        # Periodic-frequent patterns of a temporal database given as integer arrays.
        {"name": "pfeclat-100k", "call": "pfeclat", "data": "temporal", "n": 100_000, "items": 200, "mean": 6.0,
         "minsup": 0.005, "maxper": 0.0167},
        # The kernel functions under a caller's own search: tidsets from occurrences and one
        # full batch of pair supports; then a batch of extensions of one prefix.
        {"name": "kernels-pairs", "call": "pairs", "data": "planted", "n": 100_000, "items": 1_000, "mean": 10.0,
         "candidates": 65_536, "width": 2},
        {"name": "kernels-extend", "call": "extend", "n": 1_000_000, "extensions": 512},
        # A comma-separated file of integer baskets, from the path to the patterns.
        {"name": "text-200k", "call": "text", "data": "planted", "n": 200_000, "items": 500, "mean": 8.0,
         "minsup": 0.01},
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    call = rng.choice(["eclat", "eclat", "eclat", "apriori", "long", "batch", "pfeclat", "pfapriori", "pairs",
                       "extend", "text"])
    if call in ("eclat", "apriori"):
        data = rng.choice(["uniform", "planted", "dense", "sparse"] if call == "eclat" else ["uniform", "planted"])
        if data == "uniform":
            return {"call": call, "data": data, "n": _log(rng, 1_000, 60_000), "items": rng.randint(20, 90),
                    "mean": rng.uniform(3, 9), "minsup": rng.uniform(0.01, 0.03)}
        if data == "planted":
            return {"call": call, "data": data, "n": _log(rng, 5_000, 400_000), "items": _log(rng, 150, 3_000),
                    "mean": rng.uniform(6, 12), "minsup": rng.uniform(0.005, 0.02)}
        if data == "dense":
            return {"call": call, "data": data, "n": _log(rng, 2_000, 130_000), "items": rng.randint(40, 128),
                    "minsup": rng.uniform(0.6, 0.75)}
        return {"call": call, "data": data, "n": _log(rng, 60_000, 700_000), "items": _log(rng, 5_000, 20_000),
                "mean": rng.uniform(20, 40), "minsup": rng.uniform(0.002, 0.006)}
    if call == "long":
        return {"call": "eclat", "data": "zipf", "n": _log(rng, 1_200_000, 2_500_000), "items": _log(rng, 60, 500),
                "mean": rng.uniform(4, 8), "minsup": rng.uniform(0.004, 0.01)}
    if call == "batch":
        return {"call": call, "data": "zipf", "databases": _log(rng, 2, 300), "low": 1_000,
                "high": _log(rng, 20_000, 200_000), "items": _log(rng, 50, 300), "mean": rng.uniform(4, 9),
                "minsup": rng.uniform(0.01, 0.03)}
    if call in ("pfeclat", "pfapriori"):
        return {"call": call, "data": "temporal", "n": _log(rng, 5_000, 400_000), "items": _log(rng, 50, 400),
                "mean": rng.uniform(4, 8), "minsup": rng.uniform(0.005, 0.02), "maxper": rng.uniform(0.01, 0.05)}
    if call == "pairs":
        return {"call": call, "data": "planted", "n": _log(rng, 2_000, 300_000), "items": _log(rng, 100, 1_200),
                "mean": rng.uniform(5, 10), "candidates": _log(rng, 500, 65_536), "width": rng.randint(2, 4)}
    if call == "extend":
        return {"call": call, "n": _log(rng, 3_000, 1_500_000), "extensions": _log(rng, 8, 500)}
    return {"call": "text", "data": "planted", "n": _log(rng, 5_000, 200_000), "items": _log(rng, 100, 1_000),
            "mean": rng.uniform(4, 10), "minsup": rng.uniform(0.01, 0.03)}


# ---- inputs ------------------------------------------------------------------


def _baskets(g, n, mean, sample, prefix=None, high=None):
    """Baskets of Poisson(mean) distinct items (at least one) from the i.i.d. stream ``sample``:
    per row the first distinct values, ascending; with ``prefix`` those come first and are kept.
    Returns (lengths int64[n], items uint32) as host arrays."""
    width = min(250, int(2 * mean + 24) + (0 if prefix is None else prefix.shape[1]))
    lengths, pieces = [], []
    for start in range(0, n, 1 << 17):
        rows = min(n, start + (1 << 17)) - start
        want = torch.poisson(torch.full((rows,), float(mean), device="cuda"), generator=g).clamp_(min=1, max=high)
        draws = sample(g, (rows, width))
        if prefix is not None:
            p = prefix[start:start + rows]
            want = torch.maximum(want, (p >= 0).sum(1).to(want.dtype))
            draws[:, :p.shape[1]] = torch.where(p >= 0, p, draws[:, -1:])
        key, _ = torch.sort(draws * 256 + torch.arange(width, dtype=torch.int32, device="cuda"), dim=1)
        value, pos = key >> 8, (key & 255).long()
        first = torch.ones_like(value, dtype=torch.bool)
        first[:, 1:] = value[:, 1:] != value[:, :-1]
        in_stream = torch.zeros_like(first).scatter_(1, pos, first)
        taken = in_stream & (in_stream.to(torch.int32).cumsum(1) <= want[:, None])
        keep = taken.gather(1, pos)
        lengths.append(keep.sum(1))
        pieces.append(value[keep].to(torch.int32))
    items = torch.cat(pieces).cpu().numpy().view(np.uint32)
    return torch.cat(lengths).cpu().numpy(), items


def _zipf(items, s):
    w = 1.0 / torch.arange(1, items + 1, dtype=torch.float64, device="cuda") ** s
    cdf = (torch.cumsum(w, 0) / w.sum()).to(torch.float32)

    def sample(g, shape):
        u = torch.rand(shape, generator=g, device="cuda")
        return (torch.searchsorted(cdf, u, out_int32=True).clamp_(max=items - 1) + 1).to(torch.int32)

    return sample


def _pool(g, count, mean, items, sample):
    """``count`` planted patterns of max(1, Poisson(mean)) items, padded with -1."""
    lengths, flat = _baskets(g, count, mean, sample, high=min(items, 24))
    pool = np.full((count, int(lengths.max())), -1, dtype=np.int32)
    pool[np.arange(pool.shape[1])[None, :] < lengths[:, None]] = flat
    return torch.from_numpy(pool).cuda()


def _offsets(lengths):
    offsets = np.zeros(lengths.size + 1, dtype=np.uint64)
    np.cumsum(lengths, out=offsets[1:])
    return offsets


def _database(case, seed):
    """Lengths and items of the case's baskets (datasets.py's families, drawn on the GPU)."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n, items, data = case["n"], case["items"], case["data"]
    if data == "uniform":
        return _baskets(g, n, case["mean"], lambda g, shape: torch.randint(
            1, items + 1, shape, generator=g, device="cuda", dtype=torch.int32), high=items)
    if data == "dense":
        rng = np.random.default_rng(seed)
        p = torch.from_numpy(rng.beta(5.0, 2.0, items).astype(np.float32)).cuda()
        m = torch.rand((n, items), generator=g, device="cuda") < p
        return m.sum(1).cpu().numpy(), (m.nonzero()[:, 1] + 1).to(torch.int32).cpu().numpy().view(np.uint32)
    if data == "planted":
        sample = _zipf(items, 1.1)
        pool = _pool(g, 2_000, 4.0, items, sample)
        choice = torch.randint(0, pool.shape[0], (n,), generator=g, device="cuda")
        return _baskets(g, n, case["mean"], sample, prefix=pool[choice], high=items)
    if data == "temporal":
        sample = _zipf(items, 1.1)
        pool = _pool(g, 40, 3.0, items, sample)
        pool = torch.cat([pool, torch.full_like(pool[:1], -1)])
        choice = torch.randint(0, 40, (n,), generator=g, device="cuda")
        choice[torch.rand(n, generator=g, device="cuda") >= 0.35] = 40
        lengths, flat = _baskets(g, n, case["mean"], sample, prefix=pool[choice], high=items)
        full = np.random.default_rng(seed).random(n) >= 0.02  # the rest are empty baskets
        return np.where(full, lengths, 0), flat[np.repeat(full, lengths)]
    return _baskets(g, n, case["mean"], _zipf(items, 1.0 if data == "sparse" else 1.1), high=items)


def _batch(case, seed):
    """Independent databases of log-uniform sizes over the same item ids."""
    rng = np.random.default_rng(seed)
    sizes = np.exp(rng.uniform(math.log(case["low"]), math.log(case["high"]), case["databases"])).astype(np.int64)
    lengths, items = _database({**case, "n": int(sizes.sum())}, seed)
    bounds = np.concatenate([[0], np.cumsum(sizes)])
    offsets = _offsets(lengths)
    out = []
    for a, b in zip(bounds[:-1], bounds[1:]):
        o = offsets[a:b + 1]
        out.append(TransactionCSR(o - o[0], items[int(o[0]):int(o[-1])], case["items"]))
    return out


# A program collects its patterns in arrays it keeps: their sizes go with the case, above
# what any seed finds (_collect raises otherwise), and the unused ends stay zero.
_MOST = {"uniform": 1 << 18, "planted": 1 << 18, "dense": 1 << 21, "zipf": 1 << 18, "temporal": 1 << 17}


def _buffers(case):
    if case["call"] in _PERIODIC:
        most = _MOST["temporal"]
        return {"size": np.zeros(2, np.int64), "patterns": np.zeros(32 * most, np.uint8),
                "values": np.zeros((most, 2), np.int64)}
    most = int(9000 / case["minsup"]) if case["data"] == "sparse" else _MOST[case["data"]]
    if case["call"] == "batch":
        most = 8_192 * case["databases"]
    return {"size": np.zeros(3, np.int64), "offsets": np.zeros(most + 1, np.uint64),
            "items": np.zeros(7 * most, np.uint32), "supports": np.zeros(most, np.uint64),
            "labels": np.zeros(case["items"], np.int64)}


def _collect(into, **found):
    for k, (name, parts) in enumerate(found.items()):
        dst, at = into[name], 0
        for x in parts:
            if at + len(x) > len(dst):
                raise ValueError(f"{name}: more than {len(dst)} values")
            if x.size < 1 << 20:
                dst[at:at + len(x)] = x
            else:  # copied by several threads
                torch.from_numpy(dst[at:at + len(x)]).copy_(torch.from_numpy(x))
            at += len(x)
        if k < len(into["size"]):
            into["size"][k] = at
    return into


def prepare(case, seed):
    call = case["call"]
    if call == "batch":
        return call, _batch(case, seed), case["minsup"], _buffers(case)
    if call == "extend":
        g = torch.Generator(device="cuda").manual_seed(seed)
        words = (case["n"] + 31) // 32
        # Rows held by an eighth to a half of the transactions.
        bits = torch.randint(-2**31, 2**31, (case["extensions"] + 1, words), generator=g, device="cuda",
                             dtype=torch.int64).to(torch.int32)
        thin = torch.randint(-2**31, 2**31, (case["extensions"] + 1, words), generator=g, device="cuda",
                             dtype=torch.int64).to(torch.int32)
        bits[1::2] &= thin[1::2]
        return call, bits[0].clone(), bits[1:].clone()
    lengths, items = _database(case, seed)
    if call in _MINERS:
        return call, TransactionCSR(_offsets(lengths), items, case["items"]), case["minsup"], _buffers(case)
    if call in _PERIODIC:
        stamps = np.cumsum(np.random.default_rng(seed + 1).integers(0, 4, case["n"])).astype(np.int64)
        return call, TemporalCSR(_offsets(lengths), items, stamps), case["minsup"], case["maxper"], _buffers(case)
    if call == "text":
        text = items.astype(str).tolist()
        ends = np.cumsum(lengths)
        rows = (",".join(text[e - k:e]) for e, k in zip(ends.tolist(), lengths.tolist()))
        folder = tempfile.TemporaryDirectory(prefix="baskets_")
        path = Path(folder.name) / "baskets.csv"
        path.write_text("\n".join(rows) + "\n", encoding="utf-8")
        return call, str(path), case["minsup"], _buffers(case), folder
    # pairs: one (row, column) per occurrence on the device, and a batch of candidates
    xp = _bitsets.array_module()
    rows = xp.asarray(np.repeat(np.arange(case["n"], dtype=np.uint64), lengths), dtype=xp.uint64)
    cols = xp.asarray(items - np.uint32(1), dtype=xp.uint32)
    rng = np.random.default_rng(seed)
    cand = rng.integers(0, case["items"] - case["width"], (case["candidates"], case["width"]), dtype=np.int64)
    cand = (np.sort(cand, axis=1) + np.arange(case["width"])).astype(np.uint32)  # increasing columns
    return call, rows, cols, case["n"], case["items"], cand


def _arrays(miner, into):
    offsets, items, supports, labels = miner.getPatternArrays()
    return _collect(into, offsets=[offsets], items=[items], supports=[supports],
                    labels=[np.array(list(map(int, labels)), dtype=np.int64)])


def run(state):
    call = state[0]
    if call in _MINERS or call == "text":
        miner = _MINERS.get(call, cuApriori)(state[1], state[2])
        miner.mine()
        return _arrays(miner, state[3])
    if call == "batch":
        found = [m.getPatternArrays() for m in cuEclat.mineBatch(state[1], state[2])]
        return _collect(state[3], offsets=[f[0] for f in found], items=[f[1] for f in found],
                        supports=[f[2] for f in found])
    if call in _PERIODIC:
        miner = _PERIODIC[call](state[1], state[2], state[3])
        miner.mine()
        found = miner.getPatterns()
        return _collect(state[4], patterns=[np.frombuffer("\n".join(found).encode(), dtype=np.uint8)],
                        values=[np.array(list(found.values()), dtype=np.int64).reshape(-1, 2)])
    xp = _bitsets.array_module()
    if call == "extend":
        children, supports = _bitsets.intersect_extensions(xp, state[1], state[2])
        return {"children": children, "supports": np.array(supports, dtype=np.int64)}
    _, rows, cols, n, items, cand = state
    bitsets = _bitsets.build_bitsets(xp, rows, cols, n, items)
    supports = _bitsets.count_supports(xp, bitsets, cand)
    return {"bitsets": bitsets, "supports": np.array(supports, dtype=np.int64)}


def work(case):
    call = case["call"]
    if call == "extend":
        row = (case["n"] + 31) // 32 * 4
        return {"bytes": row * (2 * case["extensions"] + 1) + 8 * case["extensions"], "flops": 0}
    if call == "batch":
        span = math.log(case["high"] / case["low"])
        n = case["databases"] * (case["high"] - case["low"]) / span
    else:
        n = case["n"]
    # Occurrences read once as the call gets them (4-byte ids and 8-byte offsets, text, or
    # row and column tensors); the tidsets that every support is counted from written and read once.
    nnz = n * (case["items"] * 5 / 7 if case["data"] == "dense" else case["mean"])
    bits = n / 8 * case["items"]
    if call == "pairs":
        return {"bytes": 12 * nnz + 2 * bits + case["candidates"] * (4 * case["width"] + 8), "flops": 0}
    if case["data"] == "sparse":
        bits = 4 * nnz  # sparse items as lists
    if call == "text":
        return {"bytes": 4 * nnz + 2 * bits, "flops": 0}
    return {"bytes": 4 * nnz + 8 * n + 2 * bits + (8 * n if case["data"] == "temporal" else 0), "flops": 0}


def exact(case, seed):
    """Supports are whole numbers, equal or wrong; the kernel functions' are also given from NumPy."""
    if case["call"] == "extend":
        _, prefix, extensions = prepare(case, seed)
        children = prefix & extensions
        bits = children.cpu().numpy().view(np.uint32)
        return {"children": children, "supports": np.bitwise_count(bits).astype(np.int64).sum(1)}
    return None
