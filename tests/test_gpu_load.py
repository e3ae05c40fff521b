"""Loaders: temporal rows over raw ids, batches of databases, counts of rows with items."""
import numpy as np
import pytest


def _csr(rng, n, items, mean, step=1):
    lengths = rng.poisson(mean, n)
    lengths[rng.random(n) < 0.1] = 0  # empty rows
    offsets = np.zeros(n + 1, dtype=np.uint64)
    np.cumsum(lengths, out=offsets[1:])
    return offsets, (rng.integers(0, items, int(offsets[-1])) * step).astype(np.uint32)


@pytest.mark.parametrize("n", [0, 1, (1 << 14) - 1, 1 << 14, (1 << 17) + 1])
def test_rows_with_items(n):
    from cupami_b200 import _native

    offsets, _ = _csr(np.random.default_rng(n), n, 10, 1.0)
    assert _native.count_rows(offsets) == int((np.diff(offsets.astype(np.int64)) > 0).sum())


# Ids below and above 2**23: the library's table, or NumPy's ranks.
@pytest.mark.gpu
@pytest.mark.parametrize("n,items,step", [(0, 1, 1), (1, 3, 1), (700, 40, 1), (700, 40, 1638),
                                          (20000, 60, (1 << 23) // 60), (20000, 60, (1 << 23) // 59 + 1),
                                          (700, 40, 1 << 24)])
def test_temporal_ids_match_the_oracle(n, items, step):
    from cupami_b200 import cuPFApriori, cuPFEclat
    from cupami_b200.datasets import TemporalCSR
    from oracle import periodic

    rng = np.random.default_rng(items + step)
    offsets, ids = _csr(rng, n, items, 4.0, step)
    stamps = rng.integers(0, 2 * n + 1, n)  # rows out of order, stamps shared
    minsup, maxper = max(1, n // 12), max(2, n // 8)
    rows = [[int(stamps[r]), *ids[int(offsets[r]):int(offsets[r + 1])].tolist()] for r in range(n)]
    for cls, algo in ((cuPFEclat, "eclat"), (cuPFApriori, "apriori")):
        m = cls(TemporalCSR(offsets, ids, stamps), minsup, maxper)
        m.mine()
        # The oracle drops rows without items' text only when they are blank: a stamp is not.
        want = periodic.mine(rows, minsup, maxper, algo, None)
        assert list(m.getPatterns().items()) == [(k, tuple(v)) for k, v in want.items()]
        assert m._timestamps == sorted(stamps.tolist())


@pytest.mark.gpu
# Presence bitmaps in shared memory, in device memory; ids of 2**26 and more: one database after the other.
@pytest.mark.parametrize("step", [1, 1 << 14, 1 << 23])
def test_batch_of_uneven_databases(oracle_lib, step):
    from cupami_b200 import TransactionCSR, cuEclat

    rng = np.random.default_rng(step)
    sizes = [0, 1, 40000, 3, 0, 900, 1, 257, 5000]
    sources = [TransactionCSR(*_csr(rng, n, 30, 5.0, step), 30 * step) for n in sizes]
    miners = cuEclat.mineBatch(sources, 0.02)
    for source, miner in zip(sources, miners):
        rows = int((np.diff(source.offsets.astype(np.int64)) > 0).sum())
        alone = cuEclat(source, 0.02)
        alone.mine()
        assert miner._transactionCount == rows
        assert list(miner.getPatterns().items()) == list(alone.getPatterns().items())
        if rows:
            labels, arrays = oracle_lib.mine_csr(source.offsets, source.items, miner._minSup, "eclat")
            assert miner.getPatterns() == oracle_lib.to_dict(labels, arrays)
