"""GPU: which engine a search runs on, and what it counts of it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mined(held, minsup):
    from cupami_b200 import _native

    offsets = np.zeros(held.shape[0] + 1, dtype=np.uint64)
    np.cumsum(held.sum(axis=1), out=offsets[1:])
    db = _native.Database.from_columns(_native.context(0), offsets, np.nonzero(held)[1], held.shape[1])
    return db.mine(minsup, _native.CPM_ECLAT).stats


# Baskets of exactly two or three of 40 items, every pair and triple frequent.  No frame survives below
# the pairs of two items.  Of three, each basket is one row of the class of its first item (two
# elements, one of them listed: 12 bytes), and is met once more by its first two items' unit (an
# occurrence and an element: 10 bytes); no basket is left below those.
@pytest.mark.parametrize("size,per_basket", [(2, 0), (3, 22)])
def test_bytes_of_conditional_rows(size, per_basket):
    n, items = 1_000_000, 40
    rng = np.random.default_rng(size)
    held = np.zeros((n, items), bool)
    np.put_along_axis(held, np.argsort(rng.random((n, items)), axis=1)[:, :size], True, axis=1)
    s = _mined(held, 40)
    assert s["n_patterns"] == 40 + 780 + (9880 if size == 3 else 0)
    assert s["row_units"] == s["work_items"] and (size == 2 or s["row_units"] > 0)
    assert s["bytes_alg"] == per_basket * n


# The dispatch by work: pairs counted from the rows or multiplied, deep levels over conditional rows
# (all of their units below the classes) or over tidsets (root units of the classes besides).
@pytest.mark.parametrize("n,items,mean,minsup,row_pairs,rows", [
    (4097, 700, 6, 12, False, False), (8191, 300, 15, 60, True, True), (16385, 400, 30, 480, False, True),
    (70001, 600, 60, 7000, False, False), (20000, 2500, 12, 30, True, True), (131073, 90, 4, 150, True, True),
    (2048, 500, 50, 150, False, False), (400000, 200, 20, 1600, False, True),
    # too short a search for its rows to be used again (uniform 10,000 x 50)
    (10000, 50, 6, 100, False, False),
    # long tidsets and few candidates: rows measured 1.5 to 4 times slower than the walk
    (400000, 200, 20, 4000, False, False), (600000, 60, 4, 6000, True, False), (600000, 200, 6, 3600, True, False)])
def test_engine_by_work(n, items, mean, minsup, row_pairs, rows):
    rng = np.random.default_rng(n)
    w = 1.0 / np.arange(1, items + 1) ** 0.9
    s = _mined(rng.random((n, items)) < np.minimum(0.97, w * mean / w.sum()), minsup)
    assert (s["pair_ops"] == 0) == row_pairs
    assert s["work_items"] > 0 and (s["work_items"] == s["projected_units"] + s["row_units"]) == rows


# Batches: a CTA per item and database costs small databases more than the Gram of them all; of
# tall databases over few items, whose Gram tiles are long, it costs less.
@pytest.mark.parametrize("databases,n,items,mean,row_pairs", [(100, 3000, 60, 6, False), (120, 150_000, 40, 3, True)])
def test_pairs_of_batches(databases, n, items, mean, row_pairs):
    from cupami_b200 import _native

    ctx = _native.context(0)
    rng = np.random.default_rng(n)
    w = 1.0 / np.arange(1, items + 1) ** 0.9
    held = rng.random((n, items)) < np.minimum(0.97, w * mean / w.sum())
    offsets = np.zeros(n + 1, dtype=np.uint64)
    np.cumsum(held.sum(axis=1), out=offsets[1:])
    cols = np.nonzero(held)[1].astype(np.uint32)
    dbs = _native.Database.from_ids_batch(ctx, [(offsets, cols)] * databases)
    found = _native.mine_batch(ctx, dbs, [n // 50] * databases)
    assert (found[0].stats["pair_ops"] == 0) == row_pairs
    assert all(np.array_equal(r.items, found[0].items) and np.array_equal(r.supports, found[0].supports) for r in found)
