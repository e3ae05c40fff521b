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


# Baskets of exactly two or three of 13 items, every pair and triple frequent.  No frame survives below
# the pairs of two items.  Of three, each basket is one row of the class of its first item (two
# elements, one of them listed: 12 bytes), and is met once more by its first two items' unit (an
# occurrence and an element: 10 bytes); no basket is left below those.
@pytest.mark.parametrize("size,per_basket", [(2, 0), (3, 22)])
def test_bytes_of_conditional_rows(size, per_basket):
    n, items = 1_900_000, 13
    rng = np.random.default_rng(size)
    held = np.zeros((n, items), bool)
    np.put_along_axis(held, np.argsort(rng.random((n, items)), axis=1)[:, :size], True, axis=1)
    s = _mined(held, 100)
    assert s["n_patterns"] == 13 + 78 + (286 if size == 3 else 0)
    assert s["row_units"] == s["work_items"] and (size == 2 or s["row_units"] > 0)
    assert s["bytes_alg"] == per_basket * n
