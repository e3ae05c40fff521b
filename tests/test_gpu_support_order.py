"""GPU: searches in order of support (conditional rows, and patterns ordered on the device)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _csr(held):
    from cupami_b200 import TransactionCSR

    offsets = np.zeros(held.shape[0] + 1, dtype=np.uint64)
    np.cumsum(held.sum(axis=1), out=offsets[1:])
    return TransactionCSR(offsets, np.nonzero(held)[1].astype(np.uint32), held.shape[1])


def _sparse(seed, n, items, mean, s=0.9, block=0):
    """Zipf baskets with a few empty rows and one item in nearly every basket; with ``block``,
    that many more items held together by 40 baskets."""
    rng = np.random.default_rng(seed)
    w = 1.0 / np.arange(1, items + 1) ** s
    held = rng.random((n, items + block)) < np.append(np.minimum(0.97, w * mean / w.sum()), np.zeros(block))
    held[rng.random(n) < 0.02] = False
    held[rng.choice(n, 40, replace=False), items:] = True
    return _csr(held)


def _mined(csr, minsup, **attrs):
    from cupami_b200 import cuEclat

    m = cuEclat(csr, minsup)
    for name, value in attrs.items():
        setattr(m, name, value)
    m.mine()
    return m


def _oracle(oracle_lib, csr, minsup):
    return oracle_lib.to_dict(*oracle_lib.mine_csr(csr.offsets, csr.items, minsup))


# Transactions around groups of 128 and chunks of 1,024 and 8,192 occurrences; rows of
# one, two, four and eight lanes (8 elements each); results around the one-CTA ordering's
# 16,384; a chain of 12 levels.
@pytest.mark.parametrize("n,items,mean,minsup,block", [
    (4097, 700, 6, 12, 0), (8191, 300, 15, 60, 0), (16385, 400, 30, 480, 0), (70001, 600, 60, 7000, 0),
    (20000, 2500, 12, 30, 0), (131073, 90, 4, 150, 0), (2048, 500, 50, 150, 0), (20001, 800, 8, 40, 12)])
def test_support_order_matches_the_oracle(oracle_lib, n, items, mean, minsup, block):
    csr = _sparse(n, n, items, mean, block=block)
    want = list(_oracle(oracle_lib, csr, minsup).items())
    assert list(_mined(csr, minsup).getPatterns().items()) == want
    # the tidset walk in column order, ordered on the host
    assert list(_mined(csr, minsup, _DEEP_PROJECT=1).getPatterns().items()) == want


def test_support_order_in_batches_and_every_order(oracle_lib):
    """Databases of different shapes, an empty one among them, in one pass; the C ABI's other
    orders from results ordered on the device."""
    from cupami_b200 import _native, cuEclat

    csrs = [_sparse(7, 30_000, 500, 12), _sparse(8, 900, 60, 5), _csr(np.zeros((3, 5), bool)), _sparse(9, 50_000, 200, 20)]
    for csr, m in zip(csrs, cuEclat.mineBatch(csrs, 0.004)):
        assert list(m.getPatterns().items()) == list(_oracle(oracle_lib, csr, 0.004).items())
    db = _native.Database.from_ids(_native.context(0), csrs[0].offsets, csrs[0].items)
    found = {order: db.mine(120, _native.CPM_ECLAT, order=order)
             for order in (_native.CPM_ORDER_ECLAT, _native.CPM_ORDER_APRIORI, _native.CPM_ORDER_NONE)}
    sets = {order: {tuple(r.items[r.offsets[k]:r.offsets[k + 1]].tolist()): s for k, s in enumerate(r.supports.tolist())}
            for order, r in found.items()}
    assert len(sets[0]) > 2000 and all(s == sets[0] for s in sets.values())
    listed = list(sets[_native.CPM_ORDER_APRIORI])
    assert listed == sorted(listed, key=lambda p: (len(p), p))


@pytest.mark.parametrize("minsup", [0, 1])
def test_thresholds_that_pass_everything(oracle_lib, minsup):
    """Every itemset counts, the ones no transaction holds too; enough transactions for the support order."""
    rng = np.random.default_rng(3)
    csr = _csr(rng.random((1_900_000, 13)) < rng.uniform(0.01, 0.12, 13))
    assert list(_mined(csr, minsup).getPatterns().items()) == list(_oracle(oracle_lib, csr, minsup).items())


# Frequent items around the Gram's tiles (64, 128, 256); the automatic engine counts these
# pairs row by row, the others multiply tidsets.
@pytest.mark.parametrize("n,items,mean", [(30_000, 63, 7), (30_000, 129, 7), (30_000, 257, 7), (9_000, 1_100, 7),
                                          (9_000, 1_100, 25)])
def test_pairs_counted_by_rows_match_the_grams(n, items, mean):
    csr = _sparse(items, n, items, mean, s=0.3)
    found = [list(_mined(csr, 20, _PAIR_ENGINE=engine).getPatterns().items()) for engine in (0, 1, 2)]
    assert found[0] == found[1] == found[2] and len(found[0]) >= items
