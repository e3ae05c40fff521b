"""GPU: searches at the edges of the engines' tables and limits, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def limits():
    from cupami_b200 import _native

    ctx = _native.context(0)
    yield ctx.set_limits
    ctx.set_limits()


def _csr(n, items, mean, block=0):
    """Zipf baskets; ``block`` more items held together by 40 baskets."""
    from cupami_b200 import TransactionCSR

    rng = np.random.default_rng(n + items)
    w = 1.0 / np.arange(1, items + 1) ** 0.9
    held = rng.random((n, items + block)) < np.append(np.minimum(0.97, w * mean / w.sum()), np.zeros(block))
    held[rng.choice(n, 40, replace=False), items:] = True
    offsets = np.zeros(n + 1, dtype=np.uint64)
    np.cumsum(held.sum(axis=1), out=offsets[1:])
    return TransactionCSR(offsets, np.nonzero(held)[1].astype(np.uint32), items + block)


class _Mines:
    """Mines of one database through the C ABI, each checked against the oracle."""

    def __init__(self, oracle_lib, csr, minsup):
        from cupami_b200 import _native

        self.minsup, self.csr = minsup, csr
        self.want = list(oracle_lib.to_dict(*oracle_lib.mine_csr(csr.offsets, csr.items, minsup)).items())
        self.db = _native.Database.from_ids(_native.context(0), csr.offsets, csr.items)

    def again(self, **opts):
        from cupami_b200 import _native

        o = _native.Opts()
        _native.library().cpm_default_opts(o)
        for name, value in opts.items():
            setattr(o, name, value)
        r = self.db.mine(self.minsup, _native.CPM_ECLAT, o)
        keys = _native.join_labels(r.offsets, r.items, self.db.labels)
        assert list(zip(keys, r.supports.tolist())) == self.want
        return r.stats


# Steps of less than the fifth that remembered sizes add: one of the budgets is filled to over
# four fifths, and those below overflow (frames of bitsets alone, and frames of rows).
@pytest.mark.parametrize("n,items,mean,minsup,most,least", [(20000, 2500, 12, 30, 8 << 20, 176 << 10),
                                                            (400000, 200, 20, 1600, 1300 << 20, 48 << 20)])
def test_mines_of_one_database_under_shrinking_arenas(oracle_lib, limits, n, items, mean, minsup, most, least):
    mines = _Mines(oracle_lib, _csr(n, items, mean), minsup)
    stats = []
    while most > least:
        limits(arena_bytes=most)
        stats += [mines.again(), mines.again()]
        most = most * 6 // 7
    assert stats[0]["retries"] == 0 and stats[0]["deep_rounds"] == 0
    assert any(s["retries"] for s in stats) and (n < 400000 or any(s["deep_rounds"] for s in stats))


def test_a_search_that_overflows_both_engines_is_mined_again(oracle_lib, limits):
    """Rows, then tidsets, overflow the same arena; the next mines go in rounds from the start."""
    limits(arena_bytes=64 << 20)
    mines = _Mines(oracle_lib, _csr(400001, 200, 20), 1600)
    first, *rest = [mines.again() for _ in range(3)]
    assert first["retries"] >= 1 and all(s["deep_rounds"] > 0 for s in (first, *rest))


def test_a_walk_over_tidsets_does_not_steer_conditional_rows(oracle_lib, limits):
    mines = _Mines(oracle_lib, _csr(131073, 90, 4), 150)
    free = mines.again()
    limits(arena_bytes=4 << 20)
    walk = mines.again(deep_project=1)  # overflows, goes in rounds
    assert walk["deep_rounds"] > 0
    limits()
    assert mines.again()["deep_rounds"] == 0 and free["deep_rounds"] == 0


@pytest.mark.parametrize("units", [1, 40, 100])
def test_levels_outgrow_their_tables(oracle_lib, limits, units):
    mines = _Mines(oracle_lib, _csr(400002, 200, 20), 1600)
    free = mines.again()
    limits(level_units=units)
    stats = [mines.again(), mines.again()]
    assert free["row_units"] > 0 and free["retries"] == 0
    assert all(s["retries"] > 0 and s["row_units"] == free["row_units"] for s in stats)


# No room for the conditional rows (their occurrences take 25 MB); the tables of a search with
# them (frames: 9.0 MB); the counters of their levels (2 GB).  Each time there is for the walk.
@pytest.mark.parametrize("shape,limit", [
    ((800000, 60, 4, 8000), {"arena_bytes": 20 << 20, "alloc_bytes": 20 << 20}),
    ((20000, 2500, 12, 30), {"arena_bytes": 8 << 20, "alloc_bytes": 17 << 19}),
    ((400003, 200, 20, 1600), {"arena_bytes": 1 << 30, "alloc_bytes": 1200 << 20, "level_units": 1 << 20})])
def test_searches_go_on_without_the_memory_they_were_planned_with(oracle_lib, limits, shape, limit):
    n, items, mean, minsup = shape
    mines = _Mines(oracle_lib, _csr(n, items, mean), minsup)
    free = mines.again()
    limits(**limit)
    tight = mines.again()
    limits()
    again = mines.again()
    ran = [(s["pair_ops"], s["row_units"], s["bytes_alg"]) for s in (free, tight, again)]  # differ by engine
    assert ran[0] == ran[2] != ran[1]


def test_blocks_that_fit_only_as_asked_for(oracle_lib, limits):
    """The tidsets' block is allocated in a size rounded up, or, without room for that, its own."""
    from cupami_b200 import _native

    csr = _csr(400004, 200, 3)
    baskets = int(np.count_nonzero(np.diff(csr.offsets.astype(np.int64))))
    bits = 200 * (-(-baskets // 128) * 2) * 8
    limits(alloc_bytes=bits - 1)
    with pytest.raises(_native.NativeError) as e:
        _Mines(oracle_lib, csr, 8000)
    assert e.value.code == _native.CPM_ENOMEM
    limits(alloc_bytes=bits)
    mines = _Mines(oracle_lib, csr, 8000)
    assert mines.db.n_items == 200
    limits()
    mines.again()


# A thousand to half a million patterns, a chain of twelve levels among them, without room on the device
# to order them; every order of the C ABI.
@pytest.mark.parametrize("shape", [(131073, 90, 4, 150, 0), (70001, 600, 60, 7000, 0), (20001, 800, 8, 40, 12)])
def test_patterns_ordered_by_the_host(oracle_lib, limits, shape):
    from cupami_b200 import _native

    n, items, mean, minsup, block = shape
    mines = _Mines(oracle_lib, _csr(n, items, mean, block), minsup)
    orders = (_native.CPM_ORDER_ECLAT, _native.CPM_ORDER_APRIORI, _native.CPM_ORDER_NONE)
    free = [mines.db.mine(minsup, _native.CPM_ECLAT, order=o) for o in orders]
    limits(order_bytes=1)
    mines.again()
    tight = [mines.db.mine(minsup, _native.CPM_ECLAT, order=o) for o in orders]
    for a, b in list(zip(free, tight))[:2]:
        assert all(np.array_equal(getattr(a, x), getattr(b, x)) for x in ("offsets", "items", "supports"))
    sets = [{tuple(r.items[r.offsets[k]:r.offsets[k + 1]].tolist()) for k in range(len(r))} for r in (free[2], tight[2])]
    assert sets[0] == sets[1] and len(sets[1]) == len(tight[2])


def test_batches_ordered_by_the_host(oracle_lib, limits):
    from cupami_b200 import cuEclat

    csrs = [_csr(30000, 500, 12), _csr(900, 60, 5), _csr(50000, 200, 20)]
    limits(order_bytes=1)
    for csr, m in zip(csrs, cuEclat.mineBatch(csrs, 0.004)):
        want = oracle_lib.to_dict(*oracle_lib.mine_csr(csr.offsets, csr.items, 0.004))
        assert list(m.getPatterns().items()) == list(want.items())


# Occurrences of all databases together above the limit (26 MB), each database's below it; small
# ids, and ids that take one database after the other anyhow.
@pytest.mark.parametrize("step", [1, 1 << 19])
def test_batches_whose_occurrences_do_not_fit_at_once(oracle_lib, limits, step):
    from cupami_b200 import TransactionCSR, cuEclat

    csrs = [_csr(n, 200, 12) for n in (120001, 140001, 160001, 120002)]
    csrs = [TransactionCSR(c.offsets, c.items * np.uint32(step), c.universe * step) for c in csrs]
    limits(alloc_bytes=14 << 20, arena_bytes=12 << 20)
    miners = cuEclat.mineBatch(csrs, 0.2)
    for csr, m in zip(csrs, miners):
        want = oracle_lib.to_dict(*oracle_lib.mine_csr(csr.offsets, csr.items, 0.2))
        assert len(want) > 3 and list(m.getPatterns().items()) == list(want.items())


# Thresholds that itemsets of no transaction pass: baskets of one item (frames without a row below
# the classes), two items that occur among fourteen that do not, and a database without transactions.
@pytest.mark.parametrize("minsup", [0, -3])
@pytest.mark.parametrize("kind", ["single", "pair", "none"])
def test_levels_whose_units_have_no_occurrences(kind, minsup):
    from cupami_b200 import _native

    items, n = 16, 0 if kind == "none" else 1_900_000
    rng = np.random.default_rng(items)
    held = np.zeros((n, items), bool)
    if kind == "single":
        held[np.arange(n), rng.integers(0, items, n)] = True
    elif kind == "pair":
        held[:, [4, 9]] = rng.random((n, 2)) < 0.5
        held[~held.any(axis=1), 4] = True
    offsets = np.zeros(n + 1, dtype=np.uint64)
    np.cumsum(held.sum(axis=1), out=offsets[1:])
    db = _native.Database.from_columns(_native.context(0), offsets, np.nonzero(held)[1], items)
    r = db.mine(minsup, _native.CPM_ECLAT)
    got = {tuple(r.items[r.offsets[k]:r.offsets[k + 1]].tolist()): s for k, s in enumerate(r.supports.tolist())}
    assert len(got) == len(r) == 2**items - 1
    if n:  # over conditional rows
        assert r.stats["work_items"] == r.stats["projected_units"] + r.stats["row_units"] > 0
    occur = {(i,): int(held[:, i].sum()) for i in range(items)}
    occur[4, 9] = int((held[:, 4] & held[:, 9]).sum())
    assert all(s == occur.get(p, 0) for p, s in got.items())
