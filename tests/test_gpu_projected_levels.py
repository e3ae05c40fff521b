"""GPU: projected levels around the tidset lengths where their warps change form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mine(csr, minsup, arena):
    from cupami_b200 import _native, cuEclat

    m = cuEclat(csr, minsup)
    m._DEEP_PROJECT = 65408
    m._ARENA_BYTES = arena
    m.mine()
    assert m.getKernelStats()["projected_units"] > 0
    return list(m.getPatterns().items())


def _csr(held):
    from cupami_b200 import TransactionCSR

    offsets = np.zeros(held.shape[0] + 1, dtype=np.uint64)
    np.cumsum(held.sum(axis=1), out=offsets[1:])
    return TransactionCSR(offsets, np.nonzero(held)[1].astype(np.uint32), held.shape[1])


# Items 0 and 1 are in every basket: below them tidsets have one bit per basket.  Tidsets of
# one 16-byte word, groups of 2 to 32 lanes, 4 and 8 words per lane, more than 256 words, the longest;
# with room for chunks and without.
@pytest.mark.parametrize("arena", [8 << 20, 1 << 30])
@pytest.mark.parametrize("baskets", [127, 129, 4096, 4097, 8192, 8193, 16384, 16385, 32768, 32769, 40960, 40961, 65408])
def test_tidset_lengths_match_the_oracle(oracle_lib, baskets, arena):
    rng = np.random.default_rng(baskets)
    held = rng.random((baskets, 13)) < rng.uniform(0.5, 0.95, 13)
    held[:, :2] = True
    csr = _csr(held)
    minsup = baskets // 4
    want = oracle_lib.to_dict(*oracle_lib.mine_csr(csr.offsets, csr.items, minsup))
    assert max(k.count("\t") for k in want) >= 4
    assert _mine(csr, minsup, arena) == list(want.items())


# Frames of more later members than a warp lists at once (128), and enough units that
# warps keep child frames to themselves, with survivors from every member to few.
@pytest.mark.parametrize("baskets,items,hold,minsup", [(500, 150, 0.25, 28), (500, 300, 0.12, 11), (9000, 18, 0.97, 6000),
                                                       (260, 18, 0.96, 150)])
def test_wide_and_deep_searches_match_the_oracle(oracle_lib, baskets, items, hold, minsup):
    rng = np.random.default_rng(items)
    held = rng.random((baskets, items)) < hold
    held[:, 0] = True
    csr = _csr(held)
    want = oracle_lib.to_dict(*oracle_lib.mine_csr(csr.offsets, csr.items, minsup))
    assert max(k.count("\t") for k in want) >= 2
    got = _mine(csr, minsup, 1 << 30)
    assert got == list(want.items())
