"""GPU: Apriori levels around the sizes where their kernels change."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# Left rows of 15 to 18, of about 130 and of over 250 partners (shares of 16 candidates, eight
# at most), and levels of under and over 4,096 candidates (one CTA, or a scan over the grid).
@pytest.mark.parametrize("n,items,hold,minsup", [(3000, 17, 0.3, 200), (3000, 19, 0.3, 200), (2500, 33, 0.2, 40),
                                                 (4000, 132, 0.06, 12), (9000, 260, 0.03, 8)])
def test_apriori_levels_match_the_oracle(oracle_lib, n, items, hold, minsup):
    from cupami_b200 import TransactionCSR, cuApriori

    rng = np.random.default_rng(items)
    held = rng.random((n, items)) < rng.uniform(0.5, 1.5, items) * hold
    held[:, 0] |= rng.random(n) < 0.9  # the first column joins with all others
    offsets = np.zeros(n + 1, dtype=np.uint64)
    np.cumsum(held.sum(axis=1), out=offsets[1:])
    csr = TransactionCSR(offsets, np.nonzero(held)[1].astype(np.uint32), items)
    miner = cuApriori(csr, minsup)
    miner.mine()
    labels, arrays = oracle_lib.mine_csr(csr.offsets, csr.items, minsup, "apriori")
    want = oracle_lib.to_dict(labels, arrays)
    assert any(k.count("\t") >= 2 for k in want)
    assert list(miner.getPatterns().items()) == list(want.items())
