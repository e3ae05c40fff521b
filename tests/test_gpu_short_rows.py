"""GPU: the kernel functions where short rows change their kernels' form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# Counts: one, two and eight words in flight (rows of up to 32, 64 and more words).  Intersections: a
# warp or 256 threads per row (256 of the widest words: 16, 8 and 4 bytes each), one part or two.
@pytest.mark.parametrize("words", [1, 31, 32, 33, 63, 64, 65, 256, 257, 512, 514, 1024, 1028, 2048, 2049, 4096, 4098])
def test_counts_and_intersections_of_short_rows(words):
    import torch

    from cupami_b200.frequentPattern import _bitsets

    xp = _bitsets.array_module()
    rng = np.random.default_rng(words)
    bits = rng.integers(0, 2**32, (7, words), dtype=np.uint32) & rng.integers(0, 2**32, (7, words), dtype=np.uint32)
    bits[5], bits[6] = 0, 0xFFFFFFFF
    rows = torch.from_numpy(bits.view(np.int32)).cuda()
    for width in (1, 2, 3, 4):
        cand = rng.integers(0, 7, (300, width))
        want = np.bitwise_count(np.bitwise_and.reduce(bits[cand], axis=1)).sum(axis=1, dtype=np.int64).tolist()
        assert _bitsets.count_supports(xp, rows, cand) == want
    for prefix in (0, 5, 6):
        for _ in range(2):  # (supports are written, not added to what was there)
            children, supports = _bitsets.intersect_extensions(xp, rows[prefix], rows)
            want = bits & bits[prefix]
            assert np.array_equal(children.cpu().numpy().view(np.uint32), want)
            assert supports == np.bitwise_count(want).sum(axis=1, dtype=np.int64).tolist()
