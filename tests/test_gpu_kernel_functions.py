"""GPU: the kernel functions at the edges of their word widths, unrolling and parts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# Rows of an odd, an even and a multiple-of-four number of words (4-, 8- and 16-byte rows),
# around 256 and 2,048 of the widest words, and a prefix that starts off a 16-byte boundary.
@pytest.mark.parametrize("words", [1, 2, 4, 31, 255, 256, 257, 2047, 2048, 2049, 4096, 4098, 8192, 8196, 16391])
@pytest.mark.parametrize("offset", [0, 1])
def test_intersections_and_counts(words, offset):
    import torch

    from cupami_b200.frequentPattern import _bitsets

    xp = _bitsets.array_module()
    rng = np.random.default_rng(words)
    bits = rng.integers(0, 2**32, (9, words), dtype=np.uint32) & rng.integers(0, 2**32, (9, words), dtype=np.uint32)
    bits[3], bits[4] = 0, 0xFFFFFFFF
    store = torch.zeros(bits.size + offset, dtype=torch.int32, device="cuda")
    rows = store[offset:].view(9, words)
    rows.copy_(torch.from_numpy(bits.view(np.int32)))
    children, supports = _bitsets.intersect_extensions(xp, rows[0], rows[1:])
    want = bits[1:] & bits[0]
    assert np.array_equal(children.cpu().numpy().view(np.uint32), want)
    assert supports == np.bitwise_count(want).sum(axis=1, dtype=np.int64).tolist()
    for width in (1, 2, 3, 5):
        cand = rng.integers(0, 9, (70, width))
        want = np.bitwise_count(np.bitwise_and.reduce(bits[cand], axis=1)).sum(axis=1, dtype=np.int64).tolist()
        assert _bitsets.count_supports(xp, rows, cand) == want
