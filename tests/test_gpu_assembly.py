"""BWT assembly at the edges of its passes: run blocks of every piece width
around 16-byte boundaries and around the length that a whole CTA fills, blocks
that mix bytes differing in one bit, dictionary sizes around the 32-position
words of the bit vectors; byte for byte against the suffix-array BWT."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies", [2, 3, 7, 15, 16, 17, 31, 33, 100, 511, 512, 513, 700])
@pytest.mark.parametrize("base", [31, 33, 64, 97, 250])
def test_run_block_lengths(storage, orc, copies, base):
    rng = np.random.default_rng(copies * 1000 + base)
    t = np.tile(rng.integers(2, 255, size=base).astype(np.uint8), copies)
    t = np.concatenate([t, rng.integers(2, 6, size=copies % 5).astype(np.uint8)])
    assert np.array_equal(storage.pfp_bwt(t), orc.sa_bwt(t))


@pytest.mark.parametrize("a,b", [(2, 3), (2, 130), (127, 128), (253, 254), (254, 2), (85, 170)])
def test_mixed_blocks_of_two_bytes(storage, orc, a, b):
    # the same 40-byte string after either byte: its blocks mix exactly a and b
    rng = np.random.default_rng(a * 256 + b)
    s = rng.integers(2, 255, size=40).astype(np.uint8)
    t = np.concatenate([np.concatenate([[a if rng.random() < 0.5 else b], s]) for _ in range(57)]).astype(np.uint8)
    for W, P in ((5, 16), (3, 7)):
        got = storage.pfp_bwt(t, W, P)
        assert np.array_equal(got, orc.sa_bwt(t))
        want = orc.pfp_bwt(t, W, P, False)[1]
        st = storage.stats()
        assert (st["s"], st["mixed_blocks"], st["mixed_elems"]) == (want["s"], want["mixed_blocks"], want["mixed_elems"])


@pytest.mark.parametrize("n", list(range(20, 60)))
def test_dictionary_sizes_around_words(storage, orc, n):
    t = np.random.default_rng(n).integers(2, 5, size=n).astype(np.uint8)
    assert np.array_equal(storage.pfp_bwt(t), orc.sa_bwt(t))
