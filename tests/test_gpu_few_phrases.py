"""Dictionaries around the size up to which occurrences are counted in shared
memory (2048 phrases of 256 occurrences each on average), of one text and of a
batch, against the suffix-array BWT."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("alpha", [2, 16, 44, 45, 46])
@pytest.mark.parametrize("n", [511, 100_003, 530_000])
def test_pairs_of_bytes(storage, orc, alpha, n):
    # W = 1, P = 1: a phrase is a pair of bytes, alpha^2 + 1 of them (44^2 + 1 < 2048 <= 46^2 + 1)
    t = np.random.default_rng(alpha).integers(2, 2 + alpha, size=n).astype(np.uint8)
    assert np.array_equal(storage.pfp_bwt(t, 1, 1), orc.sa_bwt(t))
    assert storage.stats()["d"] <= alpha * alpha + 1


@pytest.mark.parametrize("alpha", [2, 45])
def test_batch(storage, orc, alpha):
    rng = np.random.default_rng(alpha)
    texts = [rng.integers(2, 2 + alpha, size=k).astype(np.uint8) for k in (60_000, 1, 33, 200_000, 5, 90_001)]
    for L, t in zip(storage.pfp_bwt_batch(texts, 1, 1), texts):
        assert np.array_equal(L, orc.sa_bwt(t))
