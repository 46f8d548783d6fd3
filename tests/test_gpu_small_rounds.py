"""Doubling rounds in one CTA: dictionaries and parses around its 4096 elements,
groups of every size in it (all equal, two values, many), texts whose rounds
start in many CTAs and end in one.  Byte for byte against the suffix-array BWT."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 40, 1000, 4094, 4095, 4096, 4097, 5000, 9000])
@pytest.mark.parametrize("kind", ["constant", "period 2", "period 7", "random 2", "random 200", "copies"])
@pytest.mark.parametrize("W,P", [(1, 1), (5, 16), (3, 4)])
def test_sizes(storage, orc, n, kind, W, P):
    rng = np.random.default_rng(n)
    if kind == "constant":
        t = np.full(n, 5, np.uint8)
    elif kind.startswith("period"):
        t = np.resize(rng.integers(2, 9, size=int(kind[7:])).astype(np.uint8), n)
    elif kind.startswith("random"):
        t = rng.integers(2, 2 + int(kind[7:]), size=n).astype(np.uint8)
    else:
        t = np.resize(rng.integers(2, 6, size=max(1, n // 16)).astype(np.uint8), n)
        t[rng.integers(0, n, size=n // 100)] = 7
    assert np.array_equal(storage.pfp_bwt(t, W, P), orc.sa_bwt(t))


@pytest.mark.parametrize("n", [30_000, 200_000])
def test_rounds_that_shrink(storage, orc, n):
    rng = np.random.default_rng(n)
    t = np.concatenate([rng.integers(2, 250, size=n).astype(np.uint8), np.full(3000, 9, np.uint8),
                        np.tile(rng.integers(2, 6, size=700).astype(np.uint8), 5)])
    for W, P in ((1, 1), (5, 16)):
        assert np.array_equal(storage.pfp_bwt(t, W, P), orc.sa_bwt(t))
        assert storage.stats()["dict_rounds"] >= 1 and storage.stats()["parse_rounds"] >= 1


def test_batch_of_short_texts(storage, orc):
    rng = np.random.default_rng(8)
    texts = [np.resize(rng.integers(2, 5, size=1 + i % 9).astype(np.uint8), 1 + (i * 37) % 150) for i in range(60)]
    for L, t in zip(storage.pfp_bwt_batch(texts), texts):
        assert np.array_equal(L, orc.sa_bwt(t))
