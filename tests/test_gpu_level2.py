"""Second-level parse: parses of 4 M phrases and more with few distinct ones.
With W = 1, P = 1 every byte ends a phrase, so short texts reach that size and
the second level's symbols are pairs of bytes.  Byte for byte against the
suffix-array BWT; row 0 (the primary index) through the inverse."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MIN_Z = 1 << 22


def _check(storage, orc, t, W=1, P=1):
    got = storage.pfp_bwt(t, W, P)
    assert np.array_equal(got, orc.sa_bwt(t))
    p = storage.stats()["primary_index"]
    assert np.array_equal(storage.unbwt(got, p), t)


def _copies(seed, base, n, alpha, rate):
    rng = np.random.default_rng(seed)
    t = np.resize(rng.integers(2, 2 + alpha, size=base).astype(np.uint8), n)
    hit = rng.random(n) < rate
    t[hit] = rng.integers(2, 2 + alpha, size=int(hit.sum())).astype(np.uint8)
    return t


@pytest.mark.parametrize("n", [MIN_Z - 1, MIN_Z, MIN_Z + 1, MIN_Z + 31, 5 * MIN_Z // 4 + 5])
@pytest.mark.parametrize("alpha", [3, 40])
def test_mutated_copies(storage, orc, n, alpha):
    _check(storage, orc, _copies(n + alpha, 50_000, n, alpha, 1e-3))


def test_window_parameters(storage, orc):
    t = _copies(9, 300_000, 16_000_000, 4, 1e-4)
    for W, P in ((1, 2), (2, 3), (3, 4)):
        _check(storage, orc, t, W, P)


@pytest.mark.parametrize("kind", ["constant", "period", "runs", "random", "two halves", "copies of copies"])
def test_shapes_that_give_up_or_tie(storage, orc, kind):
    # long runs of one phrase, no repetition, exact copies, nested repetition
    rng = np.random.default_rng(len(kind))
    n = MIN_Z + 12_345
    if kind == "constant":
        t = np.full(n, 7, np.uint8)
    elif kind == "period":
        t = np.resize(np.array([2, 9, 5], np.uint8), n)
    elif kind == "runs":
        t = _copies(3, 70_000, n, 5, 1e-3)
        t[n // 2:n // 2 + 9000] = 4
    elif kind == "random":
        t = rng.integers(2, 250, size=n).astype(np.uint8)
    elif kind == "two halves":
        t = np.tile(rng.integers(2, 12, size=n // 2 + 1).astype(np.uint8), 2)
    else:
        t = np.resize(np.resize(rng.integers(2, 6, size=997).astype(np.uint8), 40_000), n)
        t[rng.integers(0, n, size=300)] = 3
    _check(storage, orc, t)


def test_parse_suffix_array(storage, orc):
    t = _copies(21, 90_000, MIN_Z + 77, 6, 5e-4)
    ranks, sa = storage.parse(t, 1, 1)
    n = len(ranks)
    inv = np.empty(n + 1, np.int64)
    inv[sa] = np.arange(n)
    inv[n] = -1
    a, b = sa[:-1], sa[1:]
    lt = (ranks[a] < ranks[b]) | ((ranks[a] == ranks[b]) & (inv[a + 1] < inv[b + 1]))
    assert np.array_equal(np.sort(sa), np.arange(n)) and bool(lt.all())


@pytest.mark.parametrize("kind", ["even", "uneven", "shared", "tiny among large", "constant"])
def test_batch(storage, orc, kind):
    # W = 1, P = 1: as many phrases as bytes; texts that share content or end inside a repeat
    rng = np.random.default_rng(len(kind))
    if kind == "even":
        texts = [_copies(i, 4000, 150_000, 4, 1e-3) for i in range(30)]
    elif kind == "uneven":
        texts = [_copies(i, 900 + 37 * i, int(n), 5, 1e-3) for i, n in enumerate(rng.integers(1, 900_000, size=14))]
        texts.append(_copies(99, 5000, MIN_Z // 2, 5, 1e-3))
    elif kind == "shared":
        whole = _copies(5, 20_000, 700_000, 4, 1e-3)
        texts = [whole[a:] for a in rng.integers(0, 100_000, size=8)] + [whole[:300_001], whole.copy(), whole.copy()]
    elif kind == "tiny among large":
        texts = [_copies(1, 30_000, MIN_Z + 5, 4, 1e-3)] + [np.full(1 + i % 3, 2 + i % 4, np.uint8) for i in range(50)]
    else:
        texts = [np.full(400_000, 2 + i % 2, np.uint8) for i in range(12)]
    assert sum(len(t) for t in texts) >= MIN_Z
    for L, t in zip(storage.pfp_bwt_batch(texts, 1, 1), texts):
        assert np.array_equal(L, orc.sa_bwt(t)), len(t)


def test_batch_wider_windows(storage, orc):
    texts = [_copies(50 + i, 20_000 + 991 * i, 1_400_000 + 7 * i, 4, 1e-3) for i in range(12)]
    for L, t in zip(storage.pfp_bwt_batch(texts, 2, 3), texts):
        assert np.array_equal(L, orc.sa_bwt(t))
