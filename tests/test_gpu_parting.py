"""Batches kept apart by text and batches that share their dictionary: byte for
byte against the suffix-array BWT of every text, on both sides of the choice;
phrase tables that run over on the way."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dna(seed, n, copies, rate=1e-3):
    rng = np.random.default_rng(seed)
    t = np.resize(rng.integers(2, 6, size=max(1, n // copies)).astype(np.uint8), n)
    hit = rng.random(n) < rate
    t[hit] = rng.integers(2, 6, size=int(hit.sum())).astype(np.uint8)
    return t


def _check(st, orc, texts, W=5, P=16):
    got = st.pfp_bwt_batch(texts, W, P)
    for i, (L, t) in enumerate(zip(got, texts)):
        assert np.array_equal(L, orc.sa_bwt(t) if len(t) else t), (i, len(t))


def _batch(kind):
    rng = np.random.default_rng(len(kind))
    if kind == "own bases":
        return [_dna(i, int(n), 12) for i, n in enumerate(rng.integers(1, 60_000, size=40))]
    if kind == "one document":
        base = _dna(7, 50_000, 1)
        return [np.where(rng.random(50_000) < 1e-3, 3, base).astype(np.uint8) for _ in range(30)]
    if kind == "identical":
        return [_dna(1, 9000, 3)] * 20
    if kind == "short":
        return [rng.integers(2, 5, size=n).astype(np.uint8) for n in range(0, 40)] * 3
    if kind == "half shared":
        a = [_dna(i, 20_000, 5) for i in range(10)]
        return a + [t[: len(t) // 3] for t in a[:4]]
    # text ends that are triggers, prefixes and suffixes of other texts
    t = _dna(3, 30_000, 8)
    return [t[: int(k)] for k in rng.integers(1, 300, size=60)] + [t[int(k):] for k in rng.integers(29_000, 30_000, size=30)]


KINDS = ["own bases", "one document", "identical", "short", "half shared", "prefixes and suffixes"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("W,P", [(5, 16), (5, 23), (35, 81), (1, 1), (3, 2)])
def test_both_paths(storage, orc, kind, W, P):
    _check(storage, orc, _batch(kind), W, P)


def test_the_choice_follows_the_content(storage):
    # equal phrases of different texts stay distinct only where that costs little
    texts = _batch("own bases")
    storage.pfp_bwt_batch(texts)
    apart = storage.stats()["d"]
    total = 0
    for t in texts:
        if len(t):
            storage.pfp_bwt(t)
            total += storage.stats()["d"]
    assert apart == total
    storage.pfp_bwt_batch(_batch("identical"))
    assert storage.stats()["d"] * 10 < 20 * apart


@pytest.mark.parametrize("kind", ["own bases", "one document"])
def test_small_phrase_table(pkg, orc, kind):
    rng = np.random.default_rng(5)
    extra = [rng.integers(2, 250, size=1_500_000).astype(np.uint8)]      # more phrases than 2^16 slots hold
    with pkg.Storage(0, tuning={"hash_log2_max": 16}) as st:
        _check(st, orc, _batch(kind) + extra)
        assert st.stats()["hash_retries"] >= 1
        assert np.array_equal(st.pfp_bwt(extra[0]), orc.sa_bwt(extra[0]))
