"""Texts of very few phrases: every occurrence counts at the same address.  The
counts come out right around warps of one phrase and of two, and the call takes
a small multiple of the time of a text with as many phrases that differ (one
address for all of them took ten times that)."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _text(kind, n):
    if kind == "constant":
        return np.full(n, 5, np.uint8)
    if kind == "two":
        return np.resize(np.array([2, 3], np.uint8), n)
    if kind == "last differs":
        t = np.full(n, 5, np.uint8)
        t[-1] = 9
        return t
    a, b = np.array([2], np.uint8), np.array([2, 3], np.uint8)
    while len(b) < n:
        a, b = b, np.concatenate([b, a])
    return b[:n].copy()


@pytest.mark.parametrize("n", [31, 32, 33, 63, 64, 65, 255, 257, 9000, 140_003])
@pytest.mark.parametrize("kind", ["constant", "two", "last differs", "fibonacci"])
def test_counts(storage, orc, n, kind):
    t = _text(kind, n)
    for W, P in ((1, 1), (5, 16)):
        assert np.array_equal(storage.pfp_bwt(t, W, P), orc.sa_bwt(t)), (W, P)
    texts = [t, t[1:], t[: n // 2 + 1]]
    for L, q in zip(storage.pfp_bwt_batch(texts, 1, 1), texts):
        assert np.array_equal(L, orc.sa_bwt(q))


def test_phrase_stage_time(storage):
    torch = pytest.importorskip("torch")
    n, times = 8 << 20, []
    for t in (np.random.default_rng(1).integers(2, 200, size=n).astype(np.uint8), np.full(n, 5, np.uint8)):
        d = torch.from_numpy(t).cuda()
        o = torch.empty_like(d)
        torch.cuda.synchronize()
        best = 1e9
        for _ in range(4):
            storage.pfp_bwt_device(d.data_ptr(), o.data_ptr(), n, 1, 1, stage_times=True)
            best = min(best, storage.stats()["stage_ms"]["phrases"])
        times.append(best)
    assert times[1] < 3 * times[0], times
