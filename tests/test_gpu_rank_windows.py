"""First ranks of a dictionary written window by window (more than 1.5 * 2^24
positions) and at once below that: the line itself, a last window of a few
positions, and a text of little repetition over three windows.  The BWT must be
invertible to the text and equal the one that a split into other phrases gives."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LINE = 3 << 23                  # dictionary positions above which windows are used


@pytest.mark.parametrize("n,W", [(LINE - 8 - 40, 8), (LINE - 8 + 40, 8), ((1 << 25) + 5 - 8, 8)])
def test_dictionary_of_one_phrase(storage, n, W):
    # a text without triggers is one phrase: the dictionary has n + W positions
    rng = np.random.default_rng(n)
    t = rng.integers(2, 250, size=n).astype(np.uint8)
    got = storage.pfp_bwt(t, W, 65535)
    st = storage.stats()
    assert st["dict_bytes"] >= n
    assert np.array_equal(storage.unbwt(got, st["primary_index"]), t)


def test_little_repetition(storage):
    t = np.random.default_rng(3).integers(2, 6, size=(1 << 25) + 4321).astype(np.uint8)
    a = storage.pfp_bwt(t, 5, 16)
    assert storage.stats()["dict_bytes"] > LINE
    p = storage.stats()["primary_index"]
    b = storage.pfp_bwt(t, 35, 81)
    assert np.array_equal(a, b) and storage.stats()["primary_index"] == p
    assert np.array_equal(storage.unbwt(a, p), t)
