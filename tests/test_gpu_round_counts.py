"""Round counts of the parse suffix array, whether the rounds run in many CTAs,
in one, or begin in many and end in one; through every entry point that ends
after them.  With W = 1, P = 1 a constant text of n bytes parses into n - 1 equal
phrases and a last one: after r doublings the suffixes with 2^r equal phrases
ahead still tie, so it takes ceil(log2(n - 1)) of them after the first ranks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4, 40, 1000, 4096, 4097, 4098, 9000, 70_000])
@pytest.mark.parametrize("call", ["bwt", "parse", "batch"])
def test_constant_text(storage, n, call):
    t = np.full(n, 7, np.uint8)
    if call == "bwt":
        storage.pfp_bwt(t, 1, 1)
    elif call == "parse":
        storage.parse(t, 1, 1)
    else:
        storage.pfp_bwt_batch([t], 1, 1)
    assert storage.stats()["parse_rounds"] == 1 + int(np.ceil(np.log2(n - 1)))


@pytest.mark.parametrize("n", [3000, 200_000])
def test_parse_counts_as_the_whole_call(storage, n):
    rng = np.random.default_rng(n)
    t = np.tile(rng.integers(2, 6, size=n // 8).astype(np.uint8), 8)
    storage.pfp_bwt(t)
    want = storage.stats()
    storage.parse(t)
    got = storage.stats()
    for key in ("z", "d", "dict_bytes", "dict_rounds", "parse_rounds"):
        assert got[key] == want[key], key
    assert want["parse_rounds"] > 1 and want["dict_rounds"] > 1
