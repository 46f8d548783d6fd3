"""Sampled rows of a text with more groups than 32-bit keys hold beside the
bytes: 64-bit keys with values in the output sort, after the dictionary sort of
the same call has run such a sort from another source file."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_wide_keys_with_values(storage, orc):
    n, r = 17_500_001, 64
    t = np.random.default_rng(17).integers(0, 200, size=n).astype(np.uint8)
    L, rows = storage.libcubwt_bwt_aux(t, r)
    s = storage.stats()
    assert s["s"] > 1 << 24                  # 25 group bits and 8 byte bits
    want, index = storage.libcubwt_bwt(t)
    assert np.array_equal(L, want) and rows[0] == index
    sa = orc.suffix_array(t + 2)
    inv = np.empty(n, np.int64)
    inv[sa] = np.arange(n)
    assert np.array_equal(rows, inv[::r] + 1)
