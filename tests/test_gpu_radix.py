"""Radix sorts at the edges of their forms: a single tile (4096 keys, no counts
and no look-back), several tiles in one wave (look-back), and more than two
tiles per SM (tile histograms); also segments of one and of several tiles in
the batched output sort.  Byte for byte against the suffix-array BWT."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WAVE = 2 * 152 * 4096       # keys in one wave of tiles


@pytest.mark.parametrize("n", [4095, 4096, 4097, 8192, 3 * 4096 - 1, 70_000, WAVE - 5000, WAVE - 4, WAVE + 3,
                               WAVE + 4097])
@pytest.mark.parametrize("alpha", [2, 250])
def test_dictionary_of_one_phrase_per_text(storage, orc, n, alpha):
    # a text without triggers is one phrase: the dictionary sort runs over n + W keys
    rng = np.random.default_rng(n + alpha)
    t = rng.integers(2, 2 + alpha, size=n).astype(np.uint8)
    t[:64] = 2 + np.arange(64) % 2
    got = storage.pfp_bwt(t, 64, 65535)
    assert storage.stats()["dict_bytes"] >= n
    assert np.array_equal(got, orc.sa_bwt(t))


@pytest.mark.parametrize("lens", [[4096], [4095, 1], [4096, 4096, 4097], [30_000, 17, 50_000, 4096],
                                  [900_000, 5, 300_000, 70_000], [3] * 900 + [200_000]])
@pytest.mark.parametrize("knobs", [{"batch_pad_eighths": 64}, {"batch_pad_eighths": 1, "batch_seg_tiles": 2},
                                   {"batch_radix_bits": 9, "batch_seg_tiles": 400}, {"batch_radix_bits": 8}])
def test_segments(pkg, orc, lens, knobs):
    rng = np.random.default_rng(sum(lens))
    texts = [np.resize(rng.integers(2, 6, size=max(1, n // 3)).astype(np.uint8), n) for n in lens]
    with pkg.Storage(0, tuning=knobs) as st:
        for L, t in zip(st.pfp_bwt_batch(texts), texts):
            assert np.array_equal(L, orc.sa_bwt(t)), len(t)


def test_sampled_rows_with_values(storage, orc):
    # values ride through the segmented sort (row samples), one tile and several
    for n in (4000, 4097, 60_001):
        t = np.random.default_rng(n).integers(0, 200, size=n).astype(np.uint8)
        L, rows = storage.libcubwt_bwt_aux(t, 16)
        sa = orc.suffix_array(t + 2)
        inv = np.empty(n, np.int64)
        inv[sa] = np.arange(n)
        assert np.array_equal(rows, inv[np.arange(0, n, 16)] + 1)
