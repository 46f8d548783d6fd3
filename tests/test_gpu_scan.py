"""Single-pass scans at their tile edges.  With W = 1, P = 1 every window
triggers, so a text of n bytes has n phrase occurrences and the scans over
occurrences run over exactly n items: one tile or several, full and partly
filled ones, and both sides of the size that switches the tile width."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EDGE = 152 * 8 * 1024      # items in small tiles when every SM has eight


@pytest.mark.parametrize("n", [1, 2, 1023, 1024, 1025, 2048, 32 * 1024 + 1, 33 * 1024 - 1, EDGE - 1, EDGE, EDGE + 1,
                               EDGE + 4096, 4096 * 330 + 7])
def test_occurrence_scans(storage, orc, n):
    rng = np.random.default_rng(n)
    t = rng.integers(2, 9, size=n).astype(np.uint8)
    got = storage.pfp_bwt(t, 1, 1, False)
    assert storage.stats()["z"] == n
    assert np.array_equal(got, orc.sa_bwt(t))
    assert np.array_equal(storage.trigger_scan(t, 1, 1), np.arange(1, n + 1))
