"""Trigger scan: masks of the counting pass against the oracle's positions at
the edges of threads (16 windows), tiles (4096) and CTAs (16384), with texts whose
windows often share the first word's leading bytes but not the rest."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WINDOWS = [(5, 11), (5, 13), (5, 14), (5, 16), (5, 23), (5, 17), (1, 3), (4, 9), (7, 5), (8, 16), (9, 31), (16, 1000),
           (35, 81), (64, 65535)]


@pytest.mark.parametrize("W,P", WINDOWS)
def test_positions(storage, orc, W, P):
    rng = np.random.default_rng(W * 100 + P)
    for n in (15, 16, 17, 4095, 4097, 16383, 16384, 16385, 16384 + W, 3 * 16384 - 1 + W, 50_001):
        t = rng.integers(2, 4, size=n).astype(np.uint8)
        for k in range(0, n, 97):                       # copies of the first word, some cut short
            m = int(rng.integers(1, W + 3))
            t[k:k + m] = t[:min(m, n - k)]
        assert np.array_equal(storage.trigger_scan(t, W, P), orc.trigger_scan(t, W, P)), n


@pytest.mark.parametrize("W,P", [(5, 16), (5, 23), (5, 13), (9, 31), (35, 81), (2, 7)])
def test_batch_edges(storage, orc, W, P):
    # texts that end and start at every offset of a thread's windows, high and low bytes
    rng = np.random.default_rng(W + P)
    texts = []
    for i in range(150):
        n = int(rng.integers(1, 60)) if i % 10 else int(rng.integers(4000, 9000))
        t = rng.choice(np.array([2, 3, 254], np.uint8), size=n)
        texts.append(np.tile(t, 1 + i % 3))
    for L, t in zip(storage.pfp_bwt_batch(texts, W, P), texts):
        assert np.array_equal(L, orc.sa_bwt(t)), len(t)


def test_range_errors_still_found(storage, pkg):
    for n in (40, 16384 + 5):
        for at in (0, 15, 16, n - 1):
            for c, small, code in ((1, False, pkg.BAD_PARAMETER), (255, False, pkg.BAD_PARAMETER),
                                   (16, True, pkg.UNSUPPORTED_INPUT)):
                t = np.full(n, 3, np.uint8)
                t[at] = c
                with pytest.raises(pkg.GbwtError) as e:
                    storage.pfp_bwt(t, 5, 16, small)
                assert e.value.code == code
