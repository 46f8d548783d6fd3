"""Inverse BWT: row counts around powers of two (the ruler hash permutes the
next power of two), output words at every alignment, alphabets of one to 253
symbols, every ruler rate, in-place device calls, and inputs that are no BWT."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bwt(orc, t):
    L = orc.sa_bwt(t)
    return L, orc.primary_index(t)


@pytest.mark.parametrize("n", [1, 2, 3, 4, 6, 7, 8, 14, 15, 16, 17, 126, 127, 128, 4094, 4095, 4096, 4097, 65534, 65535,
                               65536, 262143, 262144])
def test_sizes(storage, orc, n):
    rng = np.random.default_rng(n)
    for alpha in (1, 2, 4, 253):
        t = (rng.integers(0, alpha, size=n) + 2).astype(np.uint8)
        L, p = _bwt(orc, t)
        assert np.array_equal(storage.unbwt(L, p), t), alpha


@pytest.mark.parametrize("rate", [2, 3, 7, 12])
def test_rates(pkg, orc, rate):
    rng = np.random.default_rng(rate)
    t = np.resize(rng.integers(2, 7, size=9001).astype(np.uint8), 1_100_003)
    t[rng.integers(0, len(t), size=500)] = 9
    L, p = _bwt(orc, t)
    with pkg.Storage(0, tuning={"unbwt_rate_log2": rate}) as st:
        assert np.array_equal(st.unbwt(L, p), t)


def test_alignments_and_in_place(storage, orc):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(3)
    for n in (1000, 50_001):
        t = rng.integers(2, 200, size=n).astype(np.uint8)
        L, p = _bwt(orc, t)
        for shift in range(9):
            buf = torch.zeros(n + 32, dtype=torch.uint8, device="cuda")
            src = torch.zeros(n + 32, dtype=torch.uint8, device="cuda")
            src[shift:shift + n] = torch.from_numpy(L).cuda()
            torch.cuda.synchronize()
            storage.unbwt_device(src.data_ptr() + shift, buf.data_ptr() + shift, n, p)
            got = buf.cpu().numpy()
            assert np.array_equal(got[shift:shift + n], t)
            assert not got[:shift].any() and not got[shift + n:].any()
            storage.unbwt_device(src.data_ptr() + shift, src.data_ptr() + shift, n, p)
            assert np.array_equal(src.cpu().numpy()[shift:shift + n], t)


def test_not_a_bwt(storage, pkg):
    rng = np.random.default_rng(4)
    refused = 0
    for n in (10, 300, 70_000):
        L = rng.integers(2, 6, size=n).astype(np.uint8)
        for p in (0, n // 2, n - 1):
            try:
                assert len(storage.unbwt(L, p)) == n          # one cycle by chance
            except pkg.GbwtError as e:
                assert e.code == pkg.BAD_PARAMETER
                refused += 1
    assert refused >= 5
