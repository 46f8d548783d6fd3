"""Inverse BWT of exactly repeated texts: between the copies a walk keeps its
row modulo the number of copies, and no thread may be left with the whole chain
of rulers.  The text comes back, in a small multiple of the time that a text
of mutated copies takes (one thread's chain was a hundred times that)."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 4 << 20


def _inverse(storage, t):
    """Best time of three inversions, in seconds; the text is compared."""
    torch = pytest.importorskip("torch")
    L = storage.pfp_bwt(t)
    p = storage.stats()["primary_index"]
    src, dst = torch.from_numpy(L).cuda(), torch.empty(len(t), dtype=torch.uint8, device="cuda")
    best = 1e9
    for _ in range(4):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        storage.unbwt_device(src.data_ptr(), dst.data_ptr(), len(t), p)
        best = min(best, time.perf_counter() - t0)
    assert np.array_equal(dst.cpu().numpy(), t)
    return best


@pytest.fixture(scope="module")
def mutated(storage):
    rng = np.random.default_rng(1)
    t = np.resize(rng.integers(2, 6, size=N // 16).astype(np.uint8), N)
    t[rng.integers(0, N, size=N // 1000)] = 4
    return _inverse(storage, t)


@pytest.mark.parametrize("copies", [2, 4, 8, 16, 32, 64, 256, 4096])
def test_exact_copies(storage, mutated, copies):
    base = np.random.default_rng(copies).integers(2, 6, size=N // copies).astype(np.uint8)
    assert _inverse(storage, np.tile(base, copies)) < 12 * mutated


@pytest.mark.parametrize("kind", ["constant", "period 2", "period 7", "half zeros", "zeros between"])
def test_long_runs(storage, mutated, kind):
    # LF leads from row to row: rulers of their own inside the runs, or one lane walks for its block
    rng = np.random.default_rng(2)
    if kind == "constant":
        t = np.full(N, 5, np.uint8)
    elif kind.startswith("period"):
        t = np.resize(rng.integers(2, 250, size=int(kind[7:])).astype(np.uint8), N)
    elif kind == "half zeros":
        t = np.concatenate([rng.integers(2, 6, size=N // 2), np.full(N // 2, 9)]).astype(np.uint8)
    else:
        t = np.full(N, 9, np.uint8)
        for a in range(0, N, N // 8):
            t[a:a + 5000] = rng.integers(10, 200, size=5000)
    assert _inverse(storage, t) < 3 * mutated


@pytest.mark.parametrize("n", [4095, 4096, 4097, 8191, 8193, 12_289, 70_000])
@pytest.mark.parametrize("runs", [1, 3])
def test_tiles_of_one_symbol(storage, pkg, orc, n, runs):
    # tiles of one symbol at every place, the row of the whole text among them; both conventions
    t = np.repeat(np.arange(runs).astype(np.uint8) * 7 + 3, -(-n // runs))[:n]
    for u in (t, t[::-1].copy(), np.concatenate([t, t])):
        L = orc.sa_bwt(u)
        assert np.array_equal(storage.unbwt(L, orc.primary_index(u)), u)
        C, i = storage.libcubwt_bwt(u)
        assert np.array_equal(storage.libcubwt_unbwt(C, i), u)
    for p in (0, n // 2, n - 1):                     # rows that no text of these symbols has
        try:
            assert len(storage.unbwt(t, p)) == n
        except pkg.GbwtError as e:
            assert e.code == pkg.BAD_PARAMETER


@pytest.mark.parametrize("run", [511, 512, 1023, 1024, 1025, 1536, 4096, 9000])
@pytest.mark.parametrize("at", [0, 1, 512, 4095, 6001])
def test_parts_of_long_runs(storage, orc, run, at):
    rng = np.random.default_rng(run + at)
    t = rng.integers(2, 6, size=20_000).astype(np.uint8)
    t[at:at + run] = 9
    L = orc.sa_bwt(t)
    assert np.array_equal(storage.unbwt(L, orc.primary_index(t)), t)
    C, i = storage.libcubwt_bwt(t)
    assert np.array_equal(storage.libcubwt_unbwt(C, i), t)
