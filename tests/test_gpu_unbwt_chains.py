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
