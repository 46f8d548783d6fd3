"""Radix scatters check their places.  radix_places.cu runs both scatter
kernels, every digit width and ranking that the library uses, over several
tiles with right counts (stable order, no error bit) and with counts that point
past the keys (error bit, nothing stored there).  And the batched output sort
with every digit width and ranking, on texts that share their content (texts
with content of their own take another path), against the suffix-array BWT."""
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


def test_places_are_checked(pkg, tmp_path):
    import importlib
    build = importlib.import_module(pkg.__name__ + ".build")
    exe = str(tmp_path / "radix_places")
    subprocess.run([build.nvcc(), "-O3", "-std=c++17", *build.ARCH, "-I", build.CSRC, "-o", exe,
                    os.path.join(HERE, "radix_places.cu")], check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("bits", [8, 9])
@pytest.mark.parametrize("ballot", [1, 2, 3])
@pytest.mark.parametrize("n,k", [(2000, 3), (4097, 2), (30_000, 9)])
def test_shared_batches(pkg, orc, bits, ballot, n, k):
    t = np.random.default_rng(n).integers(2, 250, size=n).astype(np.uint8)
    texts = [t[i:] for i in range(k)]
    with pkg.Storage(0, tuning={"batch_radix_bits": bits, "batch_ballot": ballot, "batch_seg_tiles": 400}) as st:
        for L, q in zip(st.pfp_bwt_batch(texts), texts):
            assert np.array_equal(L, orc.sa_bwt(q)), len(q)
