"""Which parses are parsed again: level2_taken.cu runs the pipeline's stages up to
the second-level parse and says whether it was taken.  Texts like those whose
results test_gpu_level2.py compares, so that those results are the second level's
(or the plain sort's, where it gives up)."""
import importlib
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
MIN_Z = 1 << 22


@pytest.fixture(scope="module")
def taken(pkg, tmp_path_factory):
    build = importlib.import_module(pkg.__name__ + ".build")
    d, lib = tmp_path_factory.mktemp("level2"), os.path.dirname(pkg.LIB_PATH)
    exe, text = str(d / "level2_taken"), str(d / "text.bin")
    subprocess.run([build.nvcc(), "-O2", "-std=c++17", *build.ARCH, "-I", build.CSRC, "-o", exe,
                    os.path.join(HERE, "level2_taken.cu"), "-L" + lib, "-lgbwt", "-Xlinker", "-rpath=" + lib],
                   check=True, capture_output=True)

    def run(t, W, P):
        t.tofile(text)
        r = subprocess.run([exe, text, str(W), str(P)], capture_output=True, text=True, timeout=120)
        assert r.returncode == 0, r.stdout + r.stderr
        return r.stdout.split()[0] == "1"
    return run


def _copies(seed, base, n, alpha, rate):
    rng = np.random.default_rng(seed)
    t = np.resize(rng.integers(2, 2 + alpha, size=base).astype(np.uint8), n)
    hit = rng.random(n) < rate
    t[hit] = rng.integers(2, 2 + alpha, size=int(hit.sum())).astype(np.uint8)
    return t


@pytest.mark.parametrize("n,want", [(MIN_Z - 1, False), (MIN_Z, True), (MIN_Z + 31, True)])
@pytest.mark.parametrize("alpha", [3, 40])
def test_mutated_copies(taken, n, want, alpha):
    assert taken(_copies(n + alpha, 50_000, n, alpha, 1e-3), 1, 1) == want


@pytest.mark.parametrize("W,P", [(1, 2), (2, 3), (3, 4)])
def test_window_parameters(taken, W, P):
    assert taken(_copies(9, 300_000, 16_000_000, 4, 1e-4), W, P)


@pytest.mark.parametrize("kind", ["constant", "period", "random"])
def test_shapes_that_give_up(taken, kind):
    n = MIN_Z + 12_345
    t = {"constant": lambda: np.full(n, 7, np.uint8),
         "period": lambda: np.resize(np.array([2, 9, 5], np.uint8), n),
         "random": lambda: np.random.default_rng(6).integers(2, 250, size=n).astype(np.uint8)}[kind]()
    assert not taken(t, 1, 1)
