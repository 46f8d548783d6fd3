"""The number of windows in which a dictionary's first ranks are written, for
dictionaries up to the largest (run on the host)."""
import importlib
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_window_counts(pkg, tmp_path):
    build = importlib.import_module(pkg.__name__ + ".build")
    exe, lib = str(tmp_path / "rank_windows"), os.path.dirname(pkg.LIB_PATH)
    r = subprocess.run([build.nvcc(), "-O1", "-std=c++17", *build.ARCH, "-I", build.CSRC, "-o", exe,
                        os.path.join(HERE, "rank_windows.cu"), "-L" + lib, "-lgbwt", "-Xlinker", "-rpath=" + lib],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
