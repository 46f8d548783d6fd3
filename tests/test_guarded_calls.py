"""A failed call's given-up wait does not fail the next call: guarded() of the C
ABI, compiled into a program of its own and run on the host."""
import importlib
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_failed_calls_leave_nothing(pkg, tmp_path):
    build = importlib.import_module(pkg.__name__ + ".build")
    exe, lib = str(tmp_path / "guarded_calls"), os.path.dirname(pkg.LIB_PATH)
    r = subprocess.run([build.nvcc(), "-O1", "-std=c++17", *build.ARCH, "-I", build.CSRC, "-o", exe,
                        os.path.join(HERE, "guarded_calls.cu"), "-L" + lib, "-lgbwt", "-Xlinker", "-rpath=" + lib],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
