"""The look-back's bounded waits run out: the kernels return, the status says
so, and every later kernel leaves the view's lists empty."""
import os
import subprocess

import pytest

from dmgs_gb300 import build as B

HERE = os.path.dirname(os.path.abspath(__file__))


def _compile(tmp_path):
    exe = str(tmp_path / "waits")
    r = subprocess.run([B._nvcc(), *B.ARCH, "-O2", "-std=c++17", "--expt-relaxed-constexpr", "-DDMGS_LB_POLLS=4096u", "-I", B.INCLUDE,
                        os.path.join(HERE, "lookback", "waits.cu"), "-o", exe, "-Xlinker", "-rpath,/usr/local/cuda/lib64"],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return exe


@pytest.mark.gpu
def test_waits_end_and_are_reported(tmp_path):
    r = subprocess.run([_compile(tmp_path)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    rows = [line.split() for line in r.stdout.splitlines()]
    assert len(rows) == 4
    for which, _, status, _, empty, _, ms in rows:
        assert int(status) == 4 | 8, r.stdout  # an index or wait failure, and which: the wait
        assert int(empty) == 1 and float(ms) < 1000.0, r.stdout
