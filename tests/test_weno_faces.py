"""The interleaved FP64 WENO faces and the branch-free divisions, compiled for the host and
compared bit for bit with the face template and the compiler's division."""
import os
import re
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "fdd3260_b200", "csrc")


def test_interleaved_faces_are_bit_identical(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "check")
    r = subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-Xcompiler", "-ffp-contract=off", "-I",
                        CSRC, "-o", exe, os.path.join(HERE, "weno_faces_check.cu")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([exe], capture_output=True, text=True, check=True).stdout
    rcp, div = map(int, re.search(r"rcp (\d+) div (\d+)", out).groups())
    bad, lim, nl = map(int, re.search(r"faces (\d+) limited (\d+) nonlinear (\d+)", out).groups())
    assert (rcp, div, bad) == (0, 0, 0), out
    assert lim > 10000 and nl > 100000, out
