"""The FP64 reciprocal and reciprocal square root of the pair terms (csrc/series.cuh) alone."""
import os
import subprocess

import pytest

from cutc_gb300 import build as b

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


def test_series_against_cuda(tmp_path):
    exe = tmp_path / "series_check"
    subprocess.check_call([os.path.join(b.cuda_home(), "bin", "nvcc"), *b.ARCH, "-O2", "-std=c++17",
                           "-I", b.CSRC, os.path.join(HERE, "c_abi", "series_check.cu"),
                           "-o", str(exe)])
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    print(r.stdout)
    assert r.returncode == 0 and r.stdout.split()[-1] == "ok", r.stdout + r.stderr
