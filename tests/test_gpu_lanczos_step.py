"""The precision of a Lanczos step (tests/lanczos_check.cu, compiled here with
nvcc for sm_103a): row products added up in FP64 whatever the vectors' type, the
start vector and each next one rounded once."""
import os
import subprocess

import pytest

from sparlab_gb300 import build as B

HERE = os.path.dirname(os.path.abspath(__file__))

pytestmark = pytest.mark.gpu


def test_step_precision(tmp_path):
    exe = str(tmp_path / "lanczos_check")
    subprocess.check_call([B.nvcc()] + B.ARCH + ["-O3", "-std=c++17", "--expt-relaxed-constexpr",
                                                  "-I", B.CSRC, "-I", os.path.join(os.path.dirname(HERE), "include"),
                                                  os.path.join(HERE, "lanczos_check.cu"), "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
