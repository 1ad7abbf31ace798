"""The device arithmetic of csrc/qpc_fixed.cuh by itself (tests/cpp/fixed_check.cu): splitting into limbs (half a unit), the one
rounding back for sums of every size up to 2^61 and, in the wide form, 2^63 (a quarter of the high word's unit cut off
and one rounding), and the Newton reciprocal from 1 to 2^130 (one unit in the last place)."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


def test_fixed_point_arithmetic(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "fixed_check")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "qpc-tdse-cpc_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "fixed_check.cu"), "-o", exe], check=True)
    out = dict(l.split() for l in subprocess.run([exe], check=True, stdout=subprocess.PIPE, text=True, timeout=120).stdout.split("\n") if l)
    assert set(out) == {"quant", "to_double_wide", "to_double", "reciprocal"}
    assert all(float(v) <= 1.0 for v in out.values()), out
