"""The link kernels' reciprocal, root and quotient round as the intrinsics do
(B200 only): every significand at exponents up to the +-80 that the kernels keep
to, and 2.6 x 10^9 quotients whose divisors span the date sums that the two-warp
kernel divides by this way (products of two roots of 1e-20 to 1e20)."""

import os
import subprocess

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


def test_correctly_rounded(tmp_path):
    csrc = os.path.join(ROOT, "i.sar.temporal_coherence_b200", "csrc")
    exe = str(tmp_path / "link_float_check")
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                    "--expt-relaxed-constexpr", "-ccbin", "g++", "-I", csrc, "-o", exe,
                    os.path.join(ROOT, "tests", "link_float_check.cu")], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=300).stdout
    assert [int(x) for x in out.split()] == [0, 0, 0]
