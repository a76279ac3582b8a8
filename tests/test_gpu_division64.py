"""The FP64 quotients by a common divisor (mk_div64: a product with the reciprocal
and a correction) and the FP64 projector's overlap weights round exactly as '/':
a test program compiled from the library's own headers runs 1e9 of each."""
import os
import subprocess

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


def test_fp64_quotients_are_the_compilers_bit_for_bit(tmp_path):
    exe = tmp_path / "div64_check"
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                    "--expt-relaxed-constexpr", "-I" + os.path.join(ROOT, "mcsart_b200", "csrc"),
                    "-I" + os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "div64_check.cu"), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    assert [int(x) for x in out.stdout.split()] == [0, 0]
