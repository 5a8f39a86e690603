"""The FP64 quotients that share a reciprocal are the division's, bit for bit:
tests/numerics/quotient_check.cu holds them to `/` on the device over random
and edge values, and the WCNS states to the formulas with one division each."""
import os
import subprocess

import pytest

from orion_b200 import build

pytestmark = pytest.mark.gpu


def test_quotients_round_as_the_division(tmp_path):
    here = os.path.dirname(os.path.abspath(__file__))
    exe = str(tmp_path / "quotient_check")
    subprocess.run([build._nvcc(), *build.ARCH, "-std=c++17", "-O3", "--fmad=false", "-prec-div=true", "-prec-sqrt=true",
                    "-I", build.INCLUDE, "-I", build.CSRC, os.path.join(here, "numerics", "quotient_check.cu"), "-o", exe],
                   check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
