"""The FP64 routines that the kernels evaluate on the integer pipe
(csrc/nsw6_soft.cuh), built with the host compiler: quotients, reciprocals,
roots and conversions equal the host's IEEE operations bit for bit (four
million operands, the special values pairwise), and exp, log and pow stay
within the errors their fixed-point widths allow."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_integer_pipe_arithmetic(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "softfp_check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    str(ROOT / "nicam_kokkos_microphysics_gb300" / "csrc"),
                    str(ROOT / "tests" / "native" / "softfp_check.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    got = dict(re.findall(r"(\w+) ([\d.]+)", out))
    assert all(int(got[n]) == 0 for n in ("div", "rcp", "sqrt", "cvt", "edge")), out
    # half a unit for the final rounding, the polynomials' remainder (2^-60.7) and truncations (a dozen units
    # of 2^-63, in log a few of 2^-64 against |log x| >= 2^-7)
    assert all(float(got[n]) < 0.55 for n in ("exp", "log", "pow")), out
