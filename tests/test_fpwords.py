"""The comparisons, sign changes and keys that the kernels form from the two
words of a double (csrc/nsw6_fpcmp.cuh): one expression for both targets, so
what the host compiler builds here is what the device runs
(tests/native/fpwords_check.cpp)."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "nicam_kokkos_microphysics_gb300" / "csrc"


def test_word_forms_match_ieee(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "fpwords_check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", str(CSRC), str(ROOT / "tests" / "native" / "fpwords_check.cpp"),
                    "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and "mismatches 0" in out.stdout, out.stdout + out.stderr


def test_one_expression_for_both_targets():
    """Only the accessors of a double's bits differ between the targets."""
    text = (CSRC / "nsw6_fpcmp.cuh").read_text()
    forks = re.findall(r"(\w+)\([^()]*\) \{\n#ifdef __CUDA_ARCH__", text)
    assert set(forks) == {"fp_bits", "fp_from_bits", "fp_hi", "fp_lo", "fp_of_words"}
    assert text.count("__CUDA_ARCH__") == len(forks)
