"""csrc/nsw6_soft.cuh on the host with seeds that are off by units in the last
place, as the device's special-function unit may have them: quotients and roots
stay correctly rounded (tests/native/softfp_check.cpp)."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.parametrize("ulps", [-2, -1, 1, 2])
def test_quotients_and_roots_with_seeds_off(tmp_path, ulps):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "softfp_check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", f"-DNSW6_SEED_ULPS={ulps}", "-I",
                    str(ROOT / "nicam_kokkos_microphysics_gb300" / "csrc"),
                    str(ROOT / "tests" / "native" / "softfp_check.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    got = dict(re.findall(r"(\w+) ([\d.]+)", out))
    assert all(int(got[n]) == 0 for n in ("div", "rcp", "sqrt")), out
