"""The fixed-point exp, log and pow (csrc/nsw6_soft.cuh, built with the host
compiler) where a result's rounding carries into its exponent and at the edges
of their tables' intervals (tests/native/softlog_check.cpp)."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_results_next_to_powers_of_two(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "softlog_check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    str(ROOT / "nicam_kokkos_microphysics_gb300" / "csrc"),
                    str(ROOT / "tests" / "native" / "softlog_check.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    got = {k: float(v) for k, v in re.findall(r"(\w+) ([\d.]+)", out)}
    # half a unit for the final rounding, the polynomials' remainder (2^-60.7) and truncations (a dozen units of
    # 2^-63, in log a few of 2^-64 against |log x| >= 2^-7): the bound of the random arguments' test
    assert set(got) == {"log", "exp", "pow"} and all(e < 0.55 for e in got.values()), out


@pytest.mark.gpu
def test_device_logarithms_next_to_powers_of_two():
    """The same logarithms on the device, against the host's (within one unit each)."""
    import numpy as np
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from nicam_kokkos_microphysics_gb300 import mp_init
    from nicam_kokkos_microphysics_gb300.state import vertical_grid
    at = np.exp(np.array([s * 2.0 ** e for s in (-1.0, 1.0) for e in range(-6, 10)]))
    x = (at.view(np.int64)[:, None] + np.arange(-600, 601)).reshape(-1).view(np.float64)
    drv = mp_init("NSW6", 8, 12, *vertical_grid(12))
    got = drv.eval_math(1, torch.from_numpy(x).cuda()).cpu().numpy()
    drv.close()
    want = np.log(x)
    assert np.all(np.abs(got - want) <= 2.0 * np.spacing(np.abs(want)))
