"""The quotients, reciprocals, roots and conversions of csrc/nsw6_soft.cuh on
the device, whose seeds are the special-function unit's, bit for bit against
the IEEE operations (tests/native/softfp_device.cu, built with nvcc), and the
seeds themselves within the bounds that the routines rely on."""
from __future__ import annotations

import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]
DIV, DIV_RN, RCP, SQRT, D2F, F2D, RCP_SEED, RSQRT_SEED = range(8)


@pytest.fixture(scope="module")
def apply(tmp_path_factory):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from nicam_kokkos_microphysics_gb300 import _native
    so = tmp_path_factory.mktemp("softfp") / "softfp_device.so"
    subprocess.run([_native.nvcc(), *_native.ARCH, *_native.NVCC_FLAGS, "-I", str(_native.CSRC),
                    str(ROOT / "tests" / "native" / "softfp_device.cu"), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    vp = ctypes.c_void_p
    lib.softfp_apply.argtypes = [ctypes.c_int, vp, vp, vp, ctypes.c_longlong]

    def run(op, a, b=None):
        b = a if b is None else b
        assert a.is_contiguous() and b.is_contiguous() and a.numel() == b.numel()
        out = torch.empty_like(a)
        torch.cuda.synchronize()
        assert lib.softfp_apply(op, a.data_ptr(), b.data_ptr(), out.data_ptr(), a.numel()) == 0
        return out
    return run


def wrong(got, want):
    """Elements that are not the same double (any NaN for a NaN)."""
    import torch
    same = (got.view(torch.int64) == want.view(torch.int64)) | (torch.isnan(got) & torch.isnan(want))
    return int((~same).sum())


def numbers(n, seed, spread):
    """Doubles of both signs, mantissas at random and next to 1 and 2, exponents within `spread`."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    r = lambda hi: torch.randint(0, hi, (n,), generator=g, device="cuda", dtype=torch.int64)  # noqa: E731
    kind, m = r(4), r(1 << 52)
    m = torch.where(kind == 0, r(4096), torch.where(kind == 1, (1 << 52) - 1 - r(4096), m))
    bits = m | ((1023 - spread + r(2 * spread)) << 52) | (r(2) << 63)
    return bits.view(torch.float64)


SPECIAL = [0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 1e-310, 2.2250738585072014e-308,
           1.7976931348623157e308, 1.0, -1.0, 2.0, 0.5, 3.0, 1e-300, 1e300, 1.1754943508222875e-38,
           1.17549429e-38, 3.4028235677973366e38, 3.4028234e38, 1e-45, 1e-39, 1.7014118346046923e38,
           4.0, 3.9999999999999996, 1.9999999999999998, 1.0000000000000002, 0.99999999999999989]


def test_quotients(apply):
    import torch
    s = torch.tensor(SPECIAL, dtype=torch.float64, device="cuda")
    a, b = (t.reshape(-1).contiguous() for t in torch.meshgrid(s, s, indexing="ij"))
    assert wrong(apply(DIV, a, b), a / b) == 0
    for seed, spread in ((1, 1), (2, 120), (3, 1020)):
        a, b = numbers(1 << 22, seed, spread), numbers(1 << 22, seed + 10, spread)
        assert wrong(apply(DIV, a, b), a / b) == 0
        assert wrong(apply(RCP, a, b), 1.0 / b) == 0
        # next to exact quotients and to the half-way points between two
        near = ((a * b).view(torch.int64) + torch.arange(a.numel(), device="cuda") % 5 - 2).view(torch.float64)
        assert wrong(apply(DIV, near, b), near / b) == 0
        if spread <= 120:   # (where 1 / b and a (1 / b) are normal its slow form rounds correctly too)
            assert wrong(apply(DIV_RN, a, b), a / b) == 0
            zero = torch.zeros_like(b)
            assert wrong(apply(DIV_RN, -zero, b.abs()), zero) == 0


def test_roots(apply):
    import torch
    s = torch.tensor(SPECIAL, dtype=torch.float64, device="cuda")
    assert wrong(apply(SQRT, s), torch.sqrt(s)) == 0
    for seed, spread in ((1, 2), (2, 120), (3, 500)):
        a = numbers(1 << 22, seed, spread).abs()
        assert wrong(apply(SQRT, a), torch.sqrt(a)) == 0
        # squares, of numbers of 26 bits and of 53, and their neighbours
        for r in (a.float().double(), a):
            x = ((r * r).view(torch.int64) + torch.arange(r.numel(), device="cuda") % 3 - 1).view(torch.float64)
            assert wrong(apply(SQRT, x), torch.sqrt(x)) == 0


def test_conversions(apply):
    import torch
    s = torch.tensor(SPECIAL, dtype=torch.float64, device="cuda")
    for a in (s, numbers(1 << 22, 4, 160), numbers(1 << 22, 5, 1020)):
        # (and the half-way points between two floats)
        tie = ((a.view(torch.int64) & ~0x1FFFFFFF) | 0x10000000).view(torch.float64)
        for x in (a, tie):
            assert wrong(apply(D2F, x), x.float().double()) == 0
            assert wrong(apply(F2D, x), x.float().double()) == 0


def test_seeds(apply):
    """Every reciprocal the divisors ask for within one unit in the last place and below 1, every reciprocal
    root within 2^-22.9."""
    import torch
    top = (torch.arange(1 << 23, device="cuda", dtype=torch.int32) + 0x3F800002).view(torch.float32)
    y, want = apply(RCP_SEED, top.double()), 1.0 / top.double()
    # (floats from 0.5 to 1 are 2^-24 apart, below 0.5 half as far)
    unit = torch.where(want < 0.5, 2.0 ** -25, 2.0 ** -24)
    assert float(((y - want).abs() / unit).max()) <= 1.0
    assert float(y.max()) < 1.0
    f = (torch.arange(1 << 24, device="cuda", dtype=torch.int32) + 0x3F800000).view(torch.float32).double()
    y = apply(RSQRT_SEED, f)
    assert float((y * torch.sqrt(f) - 1.0).abs().max()) <= 2.0 ** -22.9
