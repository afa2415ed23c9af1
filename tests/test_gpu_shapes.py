"""The launch shapes of the cell and column kernels give the same bits.

A column's result depends on the other columns of its region only through the
extrema of the departure distances, which copies of the same columns leave as
they are.  So a region of n copies equals its first copy run by itself, bit for
bit, whatever tiles and cells a thread the two sizes are launched with: 4, 8
or 16 columns a CTA, one to four cells a thread, cell tiles of one pass or
several.
"""
from __future__ import annotations

import numpy as np
import pytest

from nicam_kokkos_microphysics_gb300.state import ARG_NAMES, MP_DRIVER_ARGS, StateSpec, make_state, region_view

pytestmark = pytest.mark.gpu

ALL_SWITCHES = dict(roh2014=0, explicit_icegen=0, kk2000=0, qi_sediment=1, kin2kin=1, aerosol_indirect=1)


# levels at the edges of the cells a thread has: 16 columns up to 24 levels one, 48 two, 64 three; 8 columns above
# 48 two, above 96 four
@pytest.mark.parametrize("kall", [5, 24, 25, 42, 48, 49, 64, 65, 96, 97, 160])
@pytest.mark.parametrize("precision,options", [("fp64", None), ("mixed", None), ("fp64", ALL_SWITCHES),
                                               ("mixed", ALL_SWITCHES)],
                         ids=["fp64", "mixed", "fp64-switches", "mixed-switches"])
def test_gpu_launch_shapes_give_the_same_bits(kall, precision, options):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from nicam_kokkos_microphysics_gb300 import mp_init
    spec = StateSpec(gall=33, kall=kall, lall=1, seed=100 + kall, variant="convective")
    st = make_state(spec, out_fill=np.nan)
    if options:
        st["unccn"][...] = np.random.default_rng(9).uniform(1.0e7, 2.0e9, st["unccn"].shape)
    base = {n: torch.from_numpy(np.ascontiguousarray(v)).cuda() for n, v in region_view(st, 0).items() if n in ARG_NAMES}
    outs = [n for n, _, intent in MP_DRIVER_ARGS if intent != "in"]
    first = None
    for copies in (1, 59, 161):   # 33, 1947 and 5313 columns: 4, 8 and 16 a CTA where the levels allow
        drv = mp_init("NSW6", spec.gall * copies, kall, st["_gz"], st["_gzh"], options=options)
        drv.set_precision(precision)
        t = {n: v.repeat(*[1] * (v.dim() - 1), copies).contiguous() for n, v in base.items()}
        drv.mp_driver(0, *[t[n] for n in ARG_NAMES], dt=spec.dt, ct=0.0)
        torch.cuda.synchronize()
        drv.close()
        if first is None:
            first = {n: t[n].view(torch.int64).clone() for n in outs}
            continue
        for n in outs:
            got = t[n].view(torch.int64)
            assert torch.equal(got, first[n].repeat(*[1] * (got.dim() - 1), copies)), (n, copies)
