"""Infinities and NaNs in a step's input.

The FP64 kernels leave out terms that an absent species makes exact zeros.  A
zero times an infinity or a NaN is none, so a cell with such a value has to be
evaluated in full.  The tangent-linear step evaluates every term of every cell
and writes the step's outputs too: a poisoned state must give the same values
there, infinities and NaNs at the same places."""
from __future__ import annotations

import numpy as np
import pytest

from nicam_kokkos_microphysics_gb300.state import ARG_NAMES, OUTPUT_NAMES, StateSpec, make_state

pytestmark = pytest.mark.gpu

ALL_SWITCHES = dict(roh2014=0, explicit_icegen=0, kk2000=0, qi_sediment=1, kin2kin=1, aerosol_indirect=1)


def differences(field, variant, options, dt):
    """Elements of each output in which the two steps differ, `field` poisoned in 2 % of its elements."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from nicam_kokkos_microphysics_gb300 import NSW6Error, mp_init
    spec = StateSpec(gall=150, kall=42, lall=1, seed=31, variant=variant, dt=dt)
    st = make_state(spec, out_fill=0.0)
    rng = np.random.default_rng(8)
    st["unccn"][...] = rng.uniform(1.0e7, 2.0e9, st["unccn"].shape)
    a = st[field]
    hit = rng.random(a.shape) < 0.02
    a[hit] = rng.choice([np.nan, np.inf, -np.inf], int(hit.sum()))
    drv = mp_init("NSW6", spec.gall, spec.kall, st["_gz"], st["_gzh"], options=options)
    got = []
    for step in (True, False):
        t = {n: torch.from_numpy(st[n].copy()).cuda() for n in ARG_NAMES}
        try:
            if step:
                drv.mp_driver_batched(1, *[t[n] for n in ARG_NAMES], dt=spec.dt, ct=0.0)
            else:
                drv.tlm(1, t, {n: torch.zeros_like(t[n]) for n in ARG_NAMES}, dt=spec.dt)
        except NSW6Error:
            pass   # (a cell may not converge; every output is written all the same)
        got.append({n: t[n].cpu().numpy() for n in OUTPUT_NAMES})
    drv.close()
    bad = {n: int((~((x == y) | (np.isnan(x) & np.isnan(y)))).sum())
           for n in OUTPUT_NAMES for x, y in [(got[0][n], got[1][n])]}
    return {n: b for n, b in bad.items() if b}


# ten seconds: no tracer falls past its own layer, so the cell physics decides what a poisoned cell gives
@pytest.mark.parametrize("options", [None, ALL_SWITCHES], ids=["reference", "switches"])
@pytest.mark.parametrize("variant", ["standard", "cold"])
@pytest.mark.parametrize("field", ["tem", "q", "unccn"])
def test_poisoned_cells(field, variant, options):
    bad = differences(field, variant, options, 10.0)
    assert not bad, bad


# five minutes: departure distances of several layers, so fluxes draw on poisoned levels without the tracer
@pytest.mark.parametrize("field,options", [(f, o) for f in ("tem", "q", "vx", "ix", "unccn") for o in (None, ALL_SWITCHES)] +
                         [("rhogw", ALL_SWITCHES), ("gsgam2h", ALL_SWITCHES)],
                         ids=lambda p: p if isinstance(p, str) else "switches" if p else "reference")
@pytest.mark.parametrize("variant", ["convective", "cold"])
def test_poisoned_levels(field, variant, options):
    bad = differences(field, variant, options, 300.0)
    assert not bad, bad
