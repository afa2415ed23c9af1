"""The work that performance is measured on: calls of the package's public entry points.

A case is one call of a user's program: the step on one region, on all regions of a rank, several
steps from one captured graph, the step on host arrays, its tangent-linear and adjoint, and the
gradient of a multi-step window.  ``listed`` gives the cases, ``draw`` more of the same ranges,
``prepare`` what a program holds before the call, ``run`` the call, ``work`` the bytes and
operations it cannot do without, and ``exact`` its results from a restatement of the scheme in
plain 64-bit torch.

Before a step call the program's dynamical core has written new prognostic fields into the step's
arguments; ``run`` does the same with copies of the fields the step changes, so that every pass
works on the same weather.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from nicam_kokkos_microphysics_gb300 import mp_init
from nicam_kokkos_microphysics_gb300.state import ARG_NAMES, MP_DRIVER_ARGS, batched_shape, vertical_grid
from nicam_kokkos_microphysics_gb300.window import window_gradient

DT = 60.0
# what the step changes and reads again (copied in before every call)
EVOLVING = ["rhog", "rhogvx", "rhogvy", "rhogvz", "rhogw", "rhoge", "rhogq", "tem", "q"]
# what the step writes (less the arguments it fills with constants: ISO1/ISO2_precip, re_solid, GDCLW, GDCFRC)
OUTPUTS = ["rhog", "rhogvx", "rhogvy", "rhogvz", "rhogw", "rhoge", "rhogq", "rho", "tem", "pre", "q", "qd", "precip",
           "precip_rhoe", "precip_lh_heat", "precip_rhophi", "precip_rhokin", "re_liquid", "re_cld", "rctop", "rwtop",
           "tctop", "GPREC"]
# what a derivative is taken with respect to: the arguments the step reads
READS = ["rhog", "rhogvx", "rhogvy", "rhogvz", "rhogw", "rhoge", "rhogq", "vx", "vy", "vz", "tem", "q",
         "gsgam2", "gsgam2h", "gam2", "gam2h", "z"]
# the outputs a cost function looks at, with the size of their departures
SEEDS = {"rhog": 1.0, "rhoge": 1e-5, "rhogvx": 0.1, "rhogvy": 0.1, "rhogvz": 0.1, "rhogw": 1.0, "rhogq": 1e3,
         "rho": 1.0, "tem": 1e-2, "pre": 1e-5, "q": 1e3, "qd": 1.0, "precip": 1e4}
KIND = {n: k for n, k, _ in MP_DRIVER_ARGS}


def _case(name, call, gall, kall, lall=1, variant="standard", precision="fp64", options="", steps=1):
    return {"name": name, "call": call, "gall": gall, "kall": kall, "lall": lall, "variant": variant,
            "precision": precision, "options": options, "steps": steps}


def listed():
    return [
        # a few columns of a nested or single-column run: launches and the host path count
        _case("columns_48", "step", 48, 42),
        # one region of a glevel-8 icosahedral grid, the reference harness's loop body
        _case("region_fp64", "step", 16900, 42),
        # all regions of a rank in one call: the production step, in FP64 and in mixed precision
        _case("rank_fp64", "batched", 16900, 42, lall=10),
        _case("rank_mixed", "batched", 16900, 42, lall=10, precision="mixed"),
        # convection on an odd-sized limited area with many thin layers
        _case("deep_convective", "batched", 3001, 96, lall=2, variant="convective"),
        # the same kind of column in mixed precision
        _case("convective_mixed", "step", 4225, 78, variant="convective", precision="mixed"),
        # scheme switches that runs use together: falling cloud ice, aerosol indirect effect, KIN2KIN
        _case("switches_cold", "step", 8191, 42, variant="cold",
              options="qi_sediment,aerosol_indirect,kin2kin"),
        # twelve steps of a small domain from one captured graph
        _case("steps_small", "steps", 2500, 42, precision="mixed", steps=12),
        # a host program without device arrays (page-locked memory)
        _case("host_mixed", "host", 16900, 42, lall=3, precision="mixed"),
        # the tangent-linear and adjoint step of a data-assimilation window
        _case("tlm", "tlm", 4096, 42),
        _case("adjoint_fp64", "adjoint", 4096, 42, variant="convective"),
        # a checkpointed window of mixed steps with its gradient
        _case("window_mixed", "window", 16900, 42, precision="mixed", steps=4),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    call = rng.choice(["step", "step", "batched", "batched", "steps", "host", "tlm", "adjoint", "window"])
    variant = rng.choice(["standard", "convective", "cold"])
    precision = rng.choice(["fp64", "mixed"])
    # calls that go on from their own results keep to 42 levels: thinner layers want a shorter step than 60 s there
    kall = rng.choice([42, 42, size(12, 160)]) if call not in ("steps", "host", "window") else 42
    options = rng.choice(["", "", "qi_sediment", "aerosol_indirect,qi_sediment", "kin2kin"]) if call == "step" else ""
    gall = size(20, 20000 * 42 // kall)
    lall, steps = 1, 1
    if call == "batched":
        lall = rng.randint(2, 6)
    if call == "steps":
        gall, steps = size(20, 3000), rng.randint(2, 12)
    if call == "host":
        gall, lall = size(1000, 17000), rng.randint(1, 3)
    if call == "tlm":
        gall, precision = size(20, 5000 * 42 // kall), "fp64"
    if call in ("adjoint", "window"):
        gall, steps = size(20, 8000 * 42 // kall), rng.randint(2, 3) if call == "window" else 1
    c = _case("", call, gall, kall, lall, variant, precision, options, steps)
    del c["name"]
    return c


# ---------------------------------------------------------------------- inputs
GRAV, RDRY, CVDRY, RVAP, CL = 9.79764, 287.04, 717.56, 461.46, 4218.0
PSAT0, LHV0, LHS0, LHF0, TEM00, PSTD = 610.7, 2501000.0, 2834000.0, 333000.0, 273.15, 101325.0
EPS, UNDEF, DENS00, TEM_MIN, RADIUS = 2.220446e-16, -9.9999e30, 1.28, 10.0, 6.37122e6
QV, QC, QR, QI, QS, QG = range(6)


def _factors(gz, gzh):
    """Vertical metrics of the grid: thicknesses, reciprocals and interpolation weights."""
    n = len(gz)
    dgz, dgzh, a, c = np.zeros(n), np.zeros(n), np.zeros(n), np.zeros(n)
    dgz[:-1] = gzh[1:] - gzh[:-1]
    dgz[-1] = dgz[-2]
    dgzh[1:] = gz[1:] - gz[:-1]
    dgzh[0] = dgzh[1]
    a[1:] = (gzh[1:] - gz[:-1]) / (gz[1:] - gz[:-1])
    a[0] = 1.0
    c[1:-1] = (gz[1:-1] - gzh[1:-1]) / (gzh[2:] - gzh[1:-1])
    c[0] = 1.0
    shift = np.zeros(n)
    shift[1:] = gz[:-1]
    return {"gz": gz, "gzh": gzh, "dgz": dgz, "dgzh": dgzh, "rdgz": 1 / dgz, "rdgzh": 1 / dgzh, "afact": a,
            "bfact": 1 - a, "cfact": c, "dfact": 1 - c, "shift": shift}


def _grid(kall, dev):
    f = _factors(*vertical_grid(kall))
    return {n: torch.from_numpy(np.ascontiguousarray(v)).to(dev).view(kall, 1) for n, v in f.items()}


def _weather(case, seed, dev):
    """A seeded state on the device in the all-regions layout: hydrostatic columns with a lapse rate of 6.5 K/km,
    relative humidity 0.6 to 1.05, cloud in 30 % and each precipitating species in 20 % of the cells; the
    convective variant has saturated columns with up to 5 g/kg of rain, the cold one starts at 260 K."""
    G, K, L = case["gall"], case["kall"], case["lall"]
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed) * 7919 + 13)
    f64 = dict(dtype=torch.float64, device=dev)
    uni = lambda *s: torch.rand(*s, generator=gen, **f64)  # noqa: E731
    nor = lambda *s: torch.randn(*s, generator=gen, **f64)  # noqa: E731
    m = _grid(K, dev)
    gz = m["gz"][:, 0].tolist()
    lon, lat = uni(L, G) * (2 * math.pi), torch.asin(2 * uni(L, G) - 1)
    st = {"ix": -lon.sin(), "iy": lon.cos(), "iz": torch.zeros(L, G, **f64),
          "jx": -lat.sin() * lon.cos(), "jy": -lat.sin() * lon.sin(), "jz": lat.cos()}
    shape = (L, K, G)
    z, zh = (m[n].expand(shape).contiguous() for n in ("gz", "gzh"))
    st.update(z=z, zh=zh, gsgam2=(1 + z / RADIUS) ** 2, gsgam2h=(1 + zh / RADIUS) ** 2)
    st.update(gam2=st["gsgam2"].clone(), gam2h=st["gsgam2h"].clone())
    tem = torch.clamp((260.0 if case["variant"] == "cold" else 300.0) - 6.5e-3 * z, min=210.0) + nor(*shape)
    pre = torch.empty_like(tem)
    pre[:, 1] = 1e5 * torch.exp(-GRAV * gz[1] / (RDRY * tem[:, 1]))
    for k in range(2, K - 1):
        pre[:, k] = pre[:, k - 1] * torch.exp(-GRAV * (gz[k] - gz[k - 1]) / (RDRY * 0.5 * (tem[:, k] + tem[:, k - 1])))
    q = torch.zeros(L, 6, K, G, **f64)
    rh = 0.6 + 0.45 * uni(*shape)
    cloud, cld = uni(*shape) < 0.30, 1e-5 * torch.exp(nor(*shape))
    q[:, QC] = cld * (cloud & (tem > 273.0))
    q[:, QI] = cld * (cloud & (tem < 273.0))
    for n in (QR, QS, QG):
        q[:, n] = 1e-6 * torch.exp(nor(*shape)) * (uni(*shape) < 0.20)
    if case["variant"] == "convective":
        low = (z < 1e4) & (uni(L, 1, G) < 0.10)
        rh = torch.where(low, 1.0 + 0.02 * uni(*shape), rh)
        q[:, QC] = torch.where(low & (tem > 273.0), q[:, QC].clamp(min=2e-4), q[:, QC])
        q[:, QR] = torch.where(low, (1e-3 * torch.exp(0.5 + 0.6 * nor(*shape))).clamp(max=5e-3), q[:, QR])
    if case["call"] in ("tlm", "adjoint", "window"):
        # the background of a data assimilation has a little of every species everywhere: without it the scheme
        # has a kink there and no derivative
        for n in range(1, 6):
            q[:, n] = torch.maximum(q[:, n], 1e-9 * torch.exp(nor(*shape)))
    for a in (tem, pre):
        a[:, 0], a[:, -1] = a[:, 1], a[:, -2]
    rho = pre / (RDRY * tem)
    q[:, QV] = rh * PSAT0 * torch.exp(LHV0 / RVAP * (1 / TEM00 - 1 / tem)) / (rho * RVAP * tem)
    q[:, :, 0], q[:, :, -1] = q[:, :, 1].clone(), q[:, :, -2].clone()
    u, v, w = 10 * nor(*shape), 10 * nor(*shape), nor(*shape)
    row = lambda n: st[n].view(L, 1, G)  # noqa: E731
    vel = {"vx": u * row("ix") + v * row("jx"), "vy": u * row("iy") + v * row("jy"), "vz": u * row("iz") + v * row("jz")}
    rhog = rho * st["gsgam2"]
    rhogq = rhog.unsqueeze(1) * q
    q = rhogq / rhog.unsqueeze(1)
    qd = 1 - q[:, 1:].sum(1)
    rhogw = torch.zeros(shape, **f64)
    up = rhog[:, 1:] * m["afact"][1:] / st["gsgam2"][:, 1:] + rhog[:, :-1] * m["bfact"][1:] / st["gsgam2"][:, :-1]
    rhogw[:, 2:-1] = (w[:, 1:] * up * st["gsgam2h"][:, 1:])[:, 1:-1]
    st.update(vel, w=w, rhog=rhog, rhogvx=rhog * vel["vx"], rhogvy=rhog * vel["vy"], rhogvz=rhog * vel["vz"],
              rhogw=rhogw, rhoge=rhog * CVDRY * tem, rhogq=rhogq, q=q, rho=rho, tem=tem,
              pre=rho * tem * (qd * RDRY + q[:, QV] * RVAP), unccn=1e8 * torch.exp(nor(*shape)))
    for n, kind, _ in MP_DRIVER_ARGS:
        if n not in st:
            st[n] = torch.zeros(batched_shape(kind, L, K, G), **f64)
        st[n] = st[n].contiguous()
    return st


def _options(case):
    on = {n: 1 for n in case["options"].split(",") if n}
    return on or None


def _seeds(case, seed, dev):
    """Output adjoints (or input tangents): departures of the size of each field's own."""
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed) * 104729 + 7)
    L, K, G = case["lall"], case["kall"], case["gall"]
    return {n: s * torch.randn(batched_shape(KIND[n], L, K, G), generator=gen, dtype=torch.float64, device=dev)
            for n, s in SEEDS.items()}


def _tangents(st, seed):
    gen = torch.Generator(device=st["rhog"].device)
    gen.manual_seed(int(seed) * 104729 + 7)
    return {n: 1e-3 * st[n] * torch.randn(st[n].shape, generator=gen, dtype=torch.float64, device=st[n].device)
            for n in READS if n not in ("gsgam2", "gsgam2h", "gam2", "gam2h", "z")}


DPARAMS = [1e-5, 1e-9, 1e-1, 1e-3, 1e-2, 1e-13, 1.0]


def prepare(case, seed):
    dev = torch.device("cuda")
    G, K, L = case["gall"], case["kall"], case["lall"]
    gz, gzh = vertical_grid(K)
    st = _weather(case, seed, dev)
    drv = mp_init("NSW6", G, K, gz, gzh, lall_max=L, options=_options(case))
    s = {"case": case, "drv": drv}
    if case["call"] == "host":
        # page-locked numpy arrays, as a host program that uses the library keeps them
        host = {n: torch.empty(st[n].shape, dtype=torch.float64, pin_memory=True) for n in ARG_NAMES}
        for n in ARG_NAMES:
            host[n].copy_(st[n])
        s["host"], s["pinned"] = {n: t.numpy() for n, t in host.items()}, host
    elif case["call"] == "step":
        # one region's arrays in the reference's per-region layout
        s["args"] = {n: (st[n][:, 0] if KIND[n] == "2g" else st[n][0]).contiguous() for n in ARG_NAMES}
    else:
        s["args"] = st
    if case["call"] in ("step", "batched", "steps"):
        s["new"] = {n: s["args"][n].clone() for n in EVOLVING}
    if case["call"] == "tlm":
        s["new"] = {n: st[n].clone() for n in EVOLVING}
        s["dx"] = _tangents(st, seed)
        s["tangent"] = {n: torch.zeros_like(st[n]) for n in ARG_NAMES}
    if case["call"] == "adjoint":
        s["ybar"] = _seeds(case, seed, dev)
        s["bar"] = {n: torch.zeros_like(st[n]) for n in ARG_NAMES}
    if case["call"] not in ("window", "tlm") and case["precision"] == "mixed":
        drv.set_precision("mixed")
    return s


def _renew(s):
    """The dynamical core's new fields."""
    torch._foreach_copy_([s["args"][n] for n in EVOLVING], [s["new"][n] for n in EVOLVING])


def run(s):
    case, drv, L = s["case"], s["drv"], s["case"]["lall"]
    call = case["call"]
    if call == "host":
        drv.run(s["host"], DT)   # in place: the host program goes on with the result
        return {n: s["host"][n] for n in OUTPUTS}
    a = s["args"]
    if call == "step":
        _renew(s)
        drv.mp_driver(0, *[a[n] for n in ARG_NAMES], dt=DT, ct=0.0)
        return {n: a[n] for n in OUTPUTS}
    if call == "batched":
        _renew(s)
        drv.mp_driver_batched(L, *[a[n] for n in ARG_NAMES], dt=DT, ct=0.0)
        return {n: a[n] for n in OUTPUTS}
    if call == "steps":
        _renew(s)
        drv.mp_driver_steps(L, a, case["steps"], DT)
        return {n: a[n] for n in OUTPUTS}
    if call == "tlm":
        _renew(s)
        torch._foreach_zero_(list(s["tangent"].values()))
        torch._foreach_copy_([s["tangent"][n] for n in s["dx"]], list(s["dx"].values()))
        drv.tlm(L, a, s["tangent"], dparams=DPARAMS, dt=DT)
        return {"d_" + n: s["tangent"][n] for n in SEEDS} | {n: a[n] for n in SEEDS}
    if call == "adjoint":
        torch._foreach_zero_(list(s["bar"].values()))
        torch._foreach_copy_([s["bar"][n] for n in s["ybar"]], list(s["ybar"].values()))
        dp = drv.adjoint(L, a, s["bar"], dt=DT)
        return {n: s["bar"][n] for n in READS} | {"params": dp}
    r = window_gradient(drv, L, a, case["steps"], DT, precision=case["precision"])
    return {n: r["grad"][n] for n in READS} | {"params": r["dparams"], "J": np.array([r["J"]])}


def work(case):
    """Bytes: every argument the step reads once and every one it writes once.  Operations: those of the
    scheme as written, counted on the benchmark's weather with one for an addition, a product or a comparison,
    two for a fused one, 15 for a quotient or root, 30, 58 and 174 for exp, log and pow: 5949 for a cell's
    rates and 1003 for its transport and adjustment."""
    cells = case["gall"] * case["kall"] * case["lall"]
    reads, writes = 21, 28   # doubles a cell
    step = {"bytes": 8.0 * (reads + writes) * cells, "flops": 6952.0 * cells}
    # a reverse sweep does about twice the forward's operations besides repeating it, a tangent one as many again
    times = {"tlm": 2.0, "adjoint": 3.0, "window": 4.0 * case["steps"], "steps": 1.0 * case["steps"]}.get(case["call"], 1.0)
    return {n: v * times for n, v in step.items()}


# ---------------------------------------------------------------------- the scheme in 64-bit torch
def _gamma(x):
    """The six-term Lanczos series the scheme defines its gamma constants by."""
    co = [76.18009172947146, -86.50532032941677, 24.01409824083091, -1.231739572450155, 0.1208650973866179e-2,
          -0.5395239384953e-5]
    t = x + 5.5 - (x + 0.5) * math.log(x + 5.5)
    s = 1.000000000190015 + sum(c / (x + 1 + j) for j, c in enumerate(co))
    return math.exp(-t + math.log(2.5066282746310005 * s / x))


def _lo(a, b):
    return torch.where(b < a, b, a)


def _hi(a, b):
    return torch.where(a < b, b, a)


def _pos(a):
    return torch.where(a < 0, torch.zeros_like(a), a)


def _negfilter(rhog, rhogq, gsgam2, tem, qv):
    """Negative precipitating species are filled from the vapour, negative vapour from the dry air; the vapour's
    mixing ratio stays the caller's."""
    rq = [rhogq[0], rhogq[1]] + [_pos(x) for x in rhogq[2:]]
    diff = sum(rhogq[2:]) - sum(rq[2:])
    v = rq[0] + diff
    rq[0] = _pos(v)
    rhog = rhog * (1 - (v - rq[0]))
    q = [qv] + [x / rhog for x in rq[1:]]
    qd = 1 - (q[1] + q[2] + q[3] + q[4] + q[5])
    rho = rhog / gsgam2
    return rhog, rq, q, rho, tem * rhog * CVDRY, rho * (qd * RDRY + qv * RVAP) * tem


def _rates(p, opt, rhog, rho, tem, pre, q, unccn, dt):
    """Process rates of the six-class scheme: changes of rhogq, fall speeds, effective radii."""
    pi, where = math.pi, torch.where
    beta_saut, qicrt, Cr, Cs, Cg, ice_nuc, kk_aut = p
    zero, one = torch.zeros_like(tem), torch.ones_like(tem)
    Ar, As, Ag, N0r, N0g = pi * 1000.0 / 6, 0.069, pi * 400.0 / 6, 8e6, 4e8
    Gm = {x: _gamma(x) for x in (4.0, 5.0, 6.0, 3.5, 6.5, 4.5, 2.75)}
    qv, qc, qr, qi, qs, qg = (_pos(x) for x in q)
    rtem = 1 / _hi(tem, torch.full_like(tem, TEM_MIN))
    Ll, Li = LHV0 / RVAP, LHS0 / RVAP
    qsl = PSAT0 * torch.exp(Ll * (1 / TEM00 - rtem)) / (rho * RVAP * tem)
    qsi = PSAT0 * torch.exp(Li * (1 / TEM00 - rtem)) / (rho * RVAP * tem)
    Sliq, Sice = qv / qsl.clamp(min=EPS), qv / qsi.clamp(min=EPS)
    rd = 1 / rho
    fr = torch.sqrt(DENS00 * rd)
    tc = tem - TEM00
    cold, warm = tc < 0, ~(tc < 0)
    d1, d2, sps = qr >= 1e-4, (qr <= 1e-4) & (qs <= 1e-4), Sice >= 1
    dv, dc, dr, di, ds, dg = (x / dt for x in (qv, qc, qr, qi, qs, qg))

    def root(on, x, power):
        return where(on, where(on, x, one) ** power, zero)

    rain, grau = qr >= 1e-12, qg >= 1e-12
    lr = root(rain, rho * qr / (Ar * N0r * Gm[4.0]), 0.25)
    lr_h = root(rain, rho * qr / (Ar * N0r * Gm[4.0]), 0.125)
    lg = root(grau, rho * qg / (Ag * N0g * Gm[4.0]), 0.25)
    lg_h = root(grau, rho * qg / (Ag * N0g * Gm[4.0]), 0.125)
    # snow moments of Roh and Satoh (2014)
    ca = [5.065339, -0.062659, -3.032362, 0.029469, -0.000285, 0.31255, 0.000204, 0.003199, 0.0, -0.015952]
    cb = [0.476221, -0.015896, 0.165977, 0.007468, -0.000141, 0.060366, 0.000079, 0.000594, 0.0, -0.003577]
    x2 = rho * qs / As
    snow = x2 >= 1e-12
    lx = torch.log(where(snow, x2, one))
    ts = where(tc < -0.1, tc, torch.full_like(tc, -0.1))

    def moment(nm):
        a, b = ((c[0] + ts * (c[1] + ts * (c[4] + ts * c[8]))) + nm * ((c[2] + ts * (c[3] + ts * c[6])) + nm * (
            (c[5] + ts * c[7]) + nm * c[9])) for c in (ca, cb))
        return where(snow, torch.exp(math.log(10.0) * a + lx * b), zero)

    m0, m1, m0b, m1b, m2b, m2d, m5h = (moment(n) for n in (0.0, 1.0, 2.0, 3.0, 4.0, 2.25, 1.625))
    rmom = where(snow, m2d / where(snow, m0b, one), zero)
    vtr = -Cr * fr * (Gm[4.5] / Gm[4.0]) * lr_h
    vts = -Cs * fr * rmom
    vtg = -Cg * fr * (Gm[4.5] / Gm[4.0]) * lg_h
    vti = zero
    if "qi_sediment" in opt:
        on = qi >= 1e-8
        vti = where(on, -3.29 * where(on, rho * qi, one) ** 0.16, zero)
    Nc = torch.full_like(tem, 50.0)
    if "aerosol_indirect" in opt:
        Nc = _hi(unccn * 1e-6, Nc)
    Qi0 = ice_nuc * torch.exp(1.33 * (math.log(1000.0) + _pos(-0.1 * tc))) * rd
    Pigen = _pos(_lo(Qi0 - qi, qv - qsi)) / dt
    e6 = torch.exp(6e-2 * tc)
    Esi, betai = _lo(0.25 * one, 0.25 * e6), _lo(beta_saut * one, beta_saut * e6)
    on = qc * qr >= 1e-12
    Pracw = where(on, 67.0 * where(on, qc * qr, one) ** 1.15, zero)
    q4 = 0.25 * pi
    Psacw = qc * q4 * Cs * m2d * fr
    Pgacw = qc * q4 * N0g * Cg * Gm[3.5] * lg ** 3 * lg_h * fr
    Praci = qi * q4 * N0r * Cr * Gm[3.5] * lr ** 3 * lr_h * fr
    Psaci = qi * q4 * Esi * Cs * m2d * fr
    Piacr = qi * (Ar / 4.19e-13) * q4 * N0r * Cr * Gm[6.5] * lr ** 6 * lr_h * fr
    rel_rs, rel_gr = (vtr - vts).abs(), (vtg - vtr).abs()
    Psacr = Ar * q4 * rd * N0r * rel_rs * (Gm[4.0] * lr ** 4 * x2 + 2 * Gm[5.0] * lr ** 5 * m1 + Gm[6.0] * lr ** 6 * m0)
    Pgacr = Ar * q4 * rd * N0g * N0r * rel_gr * (
        Gm[4.0] * lr ** 4 * 2.0 * lg ** 3 + 2 * Gm[5.0] * lr ** 5 * lg ** 2 + Gm[6.0] * lr ** 6 * lg)
    Pracs = As * q4 * rd * N0r * rel_rs * (m0b * 2.0 * lr ** 3 + 2 * m1b * lr ** 2 + m2b * lr)
    on = qc > 0
    Praut = where(on, kk_aut * where(on, qc, one) ** 2.47 * Nc ** -1.79, zero)
    over = betai * (qi - qicrt)
    Psaut = where(over > 0, over, zero)
    Ka = 2.428e-2 + 7.47e-5 * tc
    Kd = (2.222e-5 + 1.37e-7 * tc) * PSTD / pre
    rNu = rho / (1.718e-5 + 5.28e-8 * tc)
    Glv = 1 / (LHV0 / (Ka * tem) * (LHV0 / (RVAP * tem) - 1) + 1 / (Kd * rho * qsl))
    Giv = 1 / (LHS0 / (Ka * tem) * (LHS0 / (RVAP * tem) - 1) + 1 / (Kd * rho * qsi))
    Gil = Ka * tc / LHF0

    def rooted(on, x):
        return where(on, torch.sqrt(where(on, x, one)), zero)

    ventr = 0.78 * lr ** 2 + 0.27 * Gm[2.75] * rooted(rain, Cr * fr * rNu * lr ** 5 * lr_h)
    Prevp = 2 * pi * rd * N0r * (1 - _lo(Sliq, one)) * Glv * ventr
    ri = _hi(rho * qi, torch.full_like(tem, EPS))
    XNi = _lo(_hi(5.38e7 * ri ** 0.75, 1e3 * one), 1e6 * one)
    Di = _lo(11.9 * torch.sqrt(ri / XNi), 500e-6 * one)

    def split(x):   # deposition where supersaturated, sublimation elsewhere
        return where(sps, x, zero), where(sps, zero, -x)

    Pidep, Pisub = split(4 * Di * XNi * rd * (Sice - 1) * Giv)
    frost = tc + 40.0 < 0
    Pihom = where(frost, dc, zero)
    efrz = torch.exp(-0.66 * tc) - 1
    Pihtr = where(~frost & cold, rho / 1000.0 * qc ** 2 / 300e6 * 100.0 * efrz, zero)
    Pimlt = where(warm, di, zero)
    vents = 0.65 * m1 + 0.39 * torch.sqrt(Cs * fr * rNu) * m5h
    Psdep, Pssub = split(2 * pi * rd * (Sice - 1) * Giv * vents)
    Psmlt = _pos(2 * pi * rd * Gil * vents + CL * tc / LHF0 * (Psacw + Psacr))
    ventg = 0.78 * lg ** 2 + 0.27 * Gm[2.75] * rooted(grau, Cg * fr * rNu * lg ** 5 * lg_h)
    Pgdep, Pgsub = split(2 * pi * rd * N0g * (Sice - 1) * Giv * ventg)
    Pgmlt = _pos(2 * pi * rd * N0g * Gil * ventg + CL * tc / LHF0 * (Pgacw + Pgacr))
    Pgfrz = 2 * pi * rd * N0r * 60.0 * 100.0 * Ar * efrz * lr ** 7

    ice, liq = (lambda x, d: where(cold, _lo(x, d), zero)), (lambda x, d: where(warm, _lo(x, d), zero))
    Pracw = Pracw + where(warm, Psacw, zero) + where(warm, Pgacw, zero)
    Pracs = ice(Pracs, ds)
    Piacr, Psacr, Praci = ice(Piacr, dr), ice(Psacr, dr), ice(Praci, di)
    P = {"igen": ice(Pigen, dv), "idep": ice(Pidep, dv), "sdep": ice(Psdep, dv), "gdep": ice(Pgdep, dv),
         "raut": _lo(Praut, dc), "racw": _lo(Pracw, dc), "ihom": ice(Pihom, dc), "ihtr": ice(Pihtr, dc),
         "sacw": ice(Psacw, dc), "gacw": ice(Pgacw, dc), "revp": _lo(Prevp, dr), "gacr": ice(Pgacr, dr),
         "gfrz": ice(Pgfrz, dr), "isub": ice(Pisub, di), "imlt": liq(Pimlt, di), "saut": ice(Psaut, di),
         "saci": ice(Psaci, di), "ssub": ice(Pssub, ds), "smlt": liq(Psmlt, ds), "gsub": ice(Pgsub, dg),
         "gmlt": liq(Pgmlt, dg), "iacr_s": where(d1, zero, Piacr), "iacr_g": where(d1, Piacr, zero),
         "raci_s": where(d1, zero, Praci), "raci_g": where(d1, Praci, zero), "sacr_s": where(d2, Psacr, zero),
         "sacr_g": where(d2, zero, Psacr), "racs": where(d2, zero, Pracs)}
    # gains and losses of each species; a species' rates are scaled back when they would use up more than there is
    budget = {"c": ("imlt", "raut racw ihom ihtr sacw gacw", dc),
              "i": ("igen idep ihom ihtr", "isub imlt saut raci_s saci raci_g", di),
              "r": ("raut racw smlt gmlt", "revp iacr_s sacr_s iacr_g sacr_g gacr gfrz", dr),
              "v": ("revp isub ssub gsub", "igen idep sdep gdep", dv),
              "s": ("sdep sacw iacr_s sacr_s saut raci_s saci", "ssub smlt racs", ds),
              "g": ("gdep gacw iacr_g sacr_g gacr gfrz raci_g racs", "gsub gmlt", dg)}

    def net(n):
        gain, loss, _ = budget[n]
        t = sum(P[x] for x in gain.split())
        for x in loss.split():
            t = t - P[x]
        return t

    for n, (gain, loss, d) in budget.items():
        t = net(n)
        over = t + EPS < 0
        part = -d / where(over, t, -one)
        fac = where(over & (part < 1), part, one)
        for x in (gain + " " + loss).split():
            P[x] = P[x] * fac
    t = {n: _hi(net(n), -budget[n][2]) for n in "crisg"}
    t["v"] = -(t["c"] + t["r"] + t["i"] + t["s"] + t["g"])
    drq = [rhog * t[n] * dt for n in "vcrisg"]

    dgam = 0.1444 / (0.146 - 5.964e-2 * math.log(50.0 / 2000.0)) ** 2
    cdg = _gamma(dgam + 2 / 3) / _gamma(dgam) * dgam ** (-2 / 3)
    cxf = 0.75 / pi / 1000.0
    r2c = cdg * (cxf * (rho * qc * 1000.0 / Nc * 1e-9) + EPS) ** (2 * 0.33333333) * (Nc * 1e6)
    r2 = r2c + 0.25 * N0r * 2.0 * lr ** 3
    big = r2 >= 1e-10
    re = where(big, (cxf * rho * qc + cxf * rho * qr) / where(big, r2, one), zero)
    bigc = r2c >= 1e-10
    rec = where(bigc, cxf * rho * qc / where(bigc, r2c, one), zero)
    top = ~big & (qc + qr >= 1e-5)
    undef = torch.full_like(tem, UNDEF)
    return drq, {QR: vtr, QI: vti, QS: vts, QG: vtg}, re, rec, where(top, re, undef), where(top, tem, undef)


def _departure(m, dz, zh, wp, first, dt):
    """Departure distances of the falling tracer, the bounds of the layers they reach over the region, and the
    departure cells, for levels first .. K-2 (negative distances: the air parcel comes from above)."""
    L, K, G = wp.shape
    last = K - 2
    mid = 0.5 * (wp[:, :-1] + wp[:, 1:])
    w = torch.cat([wp[:, :first + 1], mid[:, first:last], wp[:, last:last + 1]], 1)   # levels 0 .. last + 1
    wm, w0, wn = w[:, first - 1:last], w[:, first:last + 1], w[:, first + 1:last + 2]
    zm, z0 = dz[first - 1:last], dz[first:last + 1]
    r = (wn - wm) / (zm + z0)
    c = 2 * ((wn - w0) / z0 - (w0 - wm) / zm) / (zm + z0)
    d = dt * w0 - 0.5 * dt ** 2 * w0 * r + dt ** 3 / 6 * w0 * (r * r + w0 * c)
    d0 = dt * w0[:, :1] - 0.5 * dt ** 2 * w0[:, :1] * (wn[:, :1] - w0[:, :1]) / z0[:1]
    pad = torch.zeros(L, K, G, dtype=wp.dtype, device=wp.device)
    dis = torch.cat([pad[:, :first], d0, d[:, 1:], pad[:, last + 1:]], 1)
    with torch.no_grad():
        at_rest = dis.detach()
        k = torch.arange(K, device=wp.device).view(1, K, 1)
        tiny = torch.finfo(torch.float64).tiny
        far, near = at_rest.amax(2, keepdim=True).clamp(min=tiny), at_rest.amin(2, keepdim=True).clamp(max=tiny)
        kk = torch.arange(K - 1, device=wp.device).view(1, 1, K - 1)
        lo, up = zh[:-1, 0].view(1, 1, -1), zh[1:, 0].view(1, 1, -1)

        def reach(dist, ok, on):   # the layer that holds the departure point, if among `ok`
            p = zh.view(1, K, 1) - dist
            hit = (lo <= p) & (up > p) & ok & on
            return torch.where(hit.any(2, keepdim=True), hit.int().argmax(2, keepdim=True), k)

        own = (k >= first) & (k <= last)
        bmin = reach(far, (kk <= k) & (kk >= first), (far > 0) & own)
        bmax = reach(near, (kk >= k) & (kk <= last), (near < 0) & own)
        dep = zh.view(1, K, 1) - at_rest
        cell = torch.zeros(L, K, G, dtype=torch.long, device=wp.device)
        zz = zh[:, 0].contiguous()
        for o in range(int((bmin - k).min()), int((bmax - k).max()) + 1):
            k2 = k + o
            use = (k2 >= bmin) & (k2 <= bmax)
            at = k2.clamp(0, K - 2)
            same = (dep >= zz[at]) == (zz[at + 1] >= dep)
            cell = torch.where(use, torch.maximum(cell, torch.where(same, k2, -k2)), cell)
        cell = torch.where((bmin == k) & (bmax == k), k.expand(L, K, G), cell)
        cell = torch.where(cell == 0, first, torch.where(cell == last + 1, last, cell))
    return dis, bmin, bmax, cell


def _flux(src, dz, dis, bmin, bmax, cell, first):
    """Integrals of the sources [n][L][K][G] over what falls through each face, zero below EPS."""
    n, L, K, G = src.shape
    k = torch.arange(K, device=src.device).view(1, K, 1)
    d = dz[:, 0]
    local = (bmin == k) & (bmax == k)

    def weight(k2):
        t = d[k2]
        return torch.where(k2 > cell, t, torch.where(k2 < cell, -t, torch.zeros_like(t)))

    f = torch.zeros_like(src)
    for o in range(int((bmin - k).min()), int((bmax - k).max()) + 1):
        k2 = k + o
        use = (k2 >= bmin) & (k2 <= bmax) & ~local
        at = k2.clamp(0, K - 1)
        f = f + src[:, :, at[0, :, 0]] * torch.where(use, weight(at), torch.zeros_like(dis))
    rest = torch.where(local, dis, dis - weight(bmax))
    f = f + torch.gather(src, 2, cell.unsqueeze(0).expand(n, L, K, G)) * rest
    inside = (k >= first) & (k <= K - 2)
    return torch.where(inside & (f.abs() >= EPS), f, torch.zeros_like(f))


def _face(x):
    """x of the level above."""
    return torch.cat([x[..., 1:, :], torch.zeros_like(x[..., :1, :])], -2)


def _below(x):
    return torch.cat([torch.zeros_like(x[..., :1, :]), x[..., :-1, :]], -2)


def _exact_step(st, case, p, implicit=False):
    """One step from plain torch in 64 bits: the outputs keyed by the argument names.  ``implicit``: the adjusted
    temperature is the root of the energy equation (for derivatives), not the iteration's last value."""
    L, K, G = case["lall"], case["kall"], case["gall"]
    opt, dt = case["options"].split(",") if case["options"] else [], DT
    dev = st["rhog"].device
    m = _grid(K, dev)
    where = torch.where
    lev = torch.arange(K, device=dev).view(1, K, 1)
    inn, half = (lev >= 1) & (lev <= K - 2), (lev >= 2) & (lev <= K - 2)
    zero = torch.zeros_like(st["tem"])
    keep = lambda a, b: where(inn, a, b)  # noqa: E731
    gsg, gsgh = st["gsgam2"], st["gsgam2h"]
    rq0 = [st["rhogq"][:, n] for n in range(6)]
    q0 = [st["q"][:, n] for n in range(6)]
    # the cells' physics (interior levels)
    rhog, rq, q, rho, rhoge, pre = _negfilter(st["rhog"], rq0, gsg, st["tem"], q0[0])
    drq, vt, re, rec, rctop, tctop = _rates(p, opt, rhog, rho, st["tem"], pre, q, st["unccn"], dt)
    rq = [a + b for a, b in zip(rq, drq)]
    rhoge = rhoge - LHV0 * drq[QV] + LHF0 * (drq[QI] + drq[QS] + drq[QG])
    q = [q0[0]] + [x / rhog for x in rq[1:]]
    tem = keep(rhoge / (rhog * CVDRY), st["tem"])
    rhog, rhoge = keep(rhog, st["rhog"]), keep(rhoge, st["rhoge"])
    rq = [keep(a, b) for a, b in zip(rq, rq0)]
    q = [keep(a, b) for a, b in zip(q, q0)]
    vt = {n: where(inn, v, zero) for n, v in vt.items()}
    out = {"re_liquid": where(inn, re, zero), "re_cld": where(inn, rec, zero),
           "rctop": rctop[:, -2:-1], "tctop": tctop[:, -2:-1]}
    out["rwtop"] = where(out["tctop"] >= TEM00, out["rctop"], torch.full_like(out["rctop"], UNDEF))
    # the transport of the falling species
    rgs, rgsh = where(inn, st["gam2"] / gsg, zero), where(inn, st["gam2h"] / gsgh, zero)
    c2w0, c2w1 = m["afact"] / gsg * gsgh, m["bfact"] * _below(1 / gsg) * gsgh
    w2c0, w2c1 = (where(inn, m[n] * gsg / _face(gsgh).clamp(min=1e-30), zero) for n in ("cfact", "dfact"))
    one = torch.ones_like(zero)

    def kinetic(rhog, mom, rw):
        kh = where(inn, 0.5 * (mom[0] ** 2 + mom[1] ** 2 + mom[2] ** 2) / rhog, zero)
        rh = where(half, c2w0 * rhog + c2w1 * _below(rhog), one)
        return kh, where(half, 0.5 * rw ** 2 / rh, zero)

    mom, rw = [st["rhogvx"], st["rhogvy"], st["rhogvz"]], st["rhogw"]
    kh, kv = kinetic(rhog, mom, rw)
    e, n_ = ([st[c + x].unsqueeze(1) for x in "xyz"] for c in ("i", "j"))
    vi, vj = (sum(st[v] * u for v, u in zip(("vx", "vy", "vz"), b)) for b in (e, n_))
    dq, acc = {}, torch.zeros(5, *zero.shape, dtype=zero.dtype, device=dev)
    dkv, drw = zero, zero
    rain, snow, lheat = 0.0, 0.0, 0.0
    ground = [0.0, 0.0, 0.0]
    falling = (QR, QI, QS, QG) if "qi_sediment" in opt else (QR, QS, QG)
    for t in falling:
        dis, bmin, bmax, cell = _departure(m, m["dgz"], m["gzh"], vt[t], 1, dt)
        b = rq[t] * rgs
        src = torch.stack([b, b * CVDRY * tem, b * GRAV * st["z"], q[t] * rgs * kh, b * vi, b * vj])
        f = _flux(src, m["dgz"], dis, bmin, bmax, cell, 1)
        div = where(inn, -(_face(f) - f) * m["rdgz"], torch.zeros_like(f))
        dq[t], acc = div[0], acc + div[1:]
        vh = torch.cat([torch.zeros_like(vt[t][:, :2]), 0.5 * (vt[t][:, 2:-2] + vt[t][:, 1:-3]),
                        torch.zeros_like(vt[t][:, :2])], 1)
        dish, bminh, _, cellh = _departure(m, m["dgzh"], m["shift"], vh, 2, dt)
        qh = where(half, 0.5 * (q[t] + _below(q[t])) * rgsh, zero)
        # the upper bound is the full levels' one
        fh = _flux(torch.stack([qh * kv, qh * rw]), m["dgzh"], dish, bminh, bmax, cellh, 2)
        d = where(half, -(fh - _below(fh)) * m["rdgzh"], torch.zeros_like(fh))
        dkv, drw = dkv + d[0], drw + d[1]
        if t == QR:
            rain = rain - f[0, :, 1] / dt
            out["GPREC"] = -f[0] / dt
        else:
            snow = snow - f[0, :, 1] / dt
            lheat = lheat + f[0, :, 1] * LHF0 / dt
        ground = [a - f[i + 1, :, 1] / dt for i, a in enumerate(ground)]
    out["precip"] = torch.stack([rain, snow])
    out["precip_lh_heat"] = lheat
    out["precip_rhoe"], out["precip_rhophi"], out["precip_rhokin"] = ground
    rhoge = rhoge + acc[0] + acc[1]
    kh, kv = kh + acc[2], kv + dkv
    mom = [a + acc[3] * x + acc[4] * y for a, x, y in zip(mom, e, n_)]
    rw = rw + drw
    for t in falling:
        rq[t] = rq[t] + dq[t]
        rhog = rhog + dq[t]
        rhoge = rhoge - dq[t] * GRAV * st["z"]
    if "kin2kin" in opt:
        k0 = kh / rhog
        vel = [a / rhog for a in mom]
        k1 = 0.5 * (vel[0] ** 2 + vel[1] ** 2 + vel[2] ** 2)
        on = inn & (k1 > 1e-20)
        r = where(on, torch.sqrt((k0 / where(on, k1, one)).abs()), one)
        mom = [keep(v * r * rhog, a) for v, a in zip(vel, mom)]
        face = (lev >= 1)
        rh = where(face, c2w0 * rhog + c2w1 * _below(rhog), one)
        w = rw / rh
        on = face & (0.5 * w ** 2 > 1e-20)
        r = where(on, torch.sqrt((kv / rh / where(on, 0.5 * w ** 2, one)).abs()), one)
        rw = where(face, w * r * rh, rw)
    else:
        before = kh + (w2c0 * _face(kv) + w2c1 * kv)
        kh2, kv2 = kinetic(rhog, mom, rw)
        rhoge = rhoge + where(inn, before - (kh2 + (w2c0 * _face(kv2) + w2c1 * kv2)), zero)
    # the final state: saturation adjustment at constant energy, then the filter again
    q = [x / rhog for x in rq]
    rho, ein = rhog / gsg, rhoge / rhog
    qd = 1 - (q[1] + q[2] + q[3] + q[4] + q[5])
    out["qd"] = qd
    pre_halo = rho * (ein / CVDRY) * (qd * RDRY + q[0] * RVAP)
    em, qsum = ein + q[0] * LHV0, q[0] + q[1]
    cond = q[2] + q[3] + q[4] + q[5]
    cv1 = (qd + cond) * CVDRY
    tem = (em - qsum * LHV0) / cv1

    def qsat(t, r):
        return PSAT0 * torch.exp(LHV0 / RVAP * (1 / TEM00 - 1 / t.clamp(min=TEM_MIN))) / (r * RVAP * t)

    with torch.no_grad():
        sat = inn & (qsum - qsat(tem, rho) > EPS).detach()
        at = sat.nonzero(as_tuple=True)
        T, r, em_s, qs_s, cd = (x[at].detach() for x in (tem, rho, em, qsum, cond))
        v, live = qs_s.clone(), torch.ones_like(T, dtype=torch.bool)
        for _ in range(100):
            s = qsat(T, r)
            cv = ((1 - cd) + (qs_s - s) + cd) * CVDRY
            d = (T * cv + s * LHV0 - em_s) / (cv + LHV0 / RVAP / T ** 2 * s * LHV0)
            v, T = where(live, s, v), where(live, T - d, T)
            live = live & ~(d.abs() < 1e-8)
            if not bool(live.any()):
                break
    if implicit:
        r, em_s, qs_s = rho[at], em[at], qsum[at]
        for _ in range(2):   # twice: the root to rounding, and its derivative
            T = T.detach()
            s = qsat(T, r)
            F = T * (1 + qs_s - s) * CVDRY + s * LHV0 - em_s
            sT = s * (LHV0 / RVAP / T ** 2 - 1 / T)
            T = T - F / ((1 + qs_s - s) * CVDRY + sT * (LHV0 - T * CVDRY)).detach()
        v = qsat(T, r)
    qv, qc = qsum.index_put(at, v), zero.index_put(at, qs_s - v)
    tem = tem.index_put(at, T)
    rq[QV], rq[QC] = rhog * qv, rhog * qc
    rhoge = rhog * tem * (qd + qc + cond) * CVDRY
    g2, rq2, q2, rho2, e2, _ = _negfilter(rhog, rq, gsg, tem, qv)
    p2 = rho2 * ((1 - (q2[1] + q2[2] + q2[3] + q2[4] + q2[5])) * RDRY + qv * RVAP) * tem
    out.update(rhog=keep(g2, rhog), rhoge=keep(e2, rhoge), rho=keep(rho2, rho), tem=tem, pre=keep(p2, pre_halo),
               rhogvx=mom[0], rhogvy=mom[1], rhogvz=mom[2], rhogw=rw,
               rhogq=torch.stack([keep(a, b) for a, b in zip(rq2, rq)], 1),
               q=torch.stack([keep(a, b) for a, b in zip(q2, [qv, qc] + q[2:])], 1))
    return out


def _params(dev):
    cg = math.sqrt(4 * 400.0 * GRAV / (3 * DENS00 * 0.6))
    return [torch.tensor(v, dtype=torch.float64, device=dev) for v in (5e-3, 0.0, 130.0, 4.84, cg, 4.92e-11, 1350.0)]


def exact(case, seed):
    dev = torch.device("cuda")
    st = _weather(case, seed, dev)
    p = _params(dev)
    if case["call"] in ("step", "batched", "host", "steps"):
        with torch.no_grad():
            for _ in range(case["steps"]):
                out = _exact_step(st, case, p)
                st.update({n: out[n] for n in EVOLVING})
        if case["call"] == "step":
            out = {n: out[n][:, 0] if KIND[n] == "2g" else out[n][0] for n in OUTPUTS}
        return {n: out[n] for n in OUTPUTS}
    if case["call"] == "tlm":
        dx = _tangents(st, seed)
        with torch.autograd.forward_ad.dual_level():
            dual = torch.autograd.forward_ad
            x = st | {n: dual.make_dual(st[n], v) for n, v in dx.items()}
            p = [dual.make_dual(a, torch.full_like(a, d)) for a, d in zip(p, DPARAMS)]
            out = _exact_step(x, case, p, implicit=True)
            got = {n: dual.unpack_dual(out[n]) for n in SEEDS}
            tangents = {"d_" + n: (g.tangent if g.tangent is not None else torch.zeros_like(g.primal)).detach().clone()
                        for n, g in got.items()}
        with torch.no_grad():
            out = _exact_step(st, case, _params(dev))
        return tangents | {n: out[n] for n in SEEDS}
    x = {n: st[n].clone().requires_grad_() for n in READS}
    p = [a.requires_grad_() for a in p]
    J = torch.zeros((), dtype=torch.float64, device=dev)
    if case["call"] == "adjoint":
        out = _exact_step(st | x, case, p, implicit=True)
        for n, y in _seeds(case, seed, dev).items():
            J = J + (out[n] * y).sum()
    else:
        now = st | x
        for _ in range(case["steps"]):
            out = _exact_step(now, case, p, implicit=True)
            J = J + out["precip"].sum() * DT
            now = now | {n: out[n] for n in EVOLVING}
    g = torch.autograd.grad(J, list(x.values()) + p, allow_unused=True)
    got = {n: (torch.zeros_like(a) if d is None else d) for (n, a), d in zip(x.items(), g)}
    got["params"] = np.array([0.0 if d is None else float(d) for d in g[len(x):]])
    return got | ({"J": np.array([float(J)])} if case["call"] == "window" else {})
