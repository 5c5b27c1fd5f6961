"""Timing cases of SuperLite's per-timestep hot path on one GPU.

Each case is work that a program using the framework has it do, through its
public entry points: the physical opacity build (host arrays, as the Fortran
driver passes them, and device arrays), the differentiable opacity with its
reverse mode, the means / leakage / emission coefficients, the Saha equation
of state, the particle loop, and whole timesteps.  Sizes are those of the
benchmark configurations, the smoke test and the parity tests, with odd ones
between.

Inputs are seeded and synthetic: homologous broken-power-law ejecta (1 Msun),
T ~ U(6000, 14000) K, Dirichlet mass fractions of ten elements, log-uniform
lines, and the Verner, Sutherland and ion tables of the parity fixture.

``exact`` restates each path in 64 bits with plain torch and numpy (its
gradients by torch's own autograd).  The particle loop has no such value: its
outputs are realisations of the seeded random walk.
"""
import functools
import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from superlite_b200 import HotPath
from superlite_b200 import workloads as W
from superlite_b200.api import PACKET_DTYPE
from superlite_b200.differentiable import DifferentiableOpacity
from superlite_b200.timestep import BatchTimestep, DeviceTimestep

DEV = torch.device("cuda", 0)
F64 = torch.float64
ATOMIC = "tests/golden/atomic_data.npz"
L_BOL = 1e42
TAUDDMC, TAULUMP = 5.0, 10.0
ZS = W.ELEMENTS


def listed():
    return [
        # smallest call of the drop-in: a debugging-size grid on host arrays
        # (latency, launches and copies count)
        dict(name="opacity_host_32x100", kind="opacity", host=True, nc=32, ng=100, nline=4000, ngs=1, mix=0.0,
             t_days=10.0),
        # odd sizes with sub-groups and the Planck/Rosseland mix
        # (in_grp_ngs, in_opacmixrossel)
        dict(name="opacity_77x333_sub3", kind="opacity", host=False, nc=77, ng=333, nline=20011, ngs=3, mix=0.3,
             t_days=6.5),
        # the physical-opacity workload of one timestep, device arrays
        dict(name="opacity_256x2000", kind="opacity", host=False, nc=256, ng=2000, nline=500000, ngs=1, mix=0.0,
             t_days=10.0),
        # one spectral-fit iteration on that model: forward and reverse mode
        dict(name="gradient_256x2000", kind="gradient", nc=256, ng=2000, nline=500000, t_days=10.0),
        # the same at scale, the largest opacity build
        dict(name="gradient_4096x10000", kind="gradient", nc=4096, ng=10000, nline=2000000, t_days=10.0),
        # means, leakage and emission coefficients of a batch of models on
        # coarse groups, and of one finely grouped model of odd size
        dict(name="coefficients_batch128x100", kind="coefficients", nmodel=128, nxlo=50, nxhi=400, ng=100, t_days=5.0),
        dict(name="coefficients_1001x4003", kind="coefficients", nmodel=1, nxlo=1001, nxhi=1001, ng=4003, t_days=8.0),
        # the equation of state of a large grid
        dict(name="saha_4096", kind="saha", nc=4096, t_days=10.0, acc=1e-8),
        # one snapshot of the CPU-runnable workload driven with host arrays
        # from sources to luminosities, as the Fortran driver calls the library
        dict(name="dropin_64x100", kind="dropin", nc=64, ng=100, npart=100000, t_days=8.0),
        # the FP64 particle loop on that workload's full particle budget
        dict(name="particles_64x100_fp64", kind="particles", nc=64, ng=100, npart=1000000, t_days=6.0, prec=0),
        # a whole step of uneven models in one mixed-precision launch
        dict(name="batch32_mixed", kind="batch", nmodel=32, nxlo=50, nxhi=400, plo=50000, phi=1000000, ng=100,
             tlo=8.0, thi=30.0, prec=1),
        # a whole FP64 timestep on physical opacities: optically thick, all DDMC
        dict(name="timestep_256x2000_fp64", kind="timestep", nc=256, ng=2000, nline=500000, npart=400000,
             t_days=10.0, prec=0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["opacity", "opacity", "gradient", "coefficients", "saha", "dropin", "particles", "batch",
                       "timestep"])
    t = round(rng.uniform(3.0, 20.0), 3)
    if kind == "opacity":
        ngs = rng.choice([1, 1, 1, 2, 4])
        return dict(kind=kind, host=rng.random() < 0.3, nc=_log(rng, 24, 2500), ng=_log(rng, 60, 4000),
                    nline=_log(rng, 2000, 700000), ngs=ngs, mix=0.0 if ngs == 1 else round(rng.random(), 3), t_days=t)
    if kind == "gradient":
        return dict(kind=kind, nc=_log(rng, 24, 2500), ng=_log(rng, 60, 6000), nline=_log(rng, 5000, 1000000),
                    t_days=t)
    if kind == "coefficients":
        if rng.random() < 0.5:
            lo = rng.randrange(20, 120)
            return dict(kind=kind, nmodel=_log(rng, 2, 128), nxlo=lo, nxhi=lo + rng.randrange(1, 280),
                        ng=_log(rng, 40, 400), t_days=t)
        nx = _log(rng, 32, 4096)
        return dict(kind=kind, nmodel=1, nxlo=nx, nxhi=nx, ng=_log(rng, 60, 5000), t_days=t)
    if kind == "saha":
        return dict(kind=kind, nc=_log(rng, 32, 16384), t_days=t, acc=rng.choice([1e-8, 1e-12]))
    if kind == "dropin":
        return dict(kind=kind, nc=rng.randrange(40, 200), ng=_log(rng, 50, 300), npart=_log(rng, 5000, 200000),
                    t_days=t)
    if kind == "particles":
        return dict(kind=kind, nc=rng.randrange(40, 200), ng=_log(rng, 50, 300), npart=_log(rng, 20000, 1000000),
                    t_days=round(rng.uniform(5.0, 25.0), 3), prec=rng.choice([0, 0, 1]))
    if kind == "batch":
        return dict(kind=kind, nmodel=_log(rng, 2, 40), nxlo=50, nxhi=rng.randrange(100, 401), plo=5000,
                    phi=_log(rng, 20000, 300000), ng=_log(rng, 60, 200), tlo=5.0, thi=30.0, prec=rng.choice([0, 1, 1]))
    return dict(kind=kind, nc=rng.randrange(64, 257), ng=_log(rng, 500, 2200), nline=_log(rng, 50000, 500000),
                npart=_log(rng, 20000, 400000), t_days=round(rng.uniform(8.0, 15.0), 3), prec=rng.choice([0, 1]))


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=1)
def _atomic():
    return W.load_atomic_data(ATOMIC)


def _amass():
    return np.array([W.ELEM_MASS.get(z, 2.0 * z) for z in range(1, W.NELEM + 1)])


def _model(case, seed):
    """Grid and gas of one model (numpy)."""
    rng = np.random.default_rng([seed, 1])
    grid = W.homologous_grid(case["nc"], case["t_days"] * W.PC_DAY)
    rho, _ = W.broken_powerlaw_rho(grid)
    temp = rng.uniform(6000.0, 14000.0, grid.nx)
    X = np.zeros((grid.nx, W.NELEM))
    X[:, [z - 1 for z in ZS]] = rng.dirichlet(np.ones(len(ZS)), grid.nx)
    mass, natom, natomfr = W.composition_state(rho, X, grid.vol)
    return dict(grid=grid, rho=rho, temp=temp, X=X, mass=mass, natom=natom, natomfr=natomfr)


def _lines(case, seed):
    return W.make_lines(case["nline"], np.random.default_rng([seed, 2]))


def _analytic_cap(temp, rho, ng, seed):
    """Grey opacity with a smooth seeded spread over the groups (float32)."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    cap = 1e18 * temp ** -1.5 * rho ** 2
    x = torch.linspace(0.0, 6.0 * math.pi, ng, dtype=F64, device=DEV)
    amp, ph = torch.rand(len(cap), 1, generator=g, dtype=F64, device=DEV), torch.rand(
        len(cap), 1, generator=g, dtype=F64, device=DEV)
    return (cap[:, None] * torch.exp(1.5 * amp * torch.sin(x[None, :] + 6.3 * ph))).to(torch.float32)


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a, dtype=np.float64), device=DEV)


def _batch(case, seed):
    """Models whose sizes belong to the case; their gas and snapshot times to the seed."""
    size = np.random.default_rng([case["nmodel"], case["nxlo"], case["nxhi"], case["ng"]])
    nx = size.integers(case["nxlo"], case["nxhi"] + 1, case["nmodel"])
    lo, hi = case.get("plo", 10), case.get("phi", 10)
    npart = np.exp(size.uniform(math.log(lo), math.log(hi), case["nmodel"])).astype(np.int64)
    return W.analytic_batch(nmodel=case["nmodel"], seed=seed, ng=case["ng"], nx=nx, npart=npart,
                            t_range_days=(case.get("tlo", case.get("t_days")), case.get("thi", case.get("t_days"))))


def _hot(groups, grid, atomic=None, lines=None):
    hot = HotPath(0)
    hot.set_groups(groups.wl)
    hot.set_grid(grid.xarr, grid.vxarr, grid.vol, grid.divv)
    if atomic is not None:
        hot.set_atomic_data(np.ascontiguousarray(atomic.ion.ni, dtype=np.int32), atomic.ion.nstage - 1, lines,
                            *atomic.tables)
    return hot


# ------------------------------------------------------------------ preparation
def prepare(case, seed):
    s = globals()["_prepare_" + case["kind"]](case, seed)
    s["kind"] = case["kind"]
    torch.cuda.synchronize()
    return s


def _prepare_opacity(case, seed):
    m, at = _model(case, seed), _atomic()
    groups = W.group_grid(case["ng"])
    hot = _hot(groups, m["grid"], at, _lines(case, seed))
    nelec, oc, ginv = _populations(m)
    gas = dict(temp=_t(m["temp"]), natom=_t(m["natom"]), nelec=nelec, vol=_t(m["grid"].vol), mass=_t(m["mass"]),
               natomfr=_t(m["natomfr"]), oc=oc, ginv=ginv)
    s = dict(hot=hot, ngs=case["ngs"], mix=case["mix"], host=case["host"])
    if case["host"]:
        s["gas"] = {k: v.cpu().numpy() for k, v in gas.items()}
    else:
        nc, ng = case["nc"], case["ng"]
        s["gas"] = gas
        s["out"] = dict(sig=torch.empty(nc, dtype=F64, device=DEV), cap=torch.empty(nc, ng, device=DEV),
                        emiss=torch.empty(nc, ng, device=DEV), cap64=torch.empty(ng, nc, dtype=F64, device=DEV))
    return s


def _cotangents(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed + 77)
    nc, ng = case["nc"], case["ng"]
    r = lambda *sh: torch.randn(sh, generator=g, dtype=F64, device=DEV)
    out = [r(nc, ng), r(nc), r(nc), r(nc), r(nc, 11)]
    out[4][:, [2, 3, 4, 5, 8, 9]] = 0.0  # rows that carry no gradient
    return out


def _prepare_gradient(case, seed):
    m, at = _model(case, seed), _atomic()
    hot = _hot(W.group_grid(case["ng"]), m["grid"], at, _lines(case, seed))
    D = DifferentiableOpacity(hot, at.ion, q_temp=float(m["temp"][0]), elem_mass=_amass(), tauddmc=TAUDDMC,
                              taulump=TAULUMP)
    leaf = [_t(m[k]).requires_grad_() for k in ("temp", "rho", "X")]
    return dict(hot=hot, D=D, leaf=leaf, cot=_cotangents(case, seed))


def _prepare_coefficients(case, seed):
    b = _batch(case, seed)
    hot = HotPath(0)
    hot.set_groups(b.groups.wl)
    if case["nmodel"] == 1:
        hot.set_grid(b.xarr, b.vxarr, b.vol, b.divv)
    else:
        hot.set_models(b.nx, b.npart, b.xarr, b.vxarr, b.vol, b.divv)
    temp, rho = _t(b.temp), _t(b.rho)
    cap = _analytic_cap(temp, rho, case["ng"], seed)
    return dict(hot=hot, temp=temp, tempinv=1.0 / temp, sig=0.1 * cap[:, 0].to(F64), cap=cap)


def _prepare_saha(case, seed):
    m, at = _model(case, seed), _atomic()
    hot = _hot(W.group_grid(10), m["grid"])
    hot.set_ions(at.ion, float(m["temp"][0]))
    return dict(hot=hot, acc=case["acc"], noc=at.ion.nstage - 1, temp=_t(m["temp"]), natom=_t(m["natom"]),
                vol=_t(m["grid"].vol), natomfr=_t(m["natomfr"]),
                nelec0=torch.ones(case["nc"], dtype=F64, device=DEV))


def _prepare_dropin(case, seed):
    b = W.analytic_batch(nmodel=1, seed=seed, ng=case["ng"], nx=[case["nc"]], npart=[case["npart"]],
                         t_range_days=(case["t_days"], case["t_days"]))
    hot = HotPath(0)
    hot.set_groups(b.groups.wl)
    hot.set_grid(b.xarr, b.vxarr, b.vol, b.divv)
    return dict(hot=hot, temp=b.temp, rho=b.rho, wl=b.groups.wl, npart=case["npart"], params=W.TransportParams(),
                seed=seed, prt=np.zeros(case["npart"], dtype=PACKET_DTYPE), isv=np.ones(case["npart"], np.int32))


def _prepare_particles(case, seed):
    b = W.analytic_batch(nmodel=1, seed=seed, ng=case["ng"], nx=[case["nc"]], npart=[case["npart"]],
                         t_range_days=(case["t_days"], case["t_days"]))
    hot = HotPath(0)
    ts = BatchTimestep(hot, b, W.TransportParams(), precision=case["prec"])
    ts.prepare(seed)
    ts.sync()
    return dict(ts=ts, seed=seed, prt0=ts.prt.clone(), isv0=ts.isv.clone())


def _prepare_batch(case, seed):
    hot = HotPath(0)
    return dict(ts=BatchTimestep(hot, _batch(case, seed), W.TransportParams(), precision=case["prec"]), seed=seed)


def _prepare_timestep(case, seed):
    m, at = _model(case, seed), _atomic()
    nelec, oc, ginv = _populations(m)
    n = lambda t: t.cpu().numpy()
    gas = W.Gas(m["temp"], m["mass"], m["rho"], m["natom"], n(nelec), m["natomfr"], m["X"],
                np.ascontiguousarray(at.ion.ni, dtype=np.int32), n(oc), n(ginv))
    c = W.OpacityCase(m["grid"], W.group_grid(case["ng"]), gas, _lines(case, seed), *at.tables)
    hot = HotPath(0)
    ts = DeviceTimestep(hot, c, W.TransportParams(), npart=case["npart"], precision=case["prec"])
    emit, _ = hot.sourceenergy(m["temp"], L_BOL)
    nvol, _ = hot.sourcenumbers(emit, case["npart"])
    return dict(ts=ts, emit=emit, nvol=nvol, seed=seed)


# ------------------------------------------------------------------ one pass
# Packets are returned without their first word: an escaped particle's
# position is a marker (the largest double), which isvacant says as well.
def run(s):
    return globals()["_run_" + s["kind"]](s)


def _run_opacity(s):
    if s["host"]:
        r = s["hot"].physical_opacity(**s["gas"], ngs=s["ngs"], opacmixrossel=s["mix"], want_cap64=True)
        return {k: r[k] for k in ("sig", "cap", "emiss", "cap64", "sanity")}
    s["hot"].physical_opacity_dev(s["gas"], s["out"], ngs=s["ngs"], opacmixrossel=s["mix"])
    o = s["out"]
    return dict(sig=o["sig"], cap=o["cap"], emiss=o["emiss"], cap64=o["cap64"].T)


def _run_gradient(s):
    for p in s["leaf"]:
        p.grad = None
    outs = s["D"].opacity(*s["leaf"])
    torch.autograd.backward(outs, s["cot"])
    return dict(out=[o.detach() for o in outs], grad=[p.grad for p in s["leaf"]])


def _run_coefficients(s):
    hot = s["hot"]
    grey, ross = hot.opacity_means(s["temp"], s["sig"], s["cap"])
    lump = hot.leakage_opacity(s["tempinv"], s["sig"], s["cap"], tauddmc=TAUDDMC, taulump=TAULUMP)
    prob = hot.emission_probability(s["tempinv"], s["cap"], grey)
    hot.sync()  # the results are the context's stream's: read after it
    return dict(grey=grey, ross=ross, lump=lump, prob=prob)


def _run_saha(s):
    nelec, oc, ginv, it = s["hot"].saha_eos(s["temp"], s["natom"], s["vol"], s["natomfr"], s["nelec0"], acc=s["acc"],
                                            noc=s["noc"])
    s["hot"].sync()
    return dict(nelec=nelec, oc=oc, ginv=ginv, iterations=it)


def _run_dropin(s):
    hot, prt, isv = s["hot"], s["prt"], s["isv"]
    isv[:] = 1
    emit, _ = hot.sourceenergy(s["temp"], L_BOL)
    nvol, _ = hot.sourcenumbers(emit, s["npart"])
    hot.interior_source(s["temp"], emit, nvol, prt, isv, seed=2 * s["seed"])
    sig, cap = hot.analytic_opacity(s["temp"], s["rho"])
    grey, _ = hot.opacity_means(s["temp"], sig, cap)
    tinv = 1.0 / s["temp"]
    lump = hot.leakage_opacity(tinv, sig, cap)
    prob = hot.emission_probability(tinv, cap, grey)
    src = hot.sourcetally(prt, isv)
    r = hot.particle_advance(dict(tempinv=tinv, sig=sig, capgrey=grey, emitprob=prob, opaclump=lump, cap=cap), prt,
                             isv, s["params"], seed=2 * s["seed"] + 1)
    lum = hot.fluxtally(prt, isv, s["wl"])
    return dict(prt=prt.view(np.float64).reshape(-1, 8)[:, 1:].copy(), isv=isv.copy(), src=src, lum=lum, **_counted(r),
                **{k: r[k] for k in ("tally", "jrad", "eamp")})


COUNTS = ("npckt", "nflux", "nstepimc", "nstepddmc", "nmethodswap", "nstepmax", "nposwarn", "ierr")


def _counted(r):
    get = r.get if isinstance(r, dict) else lambda k: getattr(r, k)
    out = {k: int(get(k)) for k in COUNTS}
    out.update({k: float(get(k)) for k in ("tot_evelo", "tot_eout", "tot_sflux")})
    out["ndist"] = [int(v) for v in get("ndist")]
    return out


def _run_particles(s):
    ts = s["ts"]
    with torch.cuda.stream(ts.stream):
        ts.prt.copy_(s["prt0"])
        ts.isv.copy_(s["isv0"])
    ts.transport(s["seed"])
    ts.sync()
    return dict(prt=ts.prt[:, 1:], isv=ts.isv, tally=ts.tally, jrad=ts.jrad, eamp=ts.eamp, **_counted(ts._tout))


def _run_batch(s):
    ts = s["ts"]
    ts.step(s["seed"])
    ts.sync()
    return dict(prt=ts.prt[:, 1:], isv=ts.isv, tally=ts.tally, jrad=ts.jrad, lum=ts.lum, lumdev=ts.lumdev, lumnum=ts.lumnum,
                src=[ts.src_energy, ts.src_number], cap=ts.cap, coef=[ts.capgrey, ts.capross, ts.opaclump,
                                                                      ts.emitprob], **_counted(ts._tout))


def _run_timestep(s):
    ts = s["ts"]
    ts.hot.interior_source(ts.gas["temp"], s["emit"], s["nvol"], ts.prt, ts.isv, seed=2 * s["seed"])
    ts.step(2 * s["seed"] + 1)
    c = ts.sync()
    return dict(prt=ts.prt[:, 1:], isv=ts.isv, tally=ts.tally, jrad=ts.jrad, lum=ts.lum, lumdev=ts.lumdev, lumnum=ts.lumnum,
                src=[ts.src_energy, ts.src_number], cap=ts.cap, emiss=ts.emiss,
                coef=[ts.sig, ts.capgrey, ts.capross, ts.opaclump, ts.emitprob], **_counted(c))


# ------------------------------------------------------------------ work
TERM = 24  # flops of one line-shell term: an exp (about 20) and its products and sum


def work(case):
    k, ng = case["kind"], case.get("ng", 10)
    if k in ("opacity", "gradient"):
        nc, nl = case["nc"], case["nline"]
        pop = 16.0 * 9 * W.NELEM * nc
        if k == "opacity":
            return dict(bytes=16.0 * nl + pop + 16.0 * nc * ng, flops=TERM * float(nl) * nc + 60.0 * nc * ng)
        return dict(bytes=2 * 16.0 * nl + 32.0 * nc * ng, flops=2 * TERM * float(nl) * nc + 200.0 * nc * ng)
    if k == "coefficients":
        nc = case["nmodel"] * 0.5 * (case["nxlo"] + case["nxhi"])
        return dict(bytes=4.0 * nc * ng + 150.0 * nc, flops=40.0 * nc * ng)
    if k == "saha":
        return dict(bytes=8.0 * case["nc"] * (2 * 9 * W.NELEM + W.NELEM + 6),
                    flops=30.0 * case["nc"] * W.NELEM * 10)
    if k in ("dropin", "particles"):
        nc, npart = case["nc"], case["npart"]
    elif k == "batch":
        nc = case["nmodel"] * 0.5 * (case["nxlo"] + case["nxhi"])
        npart = case["nmodel"] * (case["phi"] - case["plo"]) / math.log(case["phi"] / case["plo"])
    else:
        nc, npart = case["nc"], case["npart"]
    # a particle is written once by its source, read and written by the loop
    # and read by the tallies; the events themselves depend on the walk
    tables = 100.0 * nc * ng
    lines = TERM * float(case["nline"]) * nc if k == "timestep" else 0.0
    return dict(bytes=(68.0 * 2 if k == "particles" else 68.0 * 5) * npart + tables, flops=lines + 3e4 * npart)


# ------------------------------------------------------------------ 64-bit values
C = 2.997924562e10
KB = 1.3806505e-16
HP = 6.6260693e-27
ME = 9.1093826e-28
QE = 4.80325e-10
RYD = 1.0973731534e5
EV = 1.60217653e-12
AMU = 1.66053886e-24
PI = math.pi
HCK = HP * C / KB
THOMSON = 8.0 * PI * QE ** 4 / (3.0 * ME ** 2 * C ** 4)
FTPI4 = 15.0 / PI ** 4


def exact(case, seed):
    f = globals().get("_exact_" + case["kind"])
    return f(case, seed) if f else None


def _ion_tensors(q_temp):
    ion = _atomic().ion
    q = np.where(np.arange(ion.nstage)[None, :] == ion.ni[:, None] - 1, 1.0, 0.0)
    for z in range(ion.nelem):
        for i in range(ion.ni[z] - 1):
            n = ion.nlevel[z, i]
            q[z, i] = (ion.glev[z, i, :n] * np.exp(-ion.elev[z, i, :n] / (KB * q_temp))).sum()
    have = torch.as_tensor(np.arange(ion.nstage)[None, :] < ion.ni[:, None], device=DEV)
    qt = torch.where(have, _t(q), 1.0)
    return _t(ion.e), qt, torch.where(have, _t(ion.g1), 1.0), have


def _stages(y, T, nd, e, q, have):
    """Stage fractions (ncell, nelem, nstage) of the Saha balance at y electrons per atom."""
    s = math.log(2.0) + 1.5 * torch.log(2 * PI * ME * KB * T / HP ** 2) - torch.log(y * nd)
    step = s[:, None, None] - e[None, :, :-1] / (KB * T)[:, None, None] + torch.log(q[:, 1:] / q[:, :-1])[None]
    phi = torch.cat([torch.zeros_like(step[..., :1]), torch.cumsum(step, -1)], -1)
    return torch.softmax(torch.where(have[None], phi, torch.full_like(phi, -1e300)), -1)


def _saha(T, natom, vol, fr, q_temp):
    """Electrons per atom, occupation densities and 1/g1 (nelem, nstage - 1, ncell)."""
    e, q, g1, have = _ion_tensors(q_temp)
    k = torch.arange(e.shape[1], dtype=F64, device=DEV)
    nd = natom / vol
    electrons = lambda y: (fr[:, 1:] * (_stages(y, T, nd, e, q, have) * k).sum(-1)).sum(-1)
    with torch.no_grad():
        lo, hi = torch.full_like(T, -30.0), torch.full_like(T, 4.0)
        for _ in range(70):
            mid = 0.5 * (lo + hi)
            up = electrons(torch.exp(mid)) > torch.exp(mid)
            lo, hi = torch.where(up, mid, lo), torch.where(up, hi, mid)
        y0 = torch.exp(0.5 * (lo + hi)).detach()
    with torch.enable_grad():
        yd = y0.clone().requires_grad_()
        d, = torch.autograd.grad((yd - electrons(yd)).sum(), yd, retain_graph=False)
    y = y0 - (y0 - electrons(y0)) / d.detach()  # a Newton step: the root, with its implicit derivative
    f = _stages(y, T, nd, e, q, have)
    oc = (nd[:, None, None] * fr[:, 1:, None] * (g1 / q)[None] * f * have[None])[..., :-1]
    ginv = (1.0 / g1)[:, :-1, None].expand(-1, -1, len(T))
    return y, oc.permute(1, 2, 0), ginv


def _populations(m):
    with torch.no_grad():
        y, oc, ginv = _saha(_t(m["temp"]), _t(m["natom"]), _t(m["grid"].vol), _t(m["natomfr"]), float(m["temp"][0]))
    return y, oc.contiguous(), ginv.contiguous()


def _exact_saha(case, seed):
    m = _model(case, seed)
    y, oc, ginv = _populations(m)
    return dict(nelec=y, oc=oc, ginv=ginv, iterations=None)


def _planck_weights(T, wl):
    """Group integrals of the normalised Planck function and of its T-derivative's weight (midpoint rule)."""
    x = HCK / T[:, None] / wl[None, :]
    xm, dx = 0.5 * (x[:, 1:] + x[:, :-1]), torch.abs(x[:, 1:] - x[:, :-1])
    xc = torch.clamp(xm, max=300.0)
    ex = torch.exp(xc)
    w = FTPI4 * dx * xc ** 3 / (ex - 1.0)
    wr = 0.25 * FTPI4 * dx * xc ** 4 * ex / (ex - 1.0) ** 2
    return w, wr


def _means(T, sig, cap, w, wr):
    return (w * cap).sum(1), 1.0 / (wr / (sig[:, None] + cap)).sum(1)


def _leakage(T, sig, cap, w, wl, X, vol, divv, first, last):
    """leakage_opacity11's rows; first/last: shells at a model's inner/outer end."""
    dx = X[1] - X[0]
    tau = (sig[:, None] + cap) * dx[:, None]
    lump = (cap * dx[:, None] >= TAULUMP) & (tau >= TAUDDMC)
    wlump = torch.where(lump, w, torch.zeros_like(w))
    sw = wlump.sum(1)
    spec = torch.where(sw > 0, 1.0 / torch.where(sw > 0, sw, torch.ones_like(sw)), torch.zeros_like(sw))
    caplump = (wlump * cap).sum(1)
    best = (wlump * cap).detach()
    top, arg = best.max(1)
    x = torch.clamp(HCK / T[:, None] / wl[None, 1:-1], max=300.0)
    thick = cap * dx[:, None] >= TAULUMP
    edge = thick[:, :-1] & ~thick[:, 1:] & (tau[:, :-1] >= TAUDDMC)
    dop = torch.where(edge, FTPI4 * x ** 4 / (torch.exp(x) - 1.0), torch.zeros_like(x)).sum(1) * divv / (3.0 * C)
    vterm = 3.0 * vol / (4.0 * PI)
    rows = []
    for side, r2, end in ((-1, X[0] ** 2, first), (1, X[1] ** 2, last)):
        nb = torch.roll(tau, -side, 0)
        bound = end[:, None] | (nb < TAUDDMC)
        a = torch.where(bound, 6.0 / (3.0 * tau + 6.0 * 0.7104), 2.0 / (tau + nb)) * (r2 / vterm)[:, None]
        rows.append((wlump * a).sum(1) * spec)
    z = torch.zeros_like(spec)
    col = [*rows, z, z, z, z, spec, caplump, z, torch.where(top > 0, arg + 1.0, 0.0).to(F64), dop]
    return torch.stack(col, 1)


def _exact_coefficients(case, seed):
    b = _batch(case, seed)
    temp, rho, wl = _t(b.temp), _t(b.rho), _t(b.groups.wl)
    cap32 = _analytic_cap(temp, rho, case["ng"], seed)
    sig, cap = 0.1 * cap32[:, 0].to(F64), cap32.to(F64)
    w, wr = _planck_weights(temp, wl)
    grey, ross = _means(temp, sig, cap, w, wr)
    co = np.concatenate([[0], np.cumsum(b.nx)])
    edge = np.arange(co[-1]) + np.repeat(np.arange(len(b.nx)), b.nx)
    X = _t(b.xarr)[torch.as_tensor(np.stack([edge, edge + 1]), device=DEV)]
    first, last = (torch.zeros(co[-1], dtype=torch.bool, device=DEV) for _ in range(2))
    first[torch.as_tensor(co[:-1], device=DEV)] = True
    last[torch.as_tensor(co[1:] - 1, device=DEV)] = True
    lump = _leakage(temp, sig, cap, w, wl, X, _t(b.vol), _t(b.divv), first, last)
    nep = int(round(math.sqrt(case["ng"])))
    nepg = math.ceil(case["ng"] / (nep + 1.0))
    run_ = torch.cumsum(w * cap, 1)
    at = torch.clamp(torch.arange(1, nep, device=DEV) * nepg, max=case["ng"]) - 1
    return dict(grey=grey, ross=ross, lump=lump, prob=torch.cat([run_[:, at], grey[:, None]], 1))


def _verner(nz, ne, e):
    """Photoionisation cross-section [Mbarn] of ion (nz, ne electrons) at energies e [eV] (numpy)."""
    ll = (0, 0, 1, 0, 1, 2, 0)
    ninn = (0, 0) + (1,) * 8 + (3,) * 8 + (5,) * 12
    ntot = (1, 1, 2, 2, 3, 3, 3, 3, 3, 3, 4, 4, 5, 5, 5, 5, 5, 5, 6, 6, 6, 6, 6, 6, 6, 6, 6, 6, 7, 7)
    at = _atomic()
    ph1 = at.bf_ph1.reshape(30, 30, 7, 6)[ne - 1, nz - 1]
    ph2 = at.bf_ph2.reshape(30, 30, 7)[ne - 1, nz - 1]
    nout = ntot[ne - 1]
    if nz > 18 and (nz == ne or (nz == ne + 1 and nz in (20, 21, 22, 25, 26))):
        nout = 7
    nint = ninn[ne - 1]
    if nz in (15, 17, 19) or (nz > 20 and nz != 26):
        einn = 0.0
    else:
        einn = float(np.float32(1e30)) if ne < 3 else float(ph1[nint - 1, 0])
    xs = np.zeros_like(e)
    for i in range(1, nout + 1):
        p = ph1[i - 1]
        on = (e >= float(ph1[nout - 1, 0])) & (e >= float(p[0]))
        if nint < i < nout:
            on &= e >= einn
        with np.errstate(all="ignore"):
            p1 = -float(p[4])
            y = e / float(p[1])
            first = (float(p[2]) * ((y - 1.0) ** 2 + float(p[5] * p[5])) * y ** (-0.5 * p1 - ll[i - 1] - 5.5) *
                     (np.sqrt(y / float(p[3])) + 1.0) ** p1)
            p1 = -float(ph2[3])
            x = e / float(ph2[0]) - float(ph2[5])
            z = np.sqrt(x * x + float(ph2[6] * ph2[6]))
            second = (float(ph2[1]) * ((x - 1.0) ** 2 + float(ph2[4] * ph2[4])) * z ** (-0.5 * p1 - 5.5) *
                      (1.0 + np.sqrt(z / float(ph2[2]))) ** p1)
            xs = xs + np.where(on, np.where((i <= nint) | (e >= einn), first, second), 0.0)
    return xs


def _line_sums(h, pop, lines, edges, slots):
    """Bound-bound sums (nsub, ncell) over each sub-group's lines, a few groups' lines at a time."""
    sub = np.searchsorted(edges, lines["wl0"].astype(np.float64) * 1e-8, side="right") - 1
    nsub = len(edges) - 1
    start = np.searchsorted(sub, np.arange(nsub + 1))
    mid, wid = 0.5 * (edges[1:] + edges[:-1]), edges[1:] - edges[:-1]
    phi = mid ** 2 / (wid * C)
    gxs, chi = lines["gxs"].astype(np.float64), _t(lines["chilw"])
    pg = _t(phi[np.clip(sub, 0, nsub - 1)] * gxs)
    slot, subt = torch.as_tensor(slots, device=DEV), torch.as_tensor(sub, device=DEV)
    most = max(1, int(3e7 / len(h)))
    out, g0 = [], 0
    while g0 < nsub:
        g1 = min(nsub, max(g0 + 1, int(np.searchsorted(start, start[g0] + most, side="right")) - 1))
        a, b = int(start[g0]), int(start[g1])

        def part(h, pop, a=a, b=b, g0=g0, g1=g1):
            v = pg[a:b, None] * pop[slot[a:b]] * torch.exp(-chi[a:b, None] * h[None, :])
            return torch.zeros(g1 - g0, len(h), dtype=F64, device=DEV).index_add(0, subt[a:b] - g0, v)

        out.append(checkpoint(part, h, pop, use_reentrant=False) if torch.is_grad_enabled() else part(h, pop))
        g0 = g1
    return torch.cat(out), _t(mid)


def _free_free(T, h, hlp, natomfr, edges):
    gff = _t(_atomic().ff_gff.reshape(41, 81).T.copy())
    wl = _t(edges[:-1])
    u = h[None, :] / wl[:, None]
    index = lambda v, n: torch.clamp(torch.floor(v.detach()), 1, n - 1).to(torch.int64)
    scale = 4.0 * QE ** 6 / (3.0 * HP * ME * C ** 4) * math.sqrt(2.0 * PI / (3.0 * ME * HP * C))
    gas = scale * torch.sqrt(h)[None, :] * (1.0 - torch.exp(-u)) * (wl ** 3)[:, None] * hlp[None, :]

    def part(h, fr, z):
        u = h[None, :] / wl[:, None]
        ru = 10.0 * (torch.log10(u) + 4.0) + 1.0
        rg = 5.0 * (torch.log10(float(z * z) * RYD * h) + 4.0) + 1.0
        iu, ig = index(ru, 81), index(rg, 41)
        du, dg = ru - iu, (rg - ig)[None, :]
        at = lambda i, j: gff[i - 1, j[None, :].expand_as(i) - 1]
        g = ((1 - du) * (1 - dg) * at(iu, ig) + du * (1 - dg) * at(iu + 1, ig) + (1 - du) * dg * at(iu, ig + 1) +
             du * dg * at(iu + 1, ig + 1))
        g = torch.where((rg > 41.0)[None, :], torch.clamp(g, min=1.0), g)
        return float(z * z) * fr[None, :] * g

    total = 0.0
    zs = range(1, W.NELEM + 1) if torch.is_grad_enabled() else ZS
    for z in zs:
        fr = natomfr[:, z]
        total = total + (checkpoint(part, h, fr, z, use_reentrant=False) if torch.is_grad_enabled()
                         else part(h, fr, z))
    return gas * total


def _opacity(T, natom, vol, natomfr, y, oc, ginv, lines, edges):
    """Sub-group opacities (nsub, ncell) and the Thomson opacity."""
    at = _atomic()
    h = HP * C / (KB * T)
    ns = oc.shape[1]
    slots = (lines["iz"].astype(np.int64) - 1) * ns + lines["ii"] - 1
    below = np.arange(ns)[None, :] < np.minimum(np.arange(1, W.NELEM + 1), at.ion.ni - 1)[:, None]
    below = torch.as_tensor(below, device=DEV)
    pop = (oc * ginv * below[..., None]).reshape(-1, len(T))
    cap, mid = _line_sums(h, pop, lines, edges, slots)
    cap = cap * (1.0 - torch.exp(-h[None, :] / mid[:, None]))
    en = HP * C / (EV * edges[:-1])
    xs = np.zeros((len(en), W.NELEM, ns))
    for z in ZS:  # the build leaves out ions without population, and their derivative
        for i in range(min(z, at.ion.ni[z - 1] - 1)):
            xs[:, z - 1, i] = _verner(z, z - i, en)
    cap = cap + (1e-18 * _t(xs.reshape(len(en), -1))) @ (oc * below[..., None]).reshape(-1, len(T))
    cap = cap + _free_free(T, h, (natom / vol) ** 2 * y, natomfr, edges)
    return cap, THOMSON * y * natom / vol


def _exact_opacity(case, seed):
    m = _model(case, seed)
    wl, ngs = W.group_grid(case["ng"]).wl, case["ngs"]
    if ngs == 1:
        edges = wl
    else:
        i = np.arange(ngs) / ngs
        edges = np.append(((1 - i)[None, :] * wl[:-1, None] + i[None, :] * wl[1:, None]).ravel(), wl[-1])
    T, natom, vol = _t(m["temp"]), _t(m["natom"]), _t(m["grid"].vol)
    with torch.no_grad():
        y, oc, ginv = _populations(m)
        sub, sig = _opacity(T, natom, vol, _t(m["natomfr"]), y, oc, ginv, _lines(case, seed), edges)
        sub = sub.reshape(case["ng"], ngs, -1)
        if ngs == 1:
            cap = sub[:, 0].T
        else:
            mean, ross = sub.mean(1), 1.0 / (1.0 / sub).mean(1)
            cap = ((1.0 - case["mix"]) * mean + case["mix"] * ross).T
        mid = _t(0.5 * (wl[1:] + wl[:-1]))
        x = torch.clamp(HCK / (mid[None, :] * T[:, None]), max=300.0)
        # B_lambda with the clamp's T/x in place of 1/wl
        b = 2.0 * HP * C ** 2 * (T[:, None] * x / HCK) ** 5 / (torch.exp(x) - 1.0) * mid ** 2 / C
        return dict(sig=sig, cap=cap, emiss=cap * b, cap64=cap, sanity=None)


def _exact_gradient(case, seed):
    m = _model(case, seed)
    T, R, X = (_t(m[k]).requires_grad_() for k in ("temp", "rho", "X"))
    g = m["grid"]
    vol, wl = _t(g.vol), W.group_grid(case["ng"]).wl
    with torch.enable_grad():
        parts = X / X.sum(1, keepdim=True) / _t(_amass())
        s = parts.sum(1)
        natom = R * vol * s / AMU
        fr = torch.cat([torch.zeros(len(T), 1, dtype=F64, device=DEV), parts / s[:, None]], 1)
        y, oc, ginv = _saha(T, natom, vol, fr, float(m["temp"][0]))
        cap, sig = _opacity(T, natom, vol, fr, y, oc, ginv, _lines(case, seed), wl)
        cap = cap.T
        w, wr = _planck_weights(T, _t(wl))
        grey, ross = _means(T, sig, cap, w, wr)
        Xe = _t(g.xarr)
        n = torch.arange(len(T), device=DEV)
        lump = _leakage(T, sig, cap, w, _t(wl), (Xe[:-1], Xe[1:]), vol, _t(g.divv), n == 0, n == len(T) - 1)
        outs = [cap, sig, grey, ross, lump]
        torch.autograd.backward(outs, _cotangents(case, seed))
    return dict(out=[o.detach() for o in outs], grad=[T.grad, R.grad, X.grad])
