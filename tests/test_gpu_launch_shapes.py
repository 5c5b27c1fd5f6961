"""Launches that would leave the chip idle: the time of a call on a grid beside the
time of one that differs from it only where a launch rule could go wrong.  Ratios
of device times (the smallest of several runs of many calls each), with a bar
well between what idle SMs cost and what the calls take.
"""
import ctypes as C

import numpy as np
import pytest
import torch

import cases
from superlite_b200 import HotPath, capi
from superlite_b200 import workloads as W
from superlite_b200.differentiable import DifferentiableOpacity
from superlite_b200.timestep import DeviceTimestep
from test_gpu_opacity import _assert_opacity_parity, _gpu_opacity, _setup

pytestmark = pytest.mark.gpu


def _us(hot, call, n=20, runs=5):
    stream = torch.cuda.ExternalStream(hot.stream())
    for _ in range(3):
        call()
    hot.sync()
    best = float("inf")
    for _ in range(runs):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        for _ in range(n):
            call()
        b.record(stream)
        b.synchronize()
        best = min(best, a.elapsed_time(b) * 1e3 / n)
    return best


def _t(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device="cuda")


def _build_us(ncell, ng, nline):
    """Device time of a physical opacity build of ncell shells (a few shells' states repeated)."""
    base = W.opacity_case(ncell=16, ng=ng, nline=nline, seed=2)
    k = np.arange(ncell) % 16
    grid = W.homologous_grid(ncell, 10 * W.PC_DAY)
    hot = HotPath(0)
    hot.set_groups(base.groups.wl)
    hot.set_grid(grid.xarr, grid.vxarr, grid.vol, grid.divv)
    g = base.gas
    hot.set_atomic_data(g.ion_ni, g.oc.shape[1], base.lines, base.bf_ph1, base.bf_ph2, base.ff_gff)
    gas = dict(temp=_t(g.temp[k]), natom=_t(g.natom[k]), nelec=_t(g.nelec[k]), vol=_t(base.grid.vol[k]),
               mass=_t(g.mass[k]), natomfr=_t(g.natomfr[k]), oc=_t(g.oc[:, :, k]), ginv=_t(g.ginv[:, :, k]))
    out = dict(sig=torch.zeros(ncell, dtype=torch.float64, device="cuda"), cap=torch.zeros(ncell, ng, device="cuda"),
               emiss=torch.zeros(ncell, ng, device="cuda"))
    torch.cuda.synchronize()
    us = _us(hot, lambda: hot.physical_opacity_dev(gas, out))
    hot.close()
    return us


def test_few_groups_on_many_shells():
    """64 groups fill neither 256 nor 1024 shells' lanes: four times the shells run
    beside one another (1.3 times the time; four groups after another in a block
    took 4.5 times)."""
    assert _build_us(1024, 64, 100_000) < 2.2 * _build_us(256, 64, 100_000)


@pytest.mark.parametrize("ncell,ng", [(96, 600), (97, 900), (128, 20), (1024, 13), (1025, 112), (2100, 7)])
def test_lines_at_the_edges_of_the_rules(hot, oracle, ncell, ng):
    case = cases.reference_opacity_case(oracle, ncell=ncell, ng=ng, nline=1500, seed=ncell, lines="synthetic")
    _setup(hot, case)
    _assert_opacity_parity(_gpu_opacity(hot, case), oracle.physical_opacity(case))


def test_several_groups_in_a_block():
    """The largest grids take groups one after another in a block: 64 shells repeated
    to 12800, 2001 groups (a remainder for four and for eight a block), against the
    64 alone, the build and its adjoint."""
    ng, n0, reps = 2001, 64, 200
    base = W.opacity_case(ncell=n0, ng=ng, nline=5000, seed=6)
    ion, g = W.ion_table(), base.gas
    rng = np.random.default_rng(8)
    weight = rng.uniform(0.5, 1.5, (n0, ng))
    res = []
    for nc in (n0, n0 * reps):
        k = np.arange(nc) % n0
        grid = W.homologous_grid(nc, 10 * W.PC_DAY)
        hot = HotPath(0)
        hot.set_groups(base.groups.wl)
        hot.set_grid(grid.xarr, grid.vxarr, grid.vol, grid.divv)
        hot.set_atomic_data(np.ascontiguousarray(ion.ni, dtype=np.int32), g.oc.shape[1], base.lines, base.bf_ph1,
                            base.bf_ph2, base.ff_gff)
        eng = DifferentiableOpacity(hot, ion, 9000.0, np.linspace(1.0, 60.0, W.NELEM), acc=1e-12)
        leaf = [_t(v).requires_grad_() for v in (g.temp[k], g.rho[k], g.massfr[k])]
        cap = eng.opacity(*leaf)[0]
        cap.backward(_t(weight)[torch.as_tensor(k, device="cuda")])
        res.append((cap.detach().cpu().numpy(), [p.grad.cpu().numpy() for p in leaf]))
        hot.close()
    (cap, grad), (caps, grads) = res
    np.testing.assert_allclose(caps.reshape(reps, n0, ng), np.broadcast_to(cap, (reps, n0, ng)), rtol=1e-11)
    for a, b in zip(grad, grads):
        b = b.reshape((reps, *a.shape))
        np.testing.assert_allclose(b, np.broadcast_to(a, b.shape), rtol=1e-8, atol=1e-10 * np.abs(a).max())


def _coefficients(hot, b, s, e):
    """Means, leakage opacities and emission probabilities of shells s (edges e) of b as one model."""
    hot.set_grid(b["xarr"][e], b["vxarr"][e], b["vol"][s], b["divv"][s])
    grey, ross = hot.opacity_means(b["temp"][s], b["sig"][s], b["cap"][s])
    tinv = 1.0 / b["temp"][s]
    return (grey, ross, hot.leakage_opacity(tinv, b["sig"][s], b["cap"][s], tauddmc=1.0, taulump=2.0),
            hot.emission_probability(tinv, b["cap"][s], grey))


@pytest.mark.parametrize("ng,sizes", [(1, [3, 2]), (33, [150, 7]), (100, [2, 350, 470]), (511, [9, 2360]),
                                      (512, [2368, 3])])
def test_cells_of_a_batch_have_the_values_of_each_alone(hot, ng, sizes):
    """Few cells run in a block each and many in a warp each: the same bits."""
    b = W.analytic_batch(nmodel=len(sizes), seed=2, ng=ng, nx=sizes, npart=[5] * len(sizes), t_range_days=(2.0, 6.0))
    rng = np.random.default_rng(ng)
    cap = ((1e18 * b.temp ** -1.5 * b.rho ** 2)[:, None] * 10 ** rng.uniform(-1.5, 1.5, (len(b.temp), ng))).astype(
        np.float32)
    d = dict(xarr=b.xarr, vxarr=b.vxarr, vol=b.vol, divv=b.divv, temp=b.temp, cap=cap, sig=0.1 * cap[:, 0].astype(
        np.float64))
    hot.set_groups(b.groups.wl)
    co = np.concatenate([[0], np.cumsum(b.nx)])
    alone = [_coefficients(hot, d, slice(co[m], co[m + 1]), slice(co[m] + m, co[m + 1] + m + 1))
             for m in range(len(sizes))]
    hot.set_models(b.nx, b.npart, b.xarr, b.vxarr, b.vol, b.divv)
    grey, ross = hot.opacity_means(b.temp, d["sig"], cap)
    lump = hot.leakage_opacity(1.0 / b.temp, d["sig"], cap, tauddmc=1.0, taulump=2.0)
    prob = hot.emission_probability(1.0 / b.temp, cap, grey)
    assert lump[:, 6].max() > 0.0  # some groups are lumped
    for m, one in enumerate(alone):
        s = slice(co[m], co[m + 1])
        for got, ref in zip(one, (grey[s], ross[s], lump[s], prob[s])):
            assert np.array_equal(got, ref)


def test_coefficients_of_few_cells():
    """64 cells of 512 groups fill the chip with a block each, as those of 513 do
    (a warp each took 2.7 times the leakage's time, 2.2 the means')."""
    us = []
    for ng in (512, 513):
        hot = HotPath(0)
        grid, rng = W.homologous_grid(64, 10 * W.PC_DAY), np.random.default_rng(1)
        hot.set_groups(W.group_grid(ng).wl)
        hot.set_grid(grid.xarr, grid.vxarr, grid.vol, grid.divv)
        temp = _t(rng.uniform(6000.0, 14000.0, 64))
        cap = _t(10 ** rng.uniform(-16.0, -10.0, (64, ng)), torch.float32)
        sig, tinv = 0.1 * cap[:, 0].double().contiguous(), 1.0 / temp
        grey, ross, lump = torch.empty_like(temp), torch.empty_like(temp), temp.new_empty((64, 11))
        p = [capi.ptr(v) for v in (temp, sig, cap, grey, ross, tinv, lump)]
        torch.cuda.synchronize()

        def call():
            hot.lib.slg_dev_opacity_means(hot.h, *p[:5])
            hot.lib.slg_dev_leakage_opacity11(hot.h, p[5], p[1], p[2], None, 5.0, 10.0, p[6])

        us.append(_us(hot, call, n=100))
        hot.close()
    assert us[0] < 1.6 * us[1]


def test_tables_of_a_launch_without_particles():
    """What a particle loop pays before its events: the FP64 loop's tables take less
    than the mixed loop's, which include the same sums (0.65; with a search for every
    guide entry and a memory access for every running sum's entry 0.81)."""
    case = W.opacity_case(ncell=256, ng=2000, nline=20000, seed=5, t_days=12.0)
    us = []
    for precision in (0, 1):
        hot = HotPath(0)
        ts = DeviceTimestep(hot, case, W.TransportParams(), npart=100, precision=precision)  # every slot vacant
        ts.opacity()
        ts.coefficients()
        hot.sync()
        us.append(_us(hot, lambda: hot.lib.slg_dev_particle_advance(
            hot.h, C.byref(ts._tin), capi.ptr(ts.prt), capi.ptr(ts.isv), 100, 7, C.byref(ts._tout))))
        hot.close()
    assert us[0] < 0.73 * us[1]
