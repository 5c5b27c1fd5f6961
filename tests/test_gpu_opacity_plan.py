"""The opacity build's layouts where they can go wrong: shell counts around the
lanes of a warp and the warps of a block, lines of one row, of every row and in
one group only, and the kept line and cross-section layout against every call
that must lay it out anew.  Against the CPU oracle (1e-12 relative, gas_cap
within one float ulp, as in test_gpu_opacity.py).
"""
import dataclasses

import numpy as np
import pytest

import cases
from test_gpu_opacity import _assert_opacity_parity, _gpu_opacity, _setup

pytestmark = pytest.mark.gpu


def _check(hot, oracle, case, **flags):
    _assert_opacity_parity(_gpu_opacity(hot, case, **flags), oracle.physical_opacity(case, **flags))


@pytest.mark.parametrize("ncell", [2, 31, 33, 63, 65, 127, 128, 129, 257, 1023, 1025])
def test_shell_counts_around_warps(hot, oracle, ncell):
    case = cases.reference_opacity_case(oracle, ncell=ncell, ng=13, nline=3000, seed=ncell, lines="synthetic")
    _setup(hot, case)
    _check(hot, oracle, case)


@pytest.mark.parametrize("which", ["one_row", "one_group", "few", "outside"])
def test_line_layouts(hot, oracle, which):
    case = cases.reference_opacity_case(oracle, ncell=37, ng=11, nline=2001, seed=3, lines="synthetic")
    lines = case.lines.copy()
    if which == "one_row":
        lines["iz"], lines["ii"] = 26, 2
    elif which == "one_group":
        lines["wl0"] = np.float32(5000.0)
    elif which == "few":
        lines = lines[:3]
    else:  # some lines below and above the groups
        lines["wl0"][:200] = np.float32(500.0)
        lines["wl0"][-200:] = np.float32(60000.0)
    case = dataclasses.replace(case, lines=lines)
    _setup(hot, case)
    _check(hot, oracle, case)


def test_cool_shell_beyond_the_fast_exp(hot, oracle):
    """A shell so cool that line exponents pass 700 (its warp takes the general exp)."""
    case = cases.reference_opacity_case(oracle, ncell=40, ng=9, nline=2000, seed=5, lines="synthetic")
    temp = case.gas.temp.copy()
    temp[7] = 60.0
    case = dataclasses.replace(case, gas=dataclasses.replace(case.gas, temp=temp))
    _setup(hot, case)
    _check(hot, oracle, case, noff=True)


def test_layout_follows_its_inputs(hot, oracle):
    """Calls in turn on one context, each after something that the kept layout depends on changed."""
    a = cases.reference_opacity_case(oracle, ncell=40, ng=30, nline=3000, seed=7, lines="synthetic")
    b = cases.reference_opacity_case(oracle, ncell=40, ng=30, nline=2000, seed=8, lines="synthetic")
    c = cases.reference_opacity_case(oracle, ncell=40, ng=45, nline=2000, seed=8, lines="synthetic")
    _setup(hot, a)
    _check(hot, oracle, a, nobb=True)
    _check(hot, oracle, a)
    _check(hot, oracle, a, ngs=3, opacmixrossel=0.25)
    _check(hot, oracle, a, nobf=True)
    _check(hot, oracle, a)
    hot.set_atomic_data(b.gas.ion_ni, b.gas.oc.shape[1], b.lines, b.bf_ph1, b.bf_ph2, b.ff_gff)
    b = dataclasses.replace(b, grid=a.grid, gas=a.gas)
    _check(hot, oracle, b)
    hot.set_groups(c.groups.wl)
    _check(hot, oracle, dataclasses.replace(b, groups=c.groups))


def test_layout_of_a_captured_graph(oracle):
    """A graph lays out what its own calls read: replays between direct calls
    with other sub-groups, and the direct calls themselves, stay right."""
    import torch
    from superlite_b200 import HotPath
    case = cases.reference_opacity_case(oracle, ncell=40, ng=30, nline=3000, seed=9, lines="synthetic")
    hot = HotPath(0)
    _setup(hot, case)
    ref1, ref2 = oracle.physical_opacity(case), oracle.physical_opacity(case, ngs=2)
    g = case.gas
    t = lambda v: torch.as_tensor(np.ascontiguousarray(v, dtype=np.float64), device="cuda")
    gas = dict(temp=t(g.temp), natom=t(g.natom), nelec=t(g.nelec), vol=t(case.grid.vol), mass=t(g.mass),
               natomfr=t(g.natomfr), oc=t(g.oc), ginv=t(g.ginv))
    nc, ng = case.grid.nx, case.groups.ng
    buf = lambda: dict(sig=torch.zeros(nc, dtype=torch.float64, device="cuda"), cap=torch.zeros(nc, ng, device="cuda"),
                       emiss=torch.zeros(nc, ng, device="cuda"),
                       cap64=torch.zeros(ng, nc, dtype=torch.float64, device="cuda"))
    one, two = buf(), buf()
    torch.cuda.synchronize()

    def ok(out, ref):
        hot.sync()
        np.testing.assert_allclose(out["cap64"].T.cpu().numpy(), ref["cap64"], rtol=1e-12)
        out["cap64"].zero_()
        torch.cuda.synchronize()

    hot.physical_opacity_dev(gas, two, ngs=2)
    ok(two, ref2)
    hot.physical_opacity_dev(gas, one)
    ok(one, ref1)
    hot.graph_begin()
    hot.physical_opacity_dev(gas, one)
    hot.graph_end()
    hot.physical_opacity_dev(gas, two, ngs=2)
    ok(two, ref2)
    hot.graph_launch(1)
    ok(one, ref1)
    hot.physical_opacity_dev(gas, two, ngs=2)
    ok(two, ref2)
    hot.graph_launch(1)
    ok(one, ref1)
    hot.physical_opacity_dev(gas, one)
    ok(one, ref1)
    hot.close()


def test_cool_shell_leaves_its_neighbours_alone(hot, oracle):
    """A shell beyond the fast exp's range does not change a bit of the others',
    whatever lane or warp they are in."""
    case = cases.reference_opacity_case(oracle, ncell=140, ng=9, nline=2000, seed=5, lines="synthetic")
    _setup(hot, case)
    a = _gpu_opacity(hot, case)["cap64"]
    cool = [6, 77, 139]
    temp = case.gas.temp.copy()
    temp[cool] = 60.0
    b = _gpu_opacity(hot, dataclasses.replace(case, gas=dataclasses.replace(case.gas, temp=temp)))["cap64"]
    rest = np.setdiff1d(np.arange(140), cool)
    assert np.array_equal(a[rest], b[rest])
    assert not np.array_equal(a[cool], b[cool])


def test_without_bound_free_tables(hot, oracle):
    """No bound-free fits set: ions without population need none, and populated ones
    give NaN and its sanity bit (no read through a null table)."""
    import ctypes as C
    from superlite_b200.capi import ptr
    case = cases.reference_opacity_case(oracle, ncell=20, ng=15, nline=500, seed=4, lines="synthetic")
    _setup(hot, case)
    ni, lines = np.ascontiguousarray(case.gas.ion_ni, dtype=np.int32), np.ascontiguousarray(case.lines)
    gff = np.ascontiguousarray(case.ff_gff, dtype=np.float64)
    rc = hot.lib.slg_set_atomic_data(hot.h, len(ni), case.gas.oc.shape[1], ptr(ni), C.c_int64(len(lines)), ptr(lines),
                                     None, None, ptr(gff))
    assert rc == 0
    bare = dataclasses.replace(case, gas=dataclasses.replace(case.gas, oc=np.zeros_like(case.gas.oc)))
    _check(hot, oracle, bare)
    got = _gpu_opacity(hot, case, nobf=True)
    _assert_opacity_parity(got, oracle.physical_opacity(case, nobf=True))
    got = _gpu_opacity(hot, case)
    assert np.isnan(got["cap64"]).any() and got["sanity"] & 4
