"""The particle loops' tables: what a launch of each precision allocates, and launches
of both in turn on one context, also between the replays of a captured graph (each
precision has buffers of its own, so neither moves the other's)."""
import numpy as np
import pytest
import torch

from superlite_b200 import HotPath
from superlite_b200 import workloads as W
from superlite_b200.timestep import DeviceTimestep

pytestmark = pytest.mark.gpu


def _step(precision, hot=None, ncell=48, ng=120, npart=4000):
    case = W.opacity_case(ncell=ncell, ng=ng, nline=5000, seed=5, t_days=20.0)
    hot = hot or HotPath(0)
    ts = DeviceTimestep(hot, case, W.TransportParams(), npart=npart, precision=precision)
    emit, _ = hot.sourceenergy(case.gas.temp, 1e42)
    nvol, _ = hot.sourcenumbers(emit, npart)
    hot.interior_source(ts.gas["temp"], emit, nvol, ts.prt, ts.isv, seed=3)
    # a thin analytic opacity keeps the histories short
    rho = 1e-13 * (1.0 + np.arange(ncell)) / ncell
    sig, cap = hot.analytic_opacity(case.gas.temp, rho, kind=2, capcoef=2e31)
    ts.sig.copy_(torch.as_tensor(sig))
    ts.cap.copy_(torch.as_tensor(cap))
    hot.sync()
    grey, _ = hot.opacity_means(ts.gas["temp"], ts.sig, ts.cap)
    ts.capgrey.copy_(grey)
    torch.cuda.synchronize()
    ts.coefficients()
    hot.sync()
    ts.prt0, ts.isv0 = ts.prt.clone(), ts.isv.clone()
    torch.cuda.synchronize()
    return hot, ts


def _run(ts, seed=7):
    ts.restore_particles()
    ts.transport(seed)


def _result(ts):
    ts.sync()
    return ts.prt.clone(), ts.isv.clone(), ts.tally.clone()


def _same(a, b):
    assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
    torch.testing.assert_close(a[2], b[2], rtol=1e-9, atol=0)


@pytest.mark.parametrize("precision,most", [(1, 110.0), (0, 150.0)])
def test_bytes_per_shell_and_group(precision, most):
    """A launch allocates what its own loop reads: 89 B per (shell, group) mixed (175
    with the FP64 loop's rates, records, guides and entries), 133 B FP64."""
    nc, ng = 400, 8000
    case = W.opacity_case(ncell=nc, ng=ng, nline=100, seed=5, t_days=12.0)
    hot = HotPath(0)
    ts = DeviceTimestep(hot, case, W.TransportParams(), npart=10, precision=precision)  # every slot vacant
    ts.opacity()
    ts.coefficients()
    hot.sync()
    before = torch.cuda.mem_get_info()[0]
    ts.transport(3)
    ts.sync()
    used = before - torch.cuda.mem_get_info()[0]
    hot.close()
    assert used < most * nc * ng


def test_precisions_in_turn():
    ref = []
    for precision in (0, 1):
        hot, ts = _step(precision)
        _run(ts)
        ref.append(_result(ts))
        assert ts.counters()["nstepddmc"] > 0 and ts.counters()["nstepimc"] > 0
        hot.close()
    hot, ts = _step(1)
    for precision in (1, 0, 1, 0):
        ts._tin.precision = precision
        _run(ts)
        _same(_result(ts), ref[precision])
    # another grid in between: both loops' tables are made anew
    _step(0, hot=hot, ncell=60, ng=90)
    hot2, ts2 = _step(0, hot=hot)
    for precision in (0, 1):
        ts2._tin.precision = precision
        _run(ts2)
        _same(_result(ts2), ref[precision])
    hot.close()


@pytest.mark.parametrize("captured", [1, 0])
def test_other_precision_between_replays(captured):
    hot, ts = _step(captured)
    _run(ts)
    ref = _result(ts)
    hot.graph_begin()
    _run(ts)
    hot.graph_end()
    ts._tin.precision = 1 - captured
    _run(ts)
    ts.sync()
    hot.graph_launch(1)
    hot.sync()
    _same((ts.prt.clone(), ts.isv.clone(), ts.tally.clone()), ref)
    hot.close()
