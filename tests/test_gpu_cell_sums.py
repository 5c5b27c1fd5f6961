"""Means, leakage opacities and emission probabilities at group counts around
the edge between a warp and a block per cell, the tiles of the emission bins
and a warp's lanes, on one model and on several, against the CPU oracle (1e-11
relative for the tree-reduced sums, 1e-13 for the emission bins, which are
summed in the reference's order)."""
import numpy as np
import pytest

import cases
from superlite_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ng,nx,t_days", [(1, 5, 5.0), (2, 9, 5.0), (31, 8, 4.0), (33, 17, 5.0), (512, 9, 5.0),
                                          (513, 9, 6.0), (4100, 3, 5.0), (9001, 2, 5.0)])
def test_sums_over_groups(hot, oracle, ng, nx, t_days):
    c = cases.transport_case(oracle, t_days=t_days, nx=nx, ng=ng, npart=nx + 20, kind="mono", seed=ng)
    hot.set_groups(c["groups"].wl)
    g, t = c["grid"], c["tables"]
    hot.set_grid(g.xarr, g.vxarr, g.vol, g.divv)
    sig = 0.2 * t["cap"][:, 0].astype(np.float64)
    grey, ross = hot.opacity_means(c["temp"], sig, t["cap"])
    np.testing.assert_allclose(grey, oracle.planckmean(c["groups"].wlinv, c["temp"], t["cap"]), rtol=1e-11)
    np.testing.assert_allclose(ross, oracle.rossmean(c["groups"].wlinv, c["temp"], sig, t["cap"]), rtol=1e-11)
    for tauddmc, taulump, capemit in ((5.0, 10.0, None), (1.0, 2.0, t["cap"][:, ::-1].copy())):
        got = hot.leakage_opacity(t["tempinv"], sig, t["cap"], capemit=capemit, tauddmc=tauddmc, taulump=taulump)
        kw = {} if capemit is None else dict(capemit=capemit)
        ref = oracle.leakage_opacity11(g, c["groups"].wlinv, t["tempinv"], sig, t["cap"], tauddmc=tauddmc,
                                       taulump=taulump, **kw)
        col = [0, 1, 6, 7, 8, 10]
        np.testing.assert_allclose(got[:, col], ref[:, col], rtol=1e-11, atol=0)
        assert np.array_equal(got[:, 9], ref[:, 9])
    got = hot.emission_probability(t["tempinv"], t["cap"], t["capgrey"])
    np.testing.assert_allclose(got, t["emitprob"], rtol=1e-13, atol=0)


@pytest.mark.parametrize("ng", [100, 600])
def test_several_models_equal_each_alone(hot, oracle, ng):
    b = W.analytic_batch(nmodel=3, seed=2, ng=ng, nx=[2, 17, 9], npart=[5, 5, 5], t_range_days=(3.0, 8.0))
    cap = (1e18 * b.temp ** -1.5 * b.rho ** 2)[:, None] * np.linspace(0.2, 5.0, ng)[None, :]
    cap, sig = cap.astype(np.float32), np.zeros(len(b.temp))
    hot.set_groups(b.groups.wl)
    hot.set_models(b.nx, b.npart, b.xarr, b.vxarr, b.vol, b.divv)
    grey, ross = hot.opacity_means(b.temp, sig, cap)
    lump = hot.leakage_opacity(1.0 / b.temp, sig, cap)
    prob = hot.emission_probability(1.0 / b.temp, cap, grey)
    co = np.concatenate([[0], np.cumsum(b.nx)])
    for m in range(3):
        s, e = slice(co[m], co[m + 1]), slice(co[m] + m, co[m + 1] + m + 1)
        hot.set_grid(b.xarr[e], b.vxarr[e], b.vol[s], b.divv[s])
        g1, r1 = hot.opacity_means(b.temp[s], sig[s], cap[s])
        assert np.array_equal(g1, grey[s]) and np.array_equal(r1, ross[s])
        assert np.array_equal(hot.leakage_opacity(1.0 / b.temp[s], sig[s], cap[s]), lump[s])
        assert np.array_equal(hot.emission_probability(1.0 / b.temp[s], cap[s], g1), prob[s])
