"""Saha balance where the populations of the stages leave the middle of the
double range: cool shells, whose upper stages underflow through the denormals,
and hot thin ones, whose products overflow so that the chain starts again at a
higher stage, with one shell more and less than a block's four.

Tolerance: a population carries the rounding of up to 30 stages' exps, each
about |e/kT| 1e-16 <= 7e-14 relative: 2e-12; below 1e-290 an ulp of a denormal
is larger than that, so those are compared absolutely."""
import numpy as np
import pytest

from superlite_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc,tlo,thi,thin", [(1, 9000.0, 9000.0, 1.0), (3, 4000.0, 6000.0, 1.0),
                                             (5, 3e4, 3e5, 1e-6), (33, 4000.0, 1e5, 1e-3)])
def test_populations_at_the_ends_of_the_range(hot, oracle, nc, tlo, thi, thin):
    ion = W.ion_table()
    rng = np.random.default_rng(nc)
    grid = W.homologous_grid(nc, 8.0 * W.PC_DAY)
    rho, _ = W.broken_powerlaw_rho(grid)
    T = np.geomspace(tlo, thi, nc)
    X = np.zeros((nc, W.NELEM))
    X[:, [z - 1 for z in W.ELEMENTS]] = rng.dirichlet(np.ones(len(W.ELEMENTS)), nc)
    mass, natom, natomfr = W.composition_state(rho * thin, X, grid.vol)
    hot.set_groups(W.group_grid(10).wl)
    hot.set_grid(grid.xarr, grid.vxarr, grid.vol, grid.divv)
    q = hot.set_ions(ion, q_temp=float(T[0]))
    nel, oc, ginv, it = hot.saha_eos(T, natom, grid.vol, natomfr, np.ones(nc), acc=1e-14, noc=4)
    no, oco, gio, ito = oracle.saha_eos(ion, q, T, natom, grid.vol, natomfr, np.ones(nc), acc=1e-14, noc=4)
    np.testing.assert_allclose(nel, no, rtol=2e-12)
    np.testing.assert_allclose(oc, oco, rtol=2e-12, atol=1e-290 * float(natom.max()))
