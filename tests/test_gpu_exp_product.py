"""The opacity kernels' exp in the form that they use it: exp(-chi h), chi a line's
single-precision energy and h one double per shell (test_gpu_exp.py has chi = 1).
Builds of one line per group, whose opacity is that exp times known factors,
against 80-bit arithmetic, over arguments from 0 to 690, among them products next
to odd multiples of ln2/128, where the nearest multiple of ln2/64 changes.

Bar, from the operations: the exp within 1 ulp (2.2e-16), three roundings of the
products (1.1e-16 each), the factor 1 - exp(-x) (x > 2.5: an ulp of exp times at most
0.09, and its own rounding) and of pg and the population (half an ulp each):
8.5e-16 relative.
"""
import math

import numpy as np
import pytest

from superlite_b200 import workloads as W

pytestmark = pytest.mark.gpu

BAR = 8.5e-16


@pytest.mark.parametrize("ncell", [20, 300])  # one and two shells per lane
def test_exp_of_products(hot, ncell):
    rng = np.random.default_rng(ncell)
    ng, iz, nst = 3000, 26, 4
    wl = np.geomspace(1000e-8, 4000e-8, ng + 1)
    grid = W.homologous_grid(ncell, 10 * W.PC_DAY)
    temp = rng.uniform(6000.0, 14000.0, ncell)
    hc = 2.997924562e10 * 6.6260693e-27
    h = hc / (1.3806505e-16 * temp)
    x = np.concatenate([rng.uniform(0.0, 690.0, ng - 1100), (2 * rng.integers(0, 127000 // 2, 1000) + 1) * (math.log(2) / 128),
                        10.0 ** rng.uniform(-8.0, 0.0, 100)])
    chi = (np.minimum(x, 690.0) / h[rng.integers(0, ncell, ng)]).astype(np.float32)
    chi = np.minimum(chi, np.float32(690.0 / h.max()))
    lines = np.zeros(ng, dtype=W.BBXS_DTYPE)
    lines["wl0"] = (0.5 * (wl[1:] + wl[:-1]) * 1e8).astype(np.float32)
    lines["gxs"] = rng.uniform(0.5, 2.0, ng).astype(np.float32)
    lines["chilw"], lines["iz"], lines["ii"] = chi, iz, 1
    hot.set_groups(wl)
    hot.set_grid(grid.xarr, grid.vxarr, grid.vol, grid.divv)
    ph1, ph2 = W.synthetic_verner()
    hot.set_atomic_data(np.full(30, 5, dtype=np.int32), nst, lines, ph1, ph2, W.synthetic_gaunt())
    oc, one = np.zeros((30, nst, ncell)), np.ones(ncell)
    oc[iz - 1, 0] = rng.uniform(1e9, 1e10, ncell)
    got = hot.physical_opacity(temp, one, one, grid.vol, one, np.zeros((ncell, 31)), oc, np.ones_like(oc), nobf=True,
                               noff=True, nothmson=True, want_cap64=True)["cap64"]
    wa, wb = wl[:-1], wl[1:]
    mid = 0.5 * (wa + wb)
    pg = mid * mid / ((wb - wa) * 2.997924562e10) * lines["gxs"].astype(np.float64)
    L = np.longdouble
    hl = h.astype(L)[:, None]
    ref = (np.exp(-chi.astype(L)[None, :] * hl) * pg.astype(L)[None, :] * oc[iz - 1, 0].astype(L)[:, None]
           * (1 - np.exp(-hl / mid.astype(L)[None, :])))
    assert np.finfo(L).eps < 2e-19
    rel = np.abs((got.astype(L) - ref) / ref).astype(np.float64)
    assert rel.max() < BAR, (rel.max(), np.unravel_index(rel.argmax(), rel.shape))
