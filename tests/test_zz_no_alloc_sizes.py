"""slg_particle_advance_static at group counts around one emission bin, ragged last
bins and its limit on shells x groups: it searches whole tables where the context
entry has guides, so the same events and results show both right."""
import numpy as np
import pytest

import cases
from superlite_b200 import capi
from test_zz_no_alloc import _dev, _run_existing, _run_static

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ng", [(64, 1), (64, 2), (64, 3), (64, 5), (64, 17), (64, 101), (64, 2047), (3, 700)])
def test_static_entry_matches_context_entry(hot, oracle, nx, ng):
    import torch
    lib = capi.load()
    c = cases.transport_case(oracle, t_days=6.0, nx=nx, ng=ng, npart=400, kind="mono", seed=ng)
    hot.set_groups(c["groups"].wl)
    hot.set_grid(c["grid"].xarr, c["grid"].vxarr, c["grid"].vol, c["grid"].divv)
    t = c["tables"]
    tables = {k: _dev(t[k], torch, torch.float32 if k == "cap" else None) for k in t}
    grid_arrays = dict(xarr=_dev(c["grid"].xarr, torch), vxarr=_dev(c["grid"].vxarr, torch),
                       divv=_dev(c["grid"].divv, torch), wl=_dev(c["groups"].wl, torch),
                       wlinv=_dev(c["groups"].wlinv, torch))
    pa = torch.as_tensor(c["prt"].view(np.float64).reshape(-1, 8)).cuda()
    va = torch.as_tensor(c["isv"]).cuda()
    pb, vb = pa.clone(), va.clone()
    oa, ta, ja, _ = _run_existing(hot, c, tables, pa, va, 21, torch)
    ob, tb, jb, _ = _run_static(lib, c, tables, pb, vb, 21, torch, grid_arrays)
    torch.cuda.synchronize()
    assert oa.nstepimc + oa.nstepddmc >= 400
    for k in ("npckt", "nflux", "nstepimc", "nstepddmc", "nmethodswap", "nstepmax", "nposwarn", "ierr"):
        assert getattr(ob, k) == getattr(oa, k), k
    assert list(ob.ndist) == list(oa.ndist)
    assert np.array_equal(vb.cpu().numpy(), va.cpu().numpy())
    live = (va == 0).cpu().numpy()
    np.testing.assert_allclose(pb.cpu().numpy()[live], pa.cpu().numpy()[live], rtol=1e-10, atol=0)
    np.testing.assert_allclose(tb.cpu().numpy(), ta.cpu().numpy(), rtol=1e-9, atol=1e-300)
    np.testing.assert_allclose(jb.cpu().numpy(), ja.cpu().numpy(), rtol=1e-9, atol=1e-300)
