"""The particle loop's per-shell tables where they can go wrong: the emission
thresholds (one flat list for the reference's two-level emission bins), and
the guide ranges, DDMC branch probabilities and resolved-group entries at
group counts around the edges of the guide sizes and emission bins.
"""
import math

import numpy as np
import pytest

import cases
from superlite_b200 import workloads as W


# ---------------------------------------------------------------- CPU: the rule
def _binsrch(x, arr):
    """MISC/binsrch.f90 with widerange, 1-based."""
    n = len(arr)
    if n == 2:
        return 1 if arr[0] <= x <= arr[1] else (0 if x < arr[0] else (n if x > arr[1] else -1))
    lo, hi, mid = 1, n, (n + 1) // 2
    while hi - lo > 1:
        if arr[lo - 1] <= x < arr[mid - 1]:
            hi, mid = mid, (mid + lo) // 2
        elif arr[mid - 1] <= x <= arr[hi - 1]:
            lo, mid = mid, (hi + mid) // 2
        else:
            return 0 if x < arr[0] else (n if x > arr[n - 1] else -1)
    return mid if mid == lo else -1


def _emitgroup(r1, ep, w, nep, nepg, ng):
    """emitgroup.f:3-54 on emission bins ep and group terms w."""
    iep = max(_binsrch(r1, ep), 0)
    ig0 = iep * nepg + 1
    top = min(ig0 + nepg - 1, ng)
    if ig0 > top - 1:
        return min(ig0, ng)
    p = 0.0 if iep == 0 else ep[iep - 1]
    for g in range(ig0, top):
        p = p + w[g - 1]
        if p > r1:
            return g
    return top


def _thresholds(ep, w, nep, nepg, ng):
    last = min(nepg + 1 if nep == 1 else nep * nepg, ng)
    t = np.full(ng, np.inf)
    for b in range(nep):
        g0 = b * nepg + 1
        g1 = min(g0 + nepg - 1, last)
        p = 0.0 if b == 0 else ep[b - 1]
        nxt = np.inf if b == nep - 1 else ep[b]
        for g in range(g0, g1):
            p = p + w[g - 1]
            t[g - 1] = min(p, nxt)
        if g0 <= g1 < last:
            t[g1 - 1] = nxt
    return t[:max(last - 1, 0)], last


@pytest.mark.parametrize("ng", [1, 2, 3, 4, 5, 6, 7, 12, 30, 31, 97, 100, 101])
@pytest.mark.parametrize("gaps", [False, True])
def test_flat_emission_thresholds_give_emitgroup(ng, gaps):
    rng = np.random.default_rng(ng)
    nep = int(round(math.sqrt(ng)))
    nepg = math.ceil(ng / (nep + 1.0))
    for trial in range(4):
        w = 10.0 ** rng.uniform(-20, 0, ng)
        if gaps:
            w[rng.random(ng) < 0.4] = 0.0  # runs of equal sums
        run, ep = 0.0, np.zeros(nep)
        for b in range(nep - 1):
            s = 0.0
            for g in range(b * nepg, min((b + 1) * nepg, ng)):
                s = s + w[g]
            run = run + s
            ep[b] = run
        ep[nep - 1] = float(np.sum(w[::-1]))  # capgrey: another order of summation
        t, last = _thresholds(ep, w, nep, nepg, ng)
        assert np.all(np.diff(t) >= 0)
        for r in np.concatenate([rng.random(300), [2.0 ** -53, 1 - 2.0 ** -53], np.clip(t / (ep[-1] or 1.0), 0, 0.999)]):
            r1 = r * ep[-1]
            got = last if nep == 1 else 1 + int(np.sum(~(t > r1)))
            assert got == _emitgroup(r1, ep, w, nep, nepg, ng), (trial, r)


# ---------------------------------------------------------------- GPU: against the oracle
@pytest.mark.gpu
@pytest.mark.parametrize("ng,nx,t_days,kind,kw", [
    (1, 6, 5.0, "grey", {}), (2, 5, 4.0, "grey", {}), (3, 2, 6.0, "grey", {}), (5, 3, 5.0, "grey", {}),
    (16, 20, 5.0, "mono", {}), (17, 20, 6.0, "mono", {}), (33, 20, 5.0, "grey+sig", {"noampfact": False}),
    (129, 24, 6.0, "mono", {}), (255, 16, 7.0, "grey+sig", {}), (64, 16, 5.0, "mono", {"puretran": True}),
    (2500, 12, 6.0, "mono", {}), (100, 24, 6.0, "mono", {"taulump": 5.0}), (100, 24, 3.0, "mono", {"tauddmc": 3.0}),
])
def test_event_sequences_at_table_edges(hot, oracle, ng, nx, t_days, kind, kw):
    from test_gpu_transport import _compare, _run_both
    c = cases.transport_case(oracle, t_days=t_days, nx=nx, ng=ng, npart=600, seed=ng, kind=kind,
                             params=W.TransportParams(max_steps=20000, errorfatal=False, **kw))
    ref, got, o, g = _run_both(hot, oracle, c)
    assert ref["nstepimc"] + ref["nstepddmc"] > 600
    _compare(ref, got, o, g)
