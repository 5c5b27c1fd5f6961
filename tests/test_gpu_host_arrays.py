"""Results of host calls around the sizes where their copies change from the
context's pinned block to direct ones (256 KiB a call): the opacity build
on host arrays against the CPU oracle (as in test_gpu_opacity.py), and after a call
that failed on the way."""
import ctypes as C

import numpy as np
import pytest

import cases
from superlite_b200 import capi
from test_gpu_opacity import _assert_opacity_parity, _gpu_opacity, _setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc,ng", [(3, 10), (64, 200), (64, 256), (64, 511), (128, 513), (200, 50)])
def test_opacity_on_host_arrays(hot, oracle, nc, ng):
    case = cases.reference_opacity_case(oracle, ncell=nc, ng=ng, nline=500, seed=nc, lines="synthetic")
    _setup(hot, case)
    want = oracle.physical_opacity(case)
    for _ in range(2):
        _assert_opacity_parity(_gpu_opacity(hot, case), want)
        gas = capi.SlgGas(*[None] * 8)  # refused: no arrays
        out = [np.full(nc, 7.0), np.full((nc, ng), 7, np.float32), np.full((nc, ng), 7, np.float32)]
        rc = hot.lib.slg_physical_opacity(hot.h, C.byref(gas), C.byref(capi.SlgOpacityFlags(0, 0, 0, 0, 1, 0.0)),
                                          *[capi.ptr(o) for o in out], None, None)
        assert rc != 0 and all((o == 7).all() for o in out)
