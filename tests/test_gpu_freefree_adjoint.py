"""The free-free part of the opacity's adjoint at group counts around a warp's
64 groups, a block's 512 and one more round of both, and shell counts around the
line kernel's 32 and 64 shells: directional derivatives of weighted group
opacities with few lines against central differences of the forward.

Tolerance: the difference quotient (step 1e-6) carries the forward's rounding,
about 1e-14 of the sum of the absolute terms over the step, 1e-8 of it, and a
truncation error of 1e-12 times a third derivative of up to (chi / kT)^3 ~ 1e4 times the
value, again 1e-8; 1e-6 of the derivative as in the other difference tests.
"""
import pytest
import torch

import cases
from test_gpu_adjoint import _setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc,ng,nline", [(2, 1, 3), (5, 63, 50), (33, 65, 50), (32, 512, 200), (65, 513, 200),
                                         (3, 1100, 50)])
def test_group_and_shell_counts(nc, ng, nline):
    hot, D, case, T, R, X = _setup(nc=nc, ng=ng, nline=nline, seed=ng, atomic=cases.atomic_data())
    gen = torch.Generator(device=T.device).manual_seed(nc)
    with torch.no_grad():
        cap = D.opacity(T, R, X)[0]
    w = torch.randn(cap.shape, generator=gen, device=T.device, dtype=torch.float64) / cap
    size = float((w * cap).abs().sum())
    leaf = [p.clone().requires_grad_() for p in (T, R, X)]
    (w * D.opacity(*leaf)[0]).sum().backward()
    h = 1e-6
    for k, base in enumerate((T, R, X)):
        v = torch.randn(base.shape, generator=gen, device=T.device, dtype=torch.float64) * base
        args = [T, R, X]

        def at(s):
            with torch.no_grad():
                return float((w * D.opacity(*args[:k], base + s * h * v, *args[k + 1:])[0]).sum())

        fd = (at(1.0) - at(-1.0)) / (2.0 * h)
        ad = float((leaf[k].grad * v).sum())
        assert abs(ad - fd) <= 1e-6 * abs(fd) + 2e-8 * size, (k, ad, fd, size)
    hot.close()
