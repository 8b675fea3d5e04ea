"""The register-cap variants of the fourth-order operator's kernels give the
same bits (every sum and product rounds as written): each variant of each
kernel, both solvers and both fallbacks."""
from __future__ import annotations

import pytest

from conftest import gpu_available

pytestmark = pytest.mark.gpu

if gpu_available():
    import torch

    import heliocubed_b200 as hc
    from heliocubed_b200.level import o4_variants


@pytest.mark.parametrize("riemann,fallback", [(1, 0), (1, 1), (2, 0), (2, 1)])
def test_variants_give_the_same_bits(riemann, fallback):
    if not gpu_available():
        pytest.skip("no CUDA device")
    sh = hc.Shell(hc.Params(nr=21, na=18, spatial_order=4, riemann_solver=riemann, berta_fallback_type=fallback))
    first = sh.init_perturbed_wind(4, amp=0.2)
    states = []
    kernels, variants = o4_variants().shape
    for choice in [(0, 0, 0)] + [tuple(v if q == k else 0 for q in range(kernels))
                                 for k in range(kernels) for v in range(1, variants)]:
        sh.set_o4_variants(*choice)
        ju = first.clone()
        for step in range(2):
            sh.rk4_step(ju, 50.0, 50.0 * step)
        states.append(ju)
    assert torch.isfinite(states[0]).all()
    for ju in states[1:]:
        assert torch.equal(ju, states[0])
