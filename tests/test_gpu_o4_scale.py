"""The fourth-order operator does not depend on units: density, momentum and
energy times 4^m and the field times 2^m give the rate times the same factors,
bit for bit (factors are powers of two and no floor is in reach), also where
the fields are constant (the reconstruction's weights are then smallest) and
far from 1."""
from __future__ import annotations

import pytest

from conftest import gpu_available

pytestmark = pytest.mark.gpu

if gpu_available():
    import torch

    import heliocubed_b200 as hc
    from heliocubed_b200.level import make_box, wind_box_state


@pytest.mark.parametrize("riemann", [1, 2])
@pytest.mark.parametrize("constant", [True, False])
def test_rate_scales_with_the_state(riemann, constant):
    if not gpu_available():
        pytest.skip("no CUDA device")
    p = hc.Params(nr=32, na=32, spatial_order=4, riemann_solver=riemann)
    sh = hc.Shell(p)
    lo, hi = (4, 4, 4), (15, 13, 12)
    n = 12 * 10 * 9
    u = torch.from_numpy(wind_box_state(p, lo, hi, 5, seed=1)).cuda().view(8, -1)
    if constant:
        u[:] = torch.tensor([1.0, 0, 0, 0, 1.0, 0, 0, 0], dtype=torch.float64, device="cuda")[:, None]

    def rate(m):
        f = torch.tensor([4.0 ** m] * 5 + [2.0 ** m] * 3, dtype=torch.float64, device="cuda")[:, None]
        k = torch.zeros(8 * n, dtype=torch.float64, device="cuda")
        sh.box_rhs_o4(make_box(lo, hi, 5, 1), (u * f).reshape(-1).contiguous(), k)
        return k.view(8, n) / f

    base = rate(0)
    assert torch.isfinite(base).all() and base[:4].abs().max() > 0
    for m in (100, 122, 130, 180, 220):
        assert torch.equal(rate(m), base), m
