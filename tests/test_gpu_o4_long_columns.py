"""Columns of the fourth-order face kernels at their full length (16 faces, as
every level from 64 x 64^2 up has them): a batch long enough for it, with boxes
whose extents along the march leave short last columns (17, 33) and boxes of
one to three cells among them, gives the same rhs and face fluxes, bit for bit,
as one call per box, where columns are one to five faces."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import gpu_available

pytestmark = pytest.mark.gpu

# whole panels carry the total; the march runs along k, or j for the faces of k
SIZES = [(64, 64, 64), (64, 17, 64), (64, 64, 33), (5, 1, 9), (9, 2, 1), (1, 3, 2), (64, 64, 64), (33, 1, 64),
         (64, 64, 64), (7, 64, 3), (64, 64, 64), (2, 16, 17)]


@pytest.mark.parametrize("riemann", [1, 2])
def test_long_columns_equal_short_ones(riemann):
    if not gpu_available():
        pytest.skip("no CUDA device")
    import torch

    import heliocubed_b200 as hc
    from heliocubed_b200.level import O4Batch, make_box, wind_box_state
    # 16 faces a column from 148 x 1024 x 16 faces on
    assert sum(np.prod(n) // n[d] * (n[d] + 1) for n in SIZES for d in range(3)) >= 16 * 148 * 1024
    p = hc.Params(nr=64, na=64, spatial_order=4, riemann_solver=riemann)
    shell = hc.Shell(p)
    z = lambda c: torch.zeros(int(c), dtype=torch.float64, device="cuda")  # noqa: E731
    works = []
    for q, n in enumerate(SIZES):
        lo = tuple((13 * (q + d)) % (65 - n[d]) for d in range(3))
        hi = tuple(lo[d] + n[d] - 1 for d in range(3))
        u = torch.from_numpy(wind_box_state(p, lo, hi, 5, seed=q)).cuda()
        works.append((make_box(lo, hi, 5, q % 6), u, z(8 * np.prod(n)),
                      [z(8 * np.prod(n) // n[d] * (n[d] + 1)) for d in range(3)]))
    batch = O4Batch(shell, works)
    batch.rhs()
    for box, u, rhs, fl in works:
        r1, f1 = torch.zeros_like(rhs), [torch.zeros_like(f) for f in fl]
        shell.box_rhs_o4(box, u, r1, f1)
        assert torch.isfinite(rhs).all() and rhs.abs().max() > 0
        assert torch.equal(rhs, r1)
        for a, b in zip(fl, f1):
            assert torch.equal(a, b)
    batch.close()
