"""Columns of the fourth-order face kernels: a batch large enough that a
thread marches over several faces (averages and final fluxes) gives the same
rhs and face fluxes, bit for bit, as one call per box, where every column is
one face.  Sizes leave partial columns, partial tiles and rows that do not
fill a CTA; both solvers."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import gpu_available

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("riemann,n", [(2, (31, 33, 29)), (1, (40, 26, 35)), (2, (8, 64, 17))])
def test_columns_equal_single_faces(riemann, n):
    if not gpu_available():
        pytest.skip("no CUDA device")
    import torch

    import heliocubed_b200 as hc
    from heliocubed_b200.level import O4Batch, make_box, wind_box_state
    # 148 x 1024 faces per face of a column: these batches march over 3 to 6
    faces = sum(np.prod(n) // n[d] * (n[d] + 1) for d in range(3))
    nbox = int(np.ceil(4 * 148 * 1024 / faces))
    p = hc.Params(nr=64, na=64, spatial_order=4, riemann_solver=riemann)
    shell = hc.Shell(p)
    z = lambda c: torch.zeros(int(c), dtype=torch.float64, device="cuda")  # noqa: E731
    works = []
    for q in range(nbox):
        lo = ((5 * q) % (65 - n[0]), (3 * q) % (65 - n[1]), (7 * q) % (65 - n[2]))
        hi = tuple(lo[d] + n[d] - 1 for d in range(3))
        u = torch.from_numpy(wind_box_state(p, lo, hi, 5, seed=q)).cuda()
        fl = [z(8 * np.prod(n) // n[d] * (n[d] + 1)) for d in range(3)]
        works.append((make_box(lo, hi, 5, q % 6), u, z(8 * np.prod(n)), fl))
    batch = O4Batch(shell, works)
    batch.rhs()
    for box, u, rhs, fl in works[::7]:
        r1, f1 = torch.zeros_like(rhs), [torch.zeros_like(f) for f in fl]
        shell.box_rhs_o4(box, u, r1, f1)
        assert torch.equal(rhs, r1)
        for a, b in zip(fl, f1):
            assert torch.equal(a, b)
    batch.close()
