"""Component counts around the groups of eight that the coarse-fine commit and
the region copies take at a time: bit for bit against the oracle, a cell whose
last component has no data left as it was."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import gpu_available

pytestmark = pytest.mark.gpu

if gpu_available():
    import torch

    import heliocubed_b200 as hc
    from heliocubed_b200.level import AmrPlan


@pytest.mark.parametrize("ncomp", [1, 7, 8, 9, 16])
def test_commit(oracle_lib, ncomp):
    if not gpu_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(ncomp)
    plan = AmrPlan(hc.Shell(hc.Params(nr=8, na=8)), [])
    lo, cn, fn, vlo, vhi, ratio = (-3, -3, -3), (9, 9, 8), (8, 8, 8), (0, 0, 0), (3, 3, 3), (2, 2, 2)
    coarse, fine = rng.normal(size=(ncomp,) + cn[::-1]), rng.normal(size=(ncomp,) + fn[::-1])
    coarse[-1, 4, 2, 3] = np.nan
    want = fine.copy()
    oracle_lib.amr_cf_interpolate(coarse, lo, want, lo, vlo, vhi, ratio)
    dc, df = torch.from_numpy(coarse).cuda(), torch.from_numpy(fine.copy()).cuda()
    plan.set_cf_interp([{"coarse": dc, "fine": df, "coarse_lo": lo, "coarse_n": cn, "fine_lo": lo, "fine_n": fn,
                         "valid_lo": vlo, "valid_hi": vhi, "ratio": ratio, "ncomp": ncomp}])
    plan.cf_interpolate(0, 1)
    got = df.cpu().numpy()
    assert np.array_equal(got, want)
    changed = np.any(got != fine, axis=0)
    assert changed.any() and not changed.all()
    plan.close()


@pytest.mark.parametrize("ncomp", [1, 7, 8, 9, 16])
def test_copy(ncomp):
    if not gpu_available():
        pytest.skip("no CUDA device")
    plan = AmrPlan(hc.Shell(hc.Params(nr=8, na=8)), [])
    src = torch.randn((ncomp, 5, 6, 7), dtype=torch.float64, device="cuda")
    dst = torch.zeros_like(src)
    # the inner cells, mirrored along i
    plan.set_copies([dict(src=src, dst=dst, src_lo=(0, 0, 0), src_n=(7, 6, 5), dst_lo=(0, 0, 0), dst_n=(7, 6, 5),
                          lo=(1, 1, 1), hi=(5, 4, 3), perm=(0, 1, 2), sign=(-1, 1, 1), shift=(6, 0, 0), ncomp=ncomp)])
    plan.copy(0, 1)
    want = torch.zeros_like(src)
    want[:, 1:4, 1:5, 1:6] = src[:, 1:4, 1:5, 1:6].flip(-1)
    assert torch.equal(dst, want)
    plan.close()
