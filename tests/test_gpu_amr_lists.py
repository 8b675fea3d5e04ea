"""AMR work lists of every chunk length (hc_amr.cu, splitChunks): element
totals on both sides of the lengths' edges, items shorter than a chunk, of one
element and with a remainder, and ranges that begin inside the list.
Tolerance: exact (the tableau's products round as written; copies move bits)."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import gpu_available

pytestmark = pytest.mark.gpu

if gpu_available():
    import torch

    import heliocubed_b200 as hc
    from heliocubed_b200.level import AmrPlan

EDGE = 1024 * 1184  # the largest total of the shortest chunk


@pytest.mark.parametrize("total", [EDGE // 8, EDGE // 8 + 1, 2 * EDGE // 8 + 1, 16 * EDGE // 8 + 3])
def test_rk_combine_at_the_chunk_edges(oracle_lib, total):
    if not gpu_available():
        pytest.skip("no CUDA device")
    po = oracle_lib
    rng = np.random.default_rng(total)
    sh = hc.Shell(hc.Params(nr=8, na=8))
    cells = [1, 129, total // 3, total - 130 - total // 3]
    host = [(rng.normal(size=8 * n), rng.normal(size=8 * n)) for n in cells]
    dev = []
    for state, k in host:
        zero = [torch.zeros(state.size, dtype=torch.float64, device="cuda") for _ in range(4)]
        zero[0].copy_(torch.from_numpy(k))
        dev.append((torch.from_numpy(state).cuda(), torch.zeros(state.size, dtype=torch.float64, device="cuda"), zero))
    plan = AmrPlan(sh, dev)
    plan.rk_stage(4, 1, 0.37)
    for (state, k), d in zip(host, dev):
        stage = np.zeros_like(state)
        po.amr_rk_stage(state, stage, [k] + [np.zeros_like(state) for _ in range(3)], 4, 1, 0.37)
        assert np.array_equal(d[1].cpu().numpy(), stage)
    plan.close()


@pytest.mark.parametrize("n", [(5, 7, 9), (106, 106, 106), (131, 107, 103)])
def test_copy_ranges_of_long_lists(n):
    if not gpu_available():
        pytest.skip("no CUDA device")
    sh = hc.Shell(hc.Params(nr=8, na=8))
    plan = AmrPlan(sh, [])
    gen = torch.Generator(device="cuda").manual_seed(1)
    sizes = [(1, 1, 1), n, (3, 2, 17), n]
    src = [torch.randn((2,) + s[::-1], dtype=torch.float64, device="cuda", generator=gen) for s in sizes]
    dst = [torch.zeros_like(s) for s in src]
    plan.set_copies([dict(src=a, dst=b, src_lo=(0, 0, 0), src_n=s, dst_lo=(0, 0, 0), dst_n=s, lo=(0, 0, 0),
                          hi=tuple(x - 1 for x in s), perm=(0, 1, 2), sign=(1, 1, 1), shift=(0, 0, 0), ncomp=2)
                     for a, b, s in zip(src, dst, sizes)])
    plan.copy(1, 2)
    torch.cuda.synchronize()
    for q in range(4):
        assert torch.equal(dst[q], src[q] if q in (1, 2) else torch.zeros_like(src[q]))
    plan.close()
