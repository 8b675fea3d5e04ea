"""AMR conversion lists (hc_amr.cu, splitChunks with kConversionCtas) on both
sides of the chunk lengths' edges.  Tolerance: exact."""
from __future__ import annotations

import pytest

from conftest import gpu_available

pytestmark = pytest.mark.gpu

if gpu_available():
    import torch

    import heliocubed_b200 as hc
    from heliocubed_b200.level import AmrPlan


@pytest.mark.parametrize("nbox", [14, 15, 30])
def test_conversions_of_long_lists(nbox):
    """<JU> and <U> recovery in lists whose boxes are one CTA's rounds each,
    cut in two, and cut with a remainder, bit for bit as one box at a time
    (whose pieces are the shortest): 34^3 mapped cells a box, 592 x 1024
    elements being the largest total of the shortest chunk."""
    if not gpu_available():
        pytest.skip("no CUDA device")
    sh = hc.Shell(hc.Params(nr=8, na=8))
    gen = torch.Generator(device="cuda").manual_seed(nbox)
    sizes = [(30, 30, 30)] * nbox + [(31, 29, 17), (5, 3, 2)]
    boxes = []
    for n in sizes:
        rand = lambda c, g: torch.rand((c,) + tuple(x + 2 * g for x in n[::-1]), dtype=torch.float64,  # noqa: E731
                                       device="cuda", generator=gen) + 0.5
        lo, grown = (0, 0, 0), lambda g: ((-g,) * 3, tuple(x + 2 * g for x in n))  # noqa: E731
        boxes.append({"jac": rand(1, 3), "donor": rand(8, 3), "state": rand(8, 0), "mapped": rand(8, 2) * 0,
                      "out": rand(8, 0) * 0, "jac_lo": grown(3)[0], "jac_n": grown(3)[1], "donor_lo": grown(3)[0],
                      "donor_n": grown(3)[1], "state_lo": lo, "state_n": n, "mapped_lo": grown(2)[0],
                      "mapped_n": grown(2)[1], "out_lo": lo, "out_n": n, "valid_lo": lo,
                      "valid_hi": tuple(x - 1 for x in n), "block_lo": (-20, -20, -20), "block_hi": (60, 60, 60)})
    plan = AmrPlan(sh, [])
    plan.set_cf_fine(boxes)
    plan.cf_mapped(0, len(boxes))
    plan.cf_quotient(0, len(boxes))
    for q in (0, nbox - 1, nbox, nbox + 1):
        one = dict(boxes[q], mapped=torch.zeros_like(boxes[q]["mapped"]), out=torch.zeros_like(boxes[q]["out"]))
        single = AmrPlan(sh, [])
        single.set_cf_fine([one])
        single.cf_mapped(0, 1)
        single.cf_quotient(0, 1)
        assert one["out"].abs().min() > 0
        assert torch.equal(boxes[q]["mapped"], one["mapped"]) and torch.equal(boxes[q]["out"], one["out"])
        single.close()
    plan.close()
