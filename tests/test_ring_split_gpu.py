"""How the ring CTAs share a call must not change a map's transform: both rings of a pair per CTA (up to 16 maps; one launch for all rings of a
small call) against one ring per CTA (more maps), whole and partial map groups.
"""

import pytest
import torch

pytestmark = pytest.mark.gpu


# nside 1: two pairs; 5, 33: Bluestein rings and few powers of two; 64: the usual mixture;
# 600: a grid with 3072-point rings
@pytest.mark.parametrize("nside,L", [(1, 3), (5, 11), (33, 40), (64, 60), (600, 24)])
@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_ring_split_agrees(cuda, nside, L, prec):
    import cuhpx_b200 as hpx

    plan = hpx.get_plan(nside, L, L, "none", prec, 0)
    gen = torch.Generator(device=cuda).manual_seed(nside)
    x = torch.randn(19, 12 * nside * nside, generator=gen, device=cuda, dtype=plan.dtype)
    a = plan.forward(x)  # one ring a CTA
    y = plan.inverse(a)
    tol = 1e-12 if prec == "fp64" else 1e-6
    for n in (3, 16):  # both rings a CTA
        assert torch.equal(plan.inverse(a[:n].contiguous()), y[:n])
        # (the analysis contraction cuts its degrees by the batch: equal to rounding)
        assert float((plan.forward(x[:n]) - a[:n]).norm() / a[:n].norm()) < tol
    # a single map goes through the one-map contraction: equal to rounding
    one = plan.inverse(plan.forward(x[18:]))
    assert float((one[0] - y[18]).norm() / y[18].norm()) < 10 * tol
