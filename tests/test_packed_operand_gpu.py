"""Tensor-core calls of few maps: packed operand rows against the 128-column ones
(17 maps take those) and against the oracle, for map counts up to the packed
limit, orders and degrees around the tiles' edges, and both 16-bit formats.
"""

import numpy as np
import pytest
import torch

from oracle import hpx_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nside,L,M", [(16, 33, 33), (32, 65, 40), (64, 260, 129), (128, 257, 255)])
@pytest.mark.parametrize("prec,tol", [("f16x3", 2e-6), ("bf16x3", 3e-5)])  # tolerances of the tensor-core paths
def test_packed_against_full_rows_and_oracle(cuda, nside, L, M, prec, tol):
    import cuhpx_b200 as hpx

    rng = np.random.default_rng(nside)
    f = rng.standard_normal((17, 12 * nside * nside))
    x = torch.from_numpy(f).float().to(cuda)
    plan = hpx.get_plan(nside, L, M, "ring", prec, 0)
    assert plan.table_bytes > 0
    a = plan.forward(x)
    y = plan.inverse(a)
    rel = lambda u, v: float((u - v).norm() / v.norm())  # noqa: E731
    for n in (1, 5, 16):
        assert rel(plan.forward(x[:n]), a[:n]) < tol
        assert rel(plan.inverse(a[:n].contiguous()), y[:n]) < tol
    ref = O.sht(f[:2], nside, L, M)
    assert np.linalg.norm(plan.forward(x[:9])[:2].cpu().numpy() - ref) < tol * np.linalg.norm(ref)
    r = plan.forward(x[:9], iters=1)
    ref1 = ref + O.sht(f[:2] - O.isht(ref, nside), nside, L, M)
    assert np.linalg.norm(r[:2].cpu().numpy() - ref1) < 2 * tol * np.linalg.norm(ref1)
    plan.check()
