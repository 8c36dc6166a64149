"""The direct analysis' groups of 1, 2 and 4 maps a CTA (FP64: 1 and 2) at partial
groups, on grids below and above the 64 ring pairs where a lane takes 2 or 4 rings.
A pass takes the widest group that leaves a CTA an SM, so the wide ones need many
degrees: ceil(M / 4) orders by ceil(L / 64) chunks of degrees come to 160 CTAs and
more here, and to 17 and fewer in the cases of narrow groups.

Tolerances: FP64 1e-11, FP32 2e-6 rel-L2, as for the other direct contractions.
"""

import numpy as np
import pytest
import torch

from oracle import hpx_oracle as O

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(a.detach().cpu().numpy() - b) / np.linalg.norm(b))


@pytest.mark.parametrize("nside,L,M", [
    (31, 577, 63),  # 62 pairs, 16 x 10 CTAs a group
    (33, 610, 66),  # 66 pairs, 17 x 10
    (31, 64, 63),   # 16 x 1: narrow groups
    (33, 66, 65),   # 17 x 2
    (66, 40, 5),    # 2 x 1, 132 pairs
])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_groups_of_maps_against_oracle(cuda, nside, L, M, dtype):
    import cuhpx_b200 as hpx

    tol = 1e-11 if dtype == torch.float64 else 2e-6
    plan = hpx.get_plan(nside, L, M, "none", "fp64" if dtype == torch.float64 else "fp32", 0)
    f = np.random.default_rng(nside + L).standard_normal((9, 12 * nside * nside))
    ref = O.sht(f, nside, L, M, quad_weights="none")
    g = O.isht(ref[:7], nside)
    x = torch.from_numpy(f).to(cuda, dtype)
    for n in (1, 2, 3, 4, 5, 9):
        a = plan.forward(x[:n])
        assert rel(a, ref[:n]) < tol, n
        assert rel(a[n - 1], ref[n - 1]) < tol, n
    r = plan.forward(x[:7], 1)  # accumulates into the coefficients
    assert rel(r, ref[:7] + O.sht(f[:7] - g, nside, L, M, quad_weights="none")) < 2 * tol
