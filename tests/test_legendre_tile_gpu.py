"""The tiled FP32 contractions of many maps (legendre_tile.cuh) at the edges of
their tiles: 32- and 64-ring stages, 64- and 128-degree blocks, map counts from
the first that takes them to a full chunk and into a second one, orders without
rings or degrees, accumulation and the adjoint weights.

Tolerance 2e-6 rel-L2, as for the direct FP32 contractions.
"""

import numpy as np
import pytest
import torch

from oracle import hpx_oracle as O

pytestmark = pytest.mark.gpu


def rel(a, b):
    a = a.detach().cpu().numpy() if torch.is_tensor(a) else a
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


CASES = [
    (2, 3, 5, 64),       # one stage of 4 rings, M > L
    (16, 64, 33, 40),    # NP = 32, L = 64
    (17, 65, 35, 64),    # NP = 34, L = 65
    (32, 129, 63, 63),   # NP = 64
    (33, 128, 67, 100),  # NP = 66, two chunks of maps
    (48, 190, 50, 64),   # L far above 2 nside: starts inside most blocks
    (64, 257, 129, 64),
]


@pytest.mark.parametrize("nside,L,M,batch", CASES)
def test_tiled_against_oracle(cuda, nside, L, M, batch):
    import cuhpx_b200 as hpx

    rng = np.random.default_rng(nside + L)
    qw = "ring" if nside & (nside - 1) == 0 else "none"
    f = rng.standard_normal((batch, 12 * nside * nside))
    ref = O.sht(f, nside, L, M, quad_weights=qw)
    x = torch.from_numpy(f).float().to(cuda)
    kw = dict(lmax=L, mmax=M, quad_weights=qw)
    a = hpx.SHTCUDA(nside, **kw)(x)
    assert rel(a, ref) < 2e-6
    low = np.arange(M)[None, :] > np.arange(L)[:, None]
    assert torch.count_nonzero(a[:, torch.from_numpy(low).to(cuda)]) == 0
    y = hpx.iSHTCUDA(nside, **kw)(torch.from_numpy(ref).to(cuda, torch.complex64))
    g = O.isht(ref, nside)
    assert rel(y, g) < 2e-6
    assert rel(y[-1], g[-1]) < 2e-6
    if batch == 64:
        r = hpx.SHTCUDA(nside, refine_iters=1, **kw)(x)
        assert rel(r, ref + O.sht(f - g, nside, L, M, quad_weights=qw)) < 4e-6


def test_tiled_adjoints_match_the_direct_ones(cuda):
    import cuhpx_b200 as hpx

    plan = hpx.get_plan(32, 70, 63, "ring", "fp32", 0)
    gen = torch.Generator(device=cuda).manual_seed(5)
    f = torch.randn(64, 12 * 32 * 32, generator=gen, device=cuda)
    g = torch.randn(64, 70, 63, dtype=torch.complex64, generator=gen, device=cuda)
    for full, part in ((plan.inverse_adjoint(f), plan.inverse_adjoint(f[:8])),
                       (plan.forward_adjoint(g), plan.forward_adjoint(g[:8]))):
        assert rel(full[:8], part.cpu().numpy()) < 2e-6
