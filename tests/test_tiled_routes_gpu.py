"""The tiled FP32 contractions (legendre_tile.cuh) where the calls of a plan really
take them.  The plan's stage counters say which kernels ran: an analysis that is
tiled folds its spectra first (stage "fold"), a tiled synthesis lays its
coefficients out in columns ("alm_to_columns"); the direct kernels do neither.

Tolerance 2e-6 rel-L2, as for the direct FP32 contractions: about log2(n) roundings
in the ring FFT (1e-6 at most) and sqrt(rings) in the sums.
"""

import numpy as np
import pytest
import torch

from oracle import hpx_oracle as O

pytestmark = pytest.mark.gpu


def rel(a, b):
    a = a.detach().cpu().numpy() if torch.is_tensor(a) else a
    b = b.detach().cpu().numpy() if torch.is_tensor(b) else b
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def run(plan, fn, *args):
    """fn(*args) and {stage: launches} of it."""
    plan.stats_enable(True)
    try:
        out = fn(*args)
        return out, {k: n for k, (n, _) in plan.stats_read().items() if n}
    finally:
        plan.stats_enable(False)


def test_more_orders_than_a_grid_side_takes(cuda):
    """65536 orders, the most a plan accepts; only the first 2 nside + 1 reach a ring."""
    import cuhpx_b200 as hpx

    nside, L, M, batch = 128, 2, 65536, 57
    plan = hpx.Plan(nside, L, M, "ring", "fp32", 0, batch_chunk=batch)
    rng = np.random.default_rng(0)
    a = np.zeros((batch, L, M), dtype=np.complex128)
    a[:, 0, 0], a[:, 1, 0] = rng.standard_normal((2, batch))
    a[:, 1, 1] = rng.standard_normal(batch) + 1j * rng.standard_normal(batch)
    f, ran = run(plan, plan.inverse, torch.from_numpy(a).to(cuda, torch.complex64))
    assert ran.get("alm_to_columns") == 1
    assert rel(f, O.isht(a[..., :L], nside)) < 2e-6
    b = plan.forward(f)
    assert rel(b[..., :L], O.sht(f.double().cpu().numpy(), nside, L, L)) < 2e-6
    assert torch.count_nonzero(b[..., L:]) == 0


# (nside, L, M, batch, tiled analysis, tiled synthesis); NP = 2 nside ring pairs.  The analysis
# tiles hold 32 rings by 128 degrees, the synthesis' 64 rings by 64 degrees
CASES = [
    (2, 130, 131, 64, True, False),     # four rings, M > L
    (16, 129, 33, 57, True, False),     # the first batch that takes them; the last block holds one degree
    (17, 193, 35, 64, True, False),     # NP = 34
    (33, 140, 67, 100, True, False),    # the second chunk of maps takes the direct kernel
    (64, 120, 115, 63, True, False),    # one block of degrees an order
    (128, 129, 70, 31, True, False),    # the first batch on larger grids
    (128, 131, 140, 124, True, True),   # two tiled chunks of maps, M > L
    (130, 150, 61, 57, True, True),     # NP = 260, uniform weights; the first tiled synthesis
    (256, 70, 41, 64, True, True),      # fewer degrees than a block; orders not a multiple of four
    (256, 65, 66, 47, False, True),     # the first tiled synthesis on larger grids, M > L
    (128, 300, 3, 64, True, True),      # few orders
]


@pytest.mark.parametrize("nside,L,M,batch,fwd,inv", CASES)
def test_tiled_against_oracle(cuda, nside, L, M, batch, fwd, inv):
    import cuhpx_b200 as hpx

    rng = np.random.default_rng(nside + L)
    qw = "ring" if nside & (nside - 1) == 0 else "none"
    f = rng.standard_normal((batch, 12 * nside * nside))
    pick = sorted({0, 1, min(batch, 64) - 1, batch - 1})  # maps of both chunks
    ref = O.sht(f[pick], nside, L, M, quad_weights=qw)
    g = O.isht(ref, nside)
    plan = hpx.Plan(nside, L, M, qw, "fp32", 0)
    x = torch.from_numpy(f).float().to(cuda)
    a, ran = run(plan, plan.forward, x)
    assert ("fold" in ran) == fwd
    assert rel(a[pick], ref) < 2e-6
    low = np.arange(M)[None, :] > np.arange(L)[:, None]
    assert torch.count_nonzero(a[:, torch.from_numpy(low).to(cuda)]) == 0
    b = a.clone()
    b[pick] = torch.from_numpy(ref).to(cuda, torch.complex64)
    y, ran = run(plan, plan.inverse, b)
    assert ("alm_to_columns" in ran) == inv
    assert rel(y[pick], g) < 2e-6
    r, _ = run(plan, plan.forward, x, 1)
    assert rel(r[pick], ref + O.sht(f[pick] - g, nside, L, M, quad_weights=qw)) < 4e-6


@pytest.mark.parametrize("nside,L,M,batch", [(128, 131, 140, 61), (130, 150, 61, 64), (256, 70, 41, 64)])
def test_tiled_adjoints(cuda, nside, L, M, batch):
    """Both adjoints against those of an FP64 plan (tested against the oracle by their
    dot products)."""
    import cuhpx_b200 as hpx

    qw = "ring" if nside & (nside - 1) == 0 else "none"
    p32, p64 = (hpx.Plan(nside, L, M, qw, p, 0) for p in ("fp32", "fp64"))
    gen = torch.Generator(device=cuda).manual_seed(nside)
    f = torch.randn(batch, 12 * nside * nside, generator=gen, device=cuda, dtype=torch.float64)
    g = torch.randn(batch, L, M, dtype=torch.complex128, generator=gen, device=cuda)
    u, ran = run(p32, p32.inverse_adjoint, f.float())
    assert "fold" in ran
    assert rel(u, p64.inverse_adjoint(f)) < 2e-6
    v, ran = run(p32, p32.forward_adjoint, g.to(torch.complex64))
    assert "alm_to_columns" in ran
    assert rel(v, p64.forward_adjoint(g)) < 2e-6
