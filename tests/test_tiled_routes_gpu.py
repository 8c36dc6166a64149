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
