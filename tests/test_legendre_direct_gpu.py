"""The direct Legendre contractions (legendre_direct.cuh) at the edges of their
tiles: orders not a multiple of the CTA's four, ring counts around the 64 and
128 rings of a warp, map groups of 1, 2 and up to 4, degree chunks of 64 and
128, both precisions, accumulation (refinement) and the adjoints.

Tolerances: FP64 1e-11 (as for every FP64 path); FP32 2e-6 rel-L2: about
log2(n) roundings in the ring FFT (1e-6 at most) and sqrt(rings) in the sums.
"""

import numpy as np
import pytest
import torch

from oracle import hpx_oracle as O

pytestmark = pytest.mark.gpu


def rel(a, b):
    a = a.detach().cpu().numpy() if torch.is_tensor(a) else a
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


# (nside, L, M, batch): NP = 2 nside ring pairs
CASES = [
    (1, 2, 1, 1),
    (16, 21, 33, 1),     # M > L: whole orders of zeros
    (31, 65, 63, 2),     # NP = 62
    (33, 66, 30, 3),     # NP = 66
    (64, 64, 129, 4),    # NP = 128
    (65, 130, 131, 5),   # NP = 130
    (96, 290, 70, 9),    # L far above 2 nside: starts inside most chunks
    (128, 511, 257, 10),  # degree chunks of 128
]


@pytest.mark.parametrize("nside,L,M,batch", CASES)
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_direct_against_oracle(cuda, nside, L, M, batch, dtype):
    import cuhpx_b200 as hpx

    tol = 1e-11 if dtype == torch.float64 else 2e-6
    rng = np.random.default_rng(nside + L)
    qw = "ring" if nside > 1 and nside & (nside - 1) == 0 else "none"
    f = rng.standard_normal((batch, 12 * nside * nside))
    ref = O.sht(f, nside, L, M, quad_weights=qw)
    x = torch.from_numpy(f).to(cuda, dtype)
    kw = dict(lmax=L, mmax=M, quad_weights=qw)
    a = hpx.SHTCUDA(nside, **kw)(x)
    assert rel(a, ref) < tol
    low = np.arange(M)[None, :] > np.arange(L)[:, None]
    assert torch.count_nonzero(a[:, torch.from_numpy(low).to(cuda)]) == 0
    # every map of the batch as it comes out alone
    one = hpx.SHTCUDA(nside, **kw)(x[batch - 1])
    assert rel(one, ref[batch - 1]) < tol
    y = hpx.iSHTCUDA(nside, **kw)(torch.from_numpy(ref).to(cuda, a.dtype))
    g = O.isht(ref, nside)
    assert rel(y, g) < tol
    r = hpx.SHTCUDA(nside, refine_iters=1, **kw)(x)
    assert rel(r, ref + O.sht(f - g, nside, L, M, quad_weights=qw)) < 2 * tol


@pytest.mark.parametrize("nside,L,M,batch", [(33, 66, 30, 3), (64, 127, 127, 6)])
def test_direct_adjoints(cuda, nside, L, M, batch):
    import cuhpx_b200 as hpx

    rng = np.random.default_rng(7)
    plan = hpx.get_plan(nside, L, M, "none", "fp64", 0)
    f = torch.from_numpy(rng.standard_normal((batch, 12 * nside * nside))).to(cuda)
    g = torch.from_numpy(rng.standard_normal((batch, L, M)) + 1j * rng.standard_normal((batch, L, M))).to(cuda)
    dot = lambda u, v: float((u.conj() * v).real.sum())  # noqa: E731
    lhs, rhs = dot(plan.forward(f), g), float((f * plan.forward_adjoint(g)).sum())
    assert abs(lhs - rhs) < 1e-11 * float(f.norm() * plan.forward_adjoint(g).norm())
    lhs, rhs = float((plan.inverse(g) * f).sum()), dot(g, plan.inverse_adjoint(f))
    assert abs(lhs - rhs) < 1e-11 * float(f.norm() * plan.inverse(g).norm())


# spin-1: one, two and an odd number of vector maps; ring counts around 64 and 128; L above 2 nside
@pytest.mark.parametrize("nside,L,M,batch", [(2, 3, 4, 1), (16, 35, 30, 2), (32, 66, 64, 3), (64, 190, 127, 1)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_direct_spin1_against_oracle(cuda, nside, L, M, batch, dtype):
    import cuhpx_b200 as hpx
    from oracle import vector_oracle as V

    tol = 1e-11 if dtype == torch.float64 else 2e-6
    rng = np.random.default_rng(nside + L)
    f = rng.standard_normal((batch, 2, 12 * nside * nside))
    ref = V.vsht(f, nside, L, M)
    a = hpx.VectorSHTCUDA(nside, L, M)(torch.from_numpy(f).to(cuda, dtype))
    assert rel(a, ref) < tol
    y = hpx.VectoriSHTCUDA(nside, L, M)(torch.from_numpy(ref).to(cuda, a.dtype))
    assert rel(y, V.visht(ref, nside)) < tol


# mixed plans: a few maps take the FP32 direct contractions (with and without the
# Legendre table), one more takes the tensor cores
@pytest.mark.parametrize("nside,L,M,few,table", [(32, 65, 63, 16, True), (128, 200, 150, 4, True), (32, 65, 63, 8, False)])
def test_mixed_plans_of_few_maps(cuda, nside, L, M, few, table):
    import cuhpx_b200 as hpx

    rng = np.random.default_rng(nside)
    f = rng.standard_normal((few + 1, 12 * nside * nside))
    ref = O.sht(f[:2], nside, L, M)
    x = torch.from_numpy(f).float().to(cuda)
    kw = dict(lmax=L, mmax=M, precision="f16x3", legendre_table=table)
    for n in (2, few, few + 1):
        a = hpx.SHTCUDA(nside, **kw)(x[:n])
        assert rel(a[:2], ref) < 2e-6
        y = hpx.iSHTCUDA(nside, **kw)(a)
        assert rel(y[:2], O.isht(ref, nside)) < 4e-6


@pytest.mark.parametrize("batch", [31, 48, 49, 67])
def test_fp64_analysis_around_the_tiled_kernel(cuda, batch):
    """FP64 analysis changes kernels above 48 maps of a block of up to 64."""
    import cuhpx_b200 as hpx

    nside, L, M = 12, 30, 29
    f = np.random.default_rng(batch).standard_normal((batch, 12 * nside * nside))
    ref = O.sht(f, nside, L, M, quad_weights="none")
    sht = hpx.SHTCUDA(nside, lmax=L, mmax=M, quad_weights="none")
    a = sht(torch.from_numpy(f).to(cuda))
    assert rel(a, ref) < 1e-11
    assert rel(a[batch - 1], ref[batch - 1]) < 1e-11
