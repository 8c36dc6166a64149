"""The tensor-core contractions where the calls of a plan really take them: mixed
plans send a few maps to the direct FP32 kernels, so these batches lie above every
such limit (16 maps with the Legendre table, 12 without), or inside the range of the
packed operand rows (up to 16 maps on grids of more than 128 ring pairs).  The
plan's stage counters say which kernels ran: an analysis on the tensor cores ends
with the stage "columns_to_alm", a synthesis begins with "alm_to_columns".

Tolerances (rel-L2) as for the other tests of these paths: one transform against the
float64 oracle 3e-5 (bf16x3) or 2e-6 (f16x3); refined analysis 1e-5 or 2e-6.
"""

import numpy as np
import pytest
import torch

from oracle import hpx_oracle as O

pytestmark = pytest.mark.gpu

TOL = {"bf16x3": 3e-5, "f16x3": 2e-6}
TOL_REFINED = {"bf16x3": 1e-5, "f16x3": 2e-6}
FULL = 17    # maps: more than any direct limit and than the packed rows hold
SHOWN = [0, 7, 16]  # maps compared with the oracle


@pytest.fixture(scope="module")
def hpx(cuda):
    import cuhpx_b200

    return cuhpx_b200


def rel(a, b):
    a = a.detach().cpu().numpy() if torch.is_tensor(a) else np.asarray(a)
    b = b.detach().cpu().numpy() if torch.is_tensor(b) else np.asarray(b)
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def rand_alm(rng, L, M, batch=(), decay=0.0):
    a = rng.standard_normal(batch + (L, M)) + 1j * rng.standard_normal(batch + (L, M))
    a = a / (np.arange(L)[:, None] + 1.0) ** decay
    a = np.where(np.arange(M)[None, :] <= np.arange(L)[:, None], a, 0)
    a[..., 0] = a[..., 0].real
    return a


def on_tensor_cores(plan, fn, *args):
    plan.stats_enable(True)
    try:
        out = fn(*args)
        ran = {k for k, (n, _) in plan.stats_read().items() if n}
    finally:
        plan.stats_enable(False)
    assert ran & {"columns_to_alm", "alm_to_columns"}, ran
    plan.check()
    return out


CASES = [(4, 9, 9), (8, 31, 17), (8, 9, 17), (8, 17, 5), (16, 33, 33), (32, 65, 65), (64, 127, 127), (128, 255, 255),
         (64, 257, 129)]


@pytest.mark.parametrize("tab", [True, False], ids=["table", "otf"])
@pytest.mark.parametrize("prec", ["bf16x3", "f16x3"])
@pytest.mark.parametrize("nside,L,M", CASES)
def test_full_rows_against_oracle(hpx, cuda, nside, L, M, prec, tab):
    rng = np.random.default_rng(nside + L + M)
    plan = hpx.get_plan(nside, L, M, "ring", prec, 0, 64, tab)
    assert (plan.table_bytes > 0) == tab
    f = rng.standard_normal((FULL, 12 * nside * nside))
    a = on_tensor_cores(plan, plan.forward, torch.from_numpy(f).float().to(cuda))
    assert rel(a[SHOWN], O.sht(f[SHOWN], nside, L, M)) < TOL[prec]
    low = np.arange(M)[None, :] > np.arange(L)[:, None]
    assert torch.count_nonzero(a[:, torch.from_numpy(low).to(cuda)]) == 0
    c = rand_alm(rng, L, M, (FULL,))
    g = on_tensor_cores(plan, plan.inverse, torch.from_numpy(c).to(cuda, torch.complex64))
    assert rel(g[SHOWN], O.isht(c[SHOWN], nside)) < TOL[prec]


# packed rows: odd orders and degrees around the tiles' edges (32-ring and 32-degree pairs of
# stages, 256-degree and 128-ring tiles)
@pytest.mark.parametrize("prec", ["bf16x3", "f16x3"])
@pytest.mark.parametrize("nside,L,M", [(65, 131, 97), (72, 64, 65), (96, 257, 33), (128, 255, 254), (128, 33, 129),
                                       (160, 63, 64)])
def test_packed_rows_against_oracle_and_full_rows(hpx, cuda, nside, L, M, prec):
    rng = np.random.default_rng(nside + L)
    qw = "ring" if nside & (nside - 1) == 0 else "none"
    plan = hpx.get_plan(nside, L, M, qw, prec, 0)
    assert plan.table_bytes > 0
    f = rng.standard_normal((FULL, 12 * nside * nside))
    x = torch.from_numpy(f).float().to(cuda)
    c = torch.from_numpy(rand_alm(rng, L, M, (FULL,)))
    z = c.to(cuda, torch.complex64)
    full_a, full_g = on_tensor_cores(plan, plan.forward, x), on_tensor_cores(plan, plan.inverse, z)
    ref, g = O.sht(f[SHOWN[:2]], nside, L, M, quad_weights=qw), O.isht(c.numpy()[SHOWN[:2]], nside)
    for n in (9, 12, 16):
        a = on_tensor_cores(plan, plan.forward, x[:n])
        y = on_tensor_cores(plan, plan.inverse, z[:n].contiguous())
        assert torch.equal(a, full_a[:n]) and torch.equal(y, full_g[:n])  # the same products and sums
        assert rel(a[SHOWN[:2]], ref) < TOL[prec]
        assert rel(y[SHOWN[:2]], g) < TOL[prec]


@pytest.mark.parametrize("nside,L,batch,tab", [(32, 63, FULL, True), (32, 63, FULL, False), (96, 120, 12, True)])
@pytest.mark.parametrize("prec", ["bf16x3", "f16x3"])
@pytest.mark.parametrize("k", [1, 2])
def test_refined_matches_fp64_refined(hpx, cuda, k, prec, nside, L, batch, tab):
    rng = np.random.default_rng(10 + k)
    qw = "ring" if nside & (nside - 1) == 0 else "none"
    pick = [0, batch - 1]
    f = O.isht(rand_alm(rng, L, L, (batch,), decay=1.0), nside) + 1e-3 ** 0.5 * rng.standard_normal((batch, 12 * nside * nside))
    ref = O.sht(f[pick], nside, L, L, quad_weights=qw)
    for _ in range(k):
        ref = ref + O.sht(f[pick] - O.isht(ref, nside), nside, L, L, quad_weights=qw)
    plan = hpx.get_plan(nside, L, L, qw, prec, 0, 64, tab)
    out = on_tensor_cores(plan, plan.forward, torch.from_numpy(f).float().to(cuda), k)
    assert rel(out[pick], ref) < TOL_REFINED[prec]


@pytest.mark.parametrize("nside,L,batch,tab", [(32, 65, FULL, True), (32, 65, FULL, False), (96, 97, 10, True)])
def test_f16x3_per_map_scale(hpx, cuda, nside, L, batch, tab):
    """Maps (and coefficient sets) many decades apart in one batch, and an all-zero
    one, each with the accuracy of an unscaled map: full rows, on the fly, packed."""
    rng = np.random.default_rng(5)
    qw = "ring" if nside & (nside - 1) == 0 else "none"
    scales = np.ones(batch)
    scales[:5] = [1.0, 1e-30, 1e30, 3e-8, 0.0]
    scales[-1] = 7e11
    pick = [0, 1, 2, 3, batch - 1]
    plan = hpx.get_plan(nside, L, L, qw, "f16x3", 0, 64, tab)
    base = rng.standard_normal((batch, 12 * nside * nside))
    a = on_tensor_cores(plan, plan.forward, torch.from_numpy(base * scales[:, None]).float().to(cuda)).cpu().numpy()
    alm = rand_alm(rng, L, L, (batch,))
    c = torch.from_numpy(alm * scales[:, None, None]).to(torch.complex64).to(cuda)
    g = on_tensor_cores(plan, plan.inverse, c).cpu().numpy()
    assert np.count_nonzero(a[4]) == 0 and np.count_nonzero(g[4]) == 0
    ref, gref = O.sht(base[pick], nside, L, L, quad_weights=qw), O.isht(alm[pick], nside)
    for k, i in enumerate(pick):
        assert rel(a[i] / scales[i], ref[k]) < 2e-6, i
        assert rel(g[i] / scales[i], gref[k]) < 2e-6, i


@pytest.mark.parametrize("prec", ["bf16x3", "f16x3"])
def test_table_matches_on_the_fly(hpx, cuda, prec):
    """Equal up to the FP32 rounding of Pbar (the two round at different points)."""
    nside, L = 64, 127
    gen = torch.Generator(device=cuda).manual_seed(11)
    f = torch.randn(FULL, 12 * nside * nside, generator=gen, device=cuda)
    pt, po = (hpx.get_plan(nside, L, L, "ring", prec, 0, 64, t) for t in (True, False))
    at, ao = on_tensor_cores(pt, pt.forward, f), on_tensor_cores(po, po.forward, f)
    assert not torch.equal(at, ao)  # two kernels
    assert rel(at, ao) < 1e-6
    assert rel(on_tensor_cores(pt, pt.inverse, at), on_tensor_cores(po, po.inverse, at)) < 1e-6


@pytest.mark.parametrize("grid", ["equiangular", "legendre-gauss", "lobatto"])
@pytest.mark.parametrize("prec", ["bf16x3", "f16x3"])
def test_latlon_against_oracle(hpx, cuda, prec, grid):
    from oracle import latlon_oracle as LO

    rng = np.random.default_rng(3)
    nlat, nlon = 96, 192
    f = rng.standard_normal((FULL, nlat, nlon))
    sht = hpx.RealSHT(nlat, nlon, grid=grid, csphase=False, precision=prec)
    L, M = sht.lmax, sht.mmax
    plan = hpx.get_latlon_plan(nlat, nlon, L, M, grid, prec, 0)
    a = on_tensor_cores(plan, sht, torch.from_numpy(f).float().to(cuda))
    assert rel(a[SHOWN], LO.latlon_sht(f[SHOWN], L, M, grid)) < TOL[prec]
    alm = rand_alm(rng, L, M, (FULL,))
    if M > nlon // 2:
        alm[..., nlon // 2] = alm[..., nlon // 2].real
    isht = hpx.InverseRealSHT(nlat, nlon, grid=grid, csphase=False, precision=prec)
    g = on_tensor_cores(plan, isht, torch.from_numpy(alm).to(torch.complex64).to(cuda))
    assert rel(g[SHOWN], LO.latlon_isht(alm[SHOWN], nlat, nlon, grid)) < TOL[prec]


def test_ragged_groups_of_many_maps(hpx, cuda):
    """Groups on the tensor cores next to one on the direct kernels, in one call."""
    gen = torch.Generator(device=cuda).manual_seed(1)
    nsides, counts = [8, 16, 32], [20, 3, 17]
    maps = [torch.randn(c, 12 * n * n, generator=gen, device=cuda) for n, c in zip(nsides, counts)]
    out = hpx.RaggedSHT(nsides, precision="f16x3")(maps)
    back = hpx.RaggedISHT(nsides, precision="f16x3")(out)
    for x, a, y, n in zip(maps, out, back, nsides):
        L = 2 * n - 1
        plan = hpx.get_plan(n, L, L, "ring", "f16x3", 0)
        assert torch.equal(a, plan.forward(x)) and torch.equal(y, plan.inverse(a))
        assert rel(a[:2], O.sht(x[:2].double().cpu().numpy(), n, L, L)) < 2e-6


@pytest.mark.parametrize("batch", [5, FULL])
def test_benchmark_size_spot_orders(hpx, cuda, batch):
    """nside 1024, L = M = 2047 on packed (5) and full rows: the first and last maps'
    orders against the oracle at the plan's own ring nodes."""
    nside, L, spot = 1024, 2047, [0, 1, 511, 1023, 2046]
    gen = torch.Generator(device=cuda).manual_seed(batch)
    p64, plan = hpx.get_plan(nside, L, L, "ring", "fp64", 0), hpx.get_plan(nside, L, L, "ring", "f16x3", 0)
    c = torch.randn(2, L, L, dtype=torch.complex128, generator=gen, device=cuda)
    c = c.tril() / (torch.arange(L, device=cuda, dtype=torch.float64)[:, None] + 1.0)
    c[..., 0] = c[..., 0].real.to(c.dtype)
    f = p64.inverse(c)
    f += 0.03 * torch.randn(f.shape, generator=gen, device=cuda, dtype=torch.float64)
    x = torch.randn(batch, 12 * nside * nside, generator=gen, device=cuda)
    x[0], x[-1] = f[0].float(), f[1].float()
    a = on_tensor_cores(plan, plan.forward, x)[[0, -1]][..., spot].cpu().numpy()
    exact = O.sht_spot(f.cpu().numpy(), nside, L, L, spot, nodes="exact")
    assert rel(a, exact) < 1e-5
    z = torch.zeros(batch, L, L, dtype=torch.complex64, device=cuda)
    z[0], z[-1] = c[0].to(z.dtype), c[1].to(z.dtype)
    y = on_tensor_cores(plan, plan.inverse, z)[[0, -1]]
    assert rel(y, p64.inverse(c)) < 1e-5
    del p64, plan, x, z
    hpx.clear_plan_cache()
    torch.cuda.empty_cache()
