"""The bounds-checked build over every contraction a call can take: the tiled FP32
kernels, the FP64 analysis of many maps, the tensor cores on the fly, with full and
with packed operand rows, and the FP32 spin-1 kernels (test_bounds_gpu.py's batches
are small enough for the direct kernels).  The stage counters say which ran.

Tolerances as there: FP64 1e-10, else 3e-5 (rel-L2, float64 oracle).
"""

import ctypes
import os

import numpy as np
import pytest
import torch

from cuhpx_b200 import _lib
from cuhpx_b200.build import VARIANTS
from oracle import hpx_oracle as O
from test_bounds_gpu import BF16X3, F16X3, FP32, FP64, HPX_ERR_BOUNDS, HPX_OK, call, make_plan, rel

pytestmark = pytest.mark.gpu

OTF = 1
EXT_SPEC, EXT_ALMT = 2, 7  # hpx_common.cuh HpxExtent


@pytest.fixture(scope="module")
def lib(cuda):
    path = VARIANTS["bounds"][1]
    if not os.path.exists(path):
        pytest.skip("checker build libhpx_b200_bounds.so not built (cuhpx_b200.build.build_variant)")
    return _lib.load_path(path)


def stages(lib, plan):
    arr, n = (_lib.HpxStageStat * 16)(), ctypes.c_int()
    assert lib.hpx_stats_read(plan, arr, 16, ctypes.byref(n)) == HPX_OK
    return {arr[i].name.decode() for i in range(n.value) if arr[i].launches}


# (nside, L, M, precision, flags, batch, stages of the analysis, of the synthesis)
CASES = [
    (16, 129, 33, FP32, 0, 70, {"fold"}, set()),                        # tiled analysis, then a direct chunk
    (128, 131, 20, FP32, 0, 60, {"fold"}, {"alm_to_columns"}),          # tiled both ways
    (256, 70, 9, FP32, 0, 64, {"fold"}, {"alm_to_columns"}),            # one block of degrees, second half empty
    (8, 17, 17, FP64, 0, 60, {"fold"}, set()),                          # FP64 analysis of many maps
    (16, 33, 31, F16X3, OTF, 20, {"fold", "columns_to_alm"}, {"alm_to_columns"}),
    (32, 63, 63, BF16X3, OTF, 13, {"fold", "columns_to_alm"}, {"alm_to_columns"}),
    (128, 131, 90, F16X3, 0, 12, {"fold", "columns_to_alm"}, {"alm_to_columns"}),   # packed rows
    (128, 66, 67, BF16X3, 0, 16, {"fold", "columns_to_alm"}, {"alm_to_columns"}),
    (64, 65, 65, F16X3, 0, 17, {"fold", "columns_to_alm"}, {"alm_to_columns"}),     # full rows
]


@pytest.mark.parametrize("nside,L,M,prec,flags,batch,fwd,inv", CASES)
def test_no_access_outside_buffers(lib, cuda, nside, L, M, prec, flags, batch, fwd, inv):
    plan = make_plan(lib, nside, L, M, prec, flags)
    try:
        dt, tol = (torch.float64, 1e-10) if prec == FP64 else (torch.float32, 3e-5)
        rng = np.random.default_rng(nside + L + prec)
        f = rng.standard_normal((batch, 12 * nside * nside))
        pick = [0, batch - 1]
        x = torch.from_numpy(f).to(cuda, dt)
        a = torch.zeros(batch, L, M, 2, dtype=dt, device=cuda)
        g = torch.zeros_like(x)
        assert lib.hpx_stats_enable(plan, 1) == HPX_OK
        assert call(lib, lib.hpx_sht_forward, plan, x, a, batch) == HPX_OK
        ran = stages(lib, plan)
        assert fwd <= ran and ("columns_to_alm" in ran) == ("columns_to_alm" in fwd)
        got = torch.view_as_complex(a).cpu().numpy()[pick]
        assert rel(got, O.sht(f[pick], nside, L, M)) < tol
        lib.hpx_stats_enable(plan, 1)
        assert call(lib, lib.hpx_sht_inverse, plan, a, g, batch) == HPX_OK
        ran = stages(lib, plan)
        assert inv <= ran and ("alm_to_columns" in ran) == ("alm_to_columns" in inv)
        lib.hpx_stats_enable(plan, 0)
        assert rel(g.cpu().numpy()[pick], O.isht(got.astype(np.complex128), nside)) < tol
        assert call(lib, lib.hpx_sht_forward_refined, plan, x, a, batch, ctypes.c_int32(1)) == HPX_OK
        assert call(lib, lib.hpx_sht_forward_adjoint, plan, a, g, batch) == HPX_OK
        assert call(lib, lib.hpx_sht_inverse_adjoint, plan, x, a, batch) == HPX_OK
    finally:
        lib.hpx_plan_destroy(plan)


@pytest.mark.parametrize("batch", [1, 3, 33])
def test_spin1_fp32_no_access_outside_buffers(lib, cuda, batch):
    from oracle import vector_oracle as V

    nside, L, M = 8, 17, 13
    plan = make_plan(lib, nside, L + 1, M + 1, FP32)
    try:
        f = np.random.default_rng(batch).standard_normal((batch, 2, 12 * nside * nside))
        x = torch.from_numpy(f).float().to(cuda)
        a = torch.zeros(batch, 2, L, M, 2, device=cuda)
        g = torch.zeros_like(x)
        for fn, src, dst in ((lib.hpx_vsht_forward, x, a), (lib.hpx_vsht_inverse, a, g),
                             (lib.hpx_vsht_forward_adjoint, a, g), (lib.hpx_vsht_inverse_adjoint, x, a)):
            assert call(lib, fn, plan, src, dst, batch, ctypes.c_int32(1)) == HPX_OK
            if fn is lib.hpx_vsht_forward:
                assert rel(torch.view_as_complex(a).cpu().numpy()[-1:], V.vsht(f[-1:], nside, L, M)) < 3e-5
    finally:
        lib.hpx_plan_destroy(plan)


@pytest.mark.parametrize("ext,fn", [(EXT_SPEC, "hpx_sht_forward"), (EXT_ALMT, "hpx_sht_inverse")])
def test_shrunk_extent_of_the_tiled_kernels_is_reported(lib, cuda, monkeypatch, ext, fn):
    """The last element of the tiled kernels' operand is skipped and reported."""
    nside, L, M, batch = 128, 131, 20, 64
    plan = make_plan(lib, nside, L, M, FP32)
    try:
        x = torch.randn(batch, 12 * nside * nside, device=cuda)
        a = torch.zeros(batch, L, M, 2, device=cuda)
        src, dst = (x, a) if fn == "hpx_sht_forward" else (a, x)
        monkeypatch.setenv("HPX_TEST_SHRINK_EXTENT", str(ext))
        assert call(lib, getattr(lib, fn), plan, src, dst, batch) == HPX_ERR_BOUNDS
        monkeypatch.delenv("HPX_TEST_SHRINK_EXTENT")
        assert call(lib, getattr(lib, fn), plan, src, dst, batch) == HPX_OK
    finally:
        lib.hpx_plan_destroy(plan)
