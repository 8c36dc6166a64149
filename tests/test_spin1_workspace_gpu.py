"""Spin-1 calls on plans whose passes hold few scalar maps stay inside the
workspace that the plan asks for: a vector map is two scalar maps, so a plan with
``batch_chunk = 1`` works on more maps than a pass of scalar transforms does.

Every call gets exactly ``hpx_workspace_size`` bytes, followed by a guard larger
than one map's ring spectra that must come back untouched.  Tolerances as for
the other spin-1 tests: FP64 1e-11, FP32 1e-5 (rel-L2, float64 oracle).
"""

import ctypes

import numpy as np
import pytest
import torch

from cuhpx_b200 import _lib
from oracle import vector_oracle as V

pytestmark = pytest.mark.gpu

GUARD, MARK = 1 << 20, 0x5A


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("prec,dtype,tol", [(0, torch.float32, 1e-5), (1, torch.float64, 1e-11)])
@pytest.mark.parametrize("chunk", [1, 2, 3])
@pytest.mark.parametrize("nside,L,M", [(1, 2, 1), (8, 17, 13), (16, 33, 33)])
def test_workspace_of_small_chunks(cuda, nside, L, M, chunk, prec, dtype, tol):
    lib = _lib.load()
    d = _lib.HpxDesc()
    d.nside, d.lmax, d.mmax, d.precision = nside, L + 1, M + 1, prec
    d.refine_iters, d.batch_chunk, d.device, d.flags = 0, chunk, 0, 0
    plan = ctypes.c_void_p()
    _lib.check(lib.hpx_plan_create(ctypes.byref(d), ctypes.byref(plan)))
    try:
        B = 3
        need = ctypes.c_size_t()
        _lib.check(lib.hpx_workspace_size(plan, B, ctypes.byref(need)), plan)
        buf = torch.full((need.value + 256 + GUARD,), MARK, dtype=torch.uint8, device=cuda)
        off = -buf.data_ptr() % 256
        ws, guard = buf.data_ptr() + off, buf[off + need.value:]
        stream = torch.cuda.current_stream(cuda).cuda_stream
        rng = np.random.default_rng(nside + chunk)
        f = rng.standard_normal((B, 2, 12 * nside * nside))
        x = torch.from_numpy(f).to(cuda, dtype)
        a = torch.zeros(B, 2, L, M, 2, dtype=dtype, device=cuda)
        y = torch.zeros_like(x)
        ref = V.vsht(f, nside, L, M, "none", csphase=False)

        def call(fn, src, dst):
            _lib.check(fn(plan, src.data_ptr(), dst.data_ptr(), B, 0, ws, need.value, stream), plan)
            assert bool((guard == MARK).all())

        call(lib.hpx_vsht_forward, x, a)
        got = torch.view_as_complex(a).cpu().numpy()
        assert rel(got, ref) < tol
        call(lib.hpx_vsht_inverse, a, y)
        assert rel(y.cpu().numpy(), V.visht(got.astype(np.complex128), nside, csphase=False)) < tol
        call(lib.hpx_vsht_forward_adjoint, a, y)
        call(lib.hpx_vsht_inverse_adjoint, x, a)
    finally:
        lib.hpx_plan_destroy(plan)
