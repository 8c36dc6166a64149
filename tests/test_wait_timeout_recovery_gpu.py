"""After a bounded wait has run out (test_wait_timeout_gpu.py), the product library's
tensor-core kernels, not only its direct ones, work on the same device."""

import numpy as np
import pytest
import torch

from oracle import hpx_oracle as O
from test_wait_timeout_gpu import F16X3, HPX_ERR_TIMEOUT, HPX_OK, L, NPIX, NSIDE, call, make_plan, waitlib  # noqa: F401

pytestmark = pytest.mark.gpu


def test_tensor_cores_usable_after_a_timeout(waitlib, cuda):  # noqa: F811
    import cuhpx_b200 as hpx

    stream = torch.cuda.current_stream(cuda).cuda_stream
    f = np.random.default_rng(5).standard_normal((17, NPIX))
    x = torch.from_numpy(f).float().to(cuda)
    alm = torch.zeros(17, L, L, 2, device=cuda)
    plan = make_plan(waitlib, F16X3)
    try:
        st, ws = call(waitlib, waitlib.hpx_sht_forward, plan, x, alm, 17, stream)
        assert st == HPX_OK and waitlib.hpx_plan_check(plan, stream) == HPX_ERR_TIMEOUT
    finally:
        waitlib.hpx_plan_destroy(plan)
    del ws
    plan = hpx.get_plan(NSIDE, L, L, "ring", "f16x3", 0)
    plan.stats_enable(True)
    got = plan.forward(x)
    ran = plan.stats_read()
    plan.stats_enable(False)
    assert ran["columns_to_alm"][0] == 1  # 17 maps: the tensor cores
    plan.check()
    ref = O.sht(f[:2], NSIDE, L, L)
    assert np.linalg.norm(got[:2].cpu().numpy() - ref) < 2e-6 * np.linalg.norm(ref)
