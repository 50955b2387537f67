"""The FFT passes wait, bounded, for the bulk copies of their inputs.  A wait
that gives up must not pass unseen: the group stores nothing and the failure
reaches the caller through srk_plan_sync, the plan's next operator, or
srk_noalloc_sync.  The wait is made to run out on a copy that is never issued
(a short limit, no copy in flight), and the context stays usable."""
import numpy as np
import pytest

import shrinkage_full_tests_b200 as srk
from oracle import oracle as O
from tests.gpu_util import dev, host, spectra
from tests.helpers import fields, kernel, rel_max_err

pytestmark = pytest.mark.gpu
N, KW, B = 128, 31, 2
E_, W_ = 15, 98


def setup(torch):
    Kx, Ky = kernel(KW)
    GX, GY = spectra(Kx, Ky, N, torch)
    f = np.stack(fields(N, B, 5))
    return Kx, Ky, GX, GY, f, dev(f, torch), torch.zeros((B, W_, W_), device="cuda")


@pytest.mark.parametrize("how", ["sync", "next_operator"])
def test_plan_reports_it_once(torch_cuda, how):
    Kx, Ky, GX, GY, f, E, R = setup(torch_cuda)
    plan = srk.SrkPlan(N, W_, E_, 1.0, B)
    assert plan.copy_wait_selftest(1 << 10) == srk.SRK_OK  # nobody went on
    with pytest.raises(srk.SrkError) as ei:
        if how == "sync":
            plan.sync()
        else:
            srk.srkTrainingForward(E, E, GX, GY, N, W_, E_, 1.0, B, None, R, plan)
    assert ei.value.status == srk.SRK_ERR_TIMEOUT and "site 20" in str(ei.value)
    srk.srkTrainingForward(E, E, GX, GY, N, W_, E_, 1.0, B, None, R, plan)
    plan.sync()
    assert rel_max_err(host(R)[1], O.forward(f[1], f[1], Kx, Ky, E_, 1.0)) < 1e-3
    plan.destroy()


def test_the_forward_without_allocation_reports_it_once(torch_cuda):
    torch = torch_cuda
    Kx, Ky, GX, GY, f, E, R = setup(torch)
    L = srk.lib()
    s = torch.cuda.current_stream().cuda_stream
    assert L.srk_noalloc_sync(s) == srk.SRK_OK
    assert L.srk_debug_copy_wait_selftest(None, 1 << 10, s) == srk.SRK_OK
    assert L.srk_noalloc_sync(s) == srk.SRK_ERR_TIMEOUT
    st = L.srk_training_forward_noalloc(E.data_ptr(), E.data_ptr(), GX.data_ptr(), GY.data_ptr(), N, W_, E_, 1.0, B, s,
                                        R.data_ptr())
    assert st == srk.SRK_OK and L.srk_noalloc_sync(s) == srk.SRK_OK
    assert rel_max_err(host(R)[0], O.forward(f[0], f[0], Kx, Ky, E_, 1.0)) < 1e-3
