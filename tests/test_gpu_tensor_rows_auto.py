"""SRK_SCHEDULE_TENSOR_ROWS (tile 512) on plans whose tile was left to the
library: the model picks smaller tiles for small batches, which must not turn
into a refusal where the 512 tile needs the least work.  FP16 storage: within
rel 1e-2 of the FP64 oracle on the same rounded inputs."""
import numpy as np
import pytest

import shrinkage_full_tests_b200 as srk
from oracle import oracle as O
from tests.gpu_util import dev, host, spectra
from tests.helpers import fields, kernel, rel_max_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bind", ["spectra", "kernel"])
@pytest.mark.parametrize("order", ["kernel_first", "schedule_first"])
def test_small_batch_moves_to_the_schedules_tile(torch_cuda, bind, order):
    torch = torch_cuda
    N, KW, B = 512, 31, 1
    e = (KW - 1) // 2
    W = N - 2 * e
    Kx, Ky = kernel(KW)
    plan = srk.SrkPlan(N, W, e, 1.0, B, spectra_M=N, dtype=srk.SRK_F16)
    assert plan.info()["tile_M"] < 512  # the latency of one image decides

    def kern():
        if bind == "kernel":
            plan.set_kernel(dev(Kx, torch), dev(Ky, torch))
        else:
            plan.import_spectra(*spectra(Kx, Ky, N, torch))

    if order == "kernel_first":
        kern()
    f, g = (torch.from_numpy(x).cuda().half() for x in fields(N, 2, 9))
    v = torch.randn((W, W), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1)).half()
    a = torch.zeros((N, N), device="cuda", dtype=torch.float16)
    b = torch.zeros_like(a)
    if order == "kernel_first":  # the former tile has run
        srk.forward(f, g, 1, torch.zeros((W, W), device="cuda", dtype=torch.float16), plan)
    plan.set_schedule(srk.SRK_SCHEDULE_TENSOR_ROWS)
    assert plan.info()["tile_M"] == 512 and plan.info()["tile_stride"] == 512 - 2 * e
    if order == "schedule_first":
        kern()
    R = torch.zeros((W, W), device="cuda", dtype=torch.float16)
    srk.forward(f, g, 1, R, plan)
    assert plan.info()["last_launches"] == 4  # the tensor-row pipeline
    srk.vjp(v, f, g, 1, a, b, plan)
    plan.sync()
    fh, gh, vh = (host(x).astype(np.float32) for x in (f, g, v))
    assert rel_max_err(host(R).astype(np.float32), O.forward(gh, fh, Kx, Ky, e, 1.0)) < 1e-2
    assert rel_max_err(host(b).astype(np.float32), O.adj_wrt_E(vh, fh, Kx, Ky, e, 1.0, "true")) < 1e-2
    plan.destroy()


def test_what_was_refused_stays_refused(torch_cuda):
    for kw in (dict(tile_M=128), dict(tile_M=256)):
        plan = srk.SrkPlan(512, 482, 15, 1.0, 1, dtype=srk.SRK_F16, **kw)
        with pytest.raises(srk.SrkError) as ei:
            plan.set_schedule(srk.SRK_SCHEDULE_TENSOR_ROWS)
        assert ei.value.status == srk.SRK_ERR_UNSUPPORTED and plan.info()["tile_M"] == kw["tile_M"]
        plan.destroy()
    plan = srk.SrkPlan(1024, 994, 15, 1.0, 1, dtype=srk.SRK_F16)  # 256 needs less work than 512
    with pytest.raises(srk.SrkError) as ei:
        plan.set_schedule(srk.SRK_SCHEDULE_TENSOR_ROWS)
    assert ei.value.status == srk.SRK_ERR_UNSUPPORTED
    plan.destroy()
