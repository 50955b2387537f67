"""The persistent schedule's hand-over of S1 and S2 between blocks of one
launch: ordinary stores by one block, bulk copies (async proxy) by another.
The order cannot be shown by running (stale data is a race), so the CPU test
reads the kernel's text for the fences on both sides of the counters; the GPU
test runs a short ring many times over with inputs that change between calls
and compares with the three-pass schedule, bit for bit."""
import os
import re

import numpy as np
import pytest

import shrinkage_full_tests_b200 as srk
from tests.helpers import kernel
from tests.gpu_util import dev

CSRC = os.path.join(os.path.dirname(srk.__file__), "csrc")


def test_scratch_is_fenced_for_the_async_proxy():
    text = open(os.path.join(CSRC, "engine.cuh")).read()
    body = re.sub(r"//.*", "", text[text.index("\nk_persist("):text.index("k_wait_selftest")])
    fence = "tc::fence_async_global();"
    order = [body.index("wait_geq"), body.index("if (!s_t[1]"), body.index(fence), body.index("phase1<"),
             body.index("phase2<"), body.index("phase3<"), body.rindex(fence), body.index("__threadfence();")]
    assert order == sorted(order) and body.count(fence) == 2
    assert "fence.proxy.async.global" in open(os.path.join(CSRC, "tc.cuh")).read()


@pytest.mark.gpu
@pytest.mark.parametrize("tile,N,KW,B", [(128, 200, 31, 40), (256, 256, 31, 90), (512, 500, 61, 60)])
def test_short_ring_many_calls(torch_cuda, tile, N, KW, B):
    torch = torch_cuda
    e = (KW - 1) // 2
    W = N - 2 * e
    Kx, Ky = (dev(k, torch) for k in kernel(KW))
    gen = torch.Generator(device="cuda").manual_seed(N)
    plans = []
    for sch in (srk.SRK_SCHEDULE_PERSISTENT, srk.SRK_SCHEDULE_THREE_PASS):
        p = srk.SrkPlan(N, W, e, 1.0, B, spectra_M=1024, tile_M=tile)
        p.set_kernel(Kx, Ky)
        p.set_schedule(sch)
        plans.append(p)
    plans[0].set_persistent(lag=2)
    for _ in range(4):
        f, g, df, dg = (torch.rand((B, N, N), device="cuda", generator=gen) for _ in range(4))
        v = torch.randn((B, W, W), device="cuda", generator=gen)
        outs = []
        for p in plans:
            h, dh = (torch.full((B, W, W), float("nan"), device="cuda") for _ in range(2))
            a, b = (torch.full((B, N, N), float("nan"), device="cuda") for _ in range(2))
            srk.forward(f, g, B, h, p)
            srk.vjp(v, f, g, B, a, b, p)
            srk.jvp(f, g, df, dg, B, dh, p)
            p.sync()
            outs.append((h, a, b, dh))
        for x, y in zip(*outs):
            assert torch.isfinite(x).all() and torch.equal(x, y)
    for p in plans:
        p.destroy()
