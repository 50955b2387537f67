"""Calls that read what the call before them wrote, without a synchronisation
between: the kernels of a call start while their predecessor still runs and
wait inside for its results.  The CPU test reads the sources: a load of an
operand must be an ordinary one that the compiler keeps behind that wait.  The
GPU test chains calls whose inputs change and compares with the same calls run
one at a time, bit for bit."""
import os
import re

import pytest

import shrinkage_full_tests_b200 as srk
from tests.helpers import kernel
from tests.gpu_util import dev

CSRC = os.path.join(os.path.dirname(srk.__file__), "csrc")


def test_operand_loads_stay_behind_the_wait():
    text = re.sub(r"//.*", "", open(os.path.join(CSRC, "engine.cuh")).read())
    assert "ld.global.nc" not in text
    loads = re.findall(r"\bldp(?:16|32|64)\(const void\* p, bool on\) \{.*?return v;", text, re.S)
    assert len(loads) == 3
    for body in loads:
        assert "asm volatile(" in body and '"memory"' in body and "@q ld.global.b" in body
    # the read-only path: the twiddle table, and the storage-typed load of the
    # direct kernel (an ordinary launch)
    assert re.findall(r"__ldg\([^)]*\)", text) == ["__ldg(p + i)"]
    assert "ldf<" not in re.sub(r"template <> .*", "", text) and "ldf(" not in text.replace("float ldf(const T* p", "")


@pytest.mark.gpu
@pytest.mark.parametrize("N,KW,dtype", [(256, 31, "f32"), (333, 31, "f32"), (1024, 61, "f16"), (777, 61, "bf16")])
def test_chained_calls(torch_cuda, N, KW, dtype):
    torch = torch_cuda
    e = (KW - 1) // 2
    W = N - 2 * e
    td = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}[dtype]
    sd = {"f32": srk.SRK_F32, "f16": srk.SRK_F16, "bf16": srk.SRK_BF16}[dtype]
    plan = srk.SrkPlan(N, W, e, 1.0, 1, spectra_M=1024, dtype=sd)
    plan.set_kernel(*(dev(k, torch) for k in kernel(KW)))
    gen = torch.Generator(device="cuda").manual_seed(N)
    ins = [[torch.rand((N, N), device="cuda", generator=gen).to(td) for _ in range(2)] for _ in range(6)]

    def run(sync):
        R, ux, uy = (torch.zeros((W, W), device="cuda", dtype=td) for _ in range(3))
        outs = []
        for f, g in ins:
            a, b, c, d = (torch.zeros((N, N), device="cuda", dtype=td) for _ in range(4))
            torch.cuda.synchronize()
            srk.srkForwardOaS(g, f, None, None, N, W, e, 1.0, None, R, plan, ux, uy)
            if sync:
                torch.cuda.synchronize()
            # R as the cotangent: v, ux and uy are all results of the call before
            srk.adjointSRK(R, ux, uy, f, None, None, N, W, e, 1.0, None, a, b, plan)
            if sync:
                torch.cuda.synchronize()
            srk.vjp(R, a, b, 1, c, d, plan)
            outs += [a, b, c, d]
        plan.sync()
        return outs

    want, got = run(True), run(False)
    for x, y in zip(want, got):
        assert torch.equal(x, y)
    plan.destroy()
