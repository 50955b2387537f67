"""The tile a plan takes when none is pinned: the fastest for the forward,
unless the derivative operators' overlapping tiles make it far slower for them
than the tile of least work.  The results do not depend on it beyond rounding
(2e-5 of their scale, as the engine's other route tests)."""
import pytest

import shrinkage_full_tests_b200 as srk
from tests.gpu_util import dev
from tests.helpers import kernel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,KW,B,tile", [(256, 31, 1, 128), (333, 61, 8, 128), (257, 101, 4, 256), (333, 75, 16, 256),
                                         (512, 31, 1, 128), (512, 121, 64, 512), (4096, 61, 1, 512)])
def test_tile(torch_cuda, N, KW, B, tile):
    torch = torch_cuda
    e = (KW - 1) // 2
    W = N - 2 * e
    K = [dev(k, torch) for k in kernel(KW)]
    gen = torch.Generator(device="cuda").manual_seed(N)
    f, g = (torch.rand((B, N, N), device="cuda", generator=gen) for _ in range(2))
    v = torch.randn((B, W, W), device="cuda", generator=gen)
    outs = []
    for pinned in (0, 512):
        plan = srk.SrkPlan(N, W, e, 1.0, B, spectra_M=1024, tile_M=pinned)
        plan.set_kernel(*K)
        assert plan.info()["tile_M"] == (pinned or tile)
        a, b = (torch.full((B, N, N), float("nan"), device="cuda") for _ in range(2))
        srk.vjp(v, f, g, B, a, b, plan)
        plan.sync()
        plan.destroy()
        outs.append((a, b))
    for x, y in zip(*outs):
        assert (x - y).abs().max() <= 2e-5 * y.abs().max()
