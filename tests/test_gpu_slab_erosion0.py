"""Column slabs at erosion 0: the central differences at a slab's first and
last column reach one column past it (include/srk_b200.h).  Slabs from buffers
that hold those columns between NaN columns, against the whole-image call: the
tiles and their pairs are the same per column, so to rounding of the transform
(2e-5 of the result's scale, as the engine's other route tests)."""
import pytest

import shrinkage_full_tests_b200 as srk
from shrinkage_full_tests_b200.shard import adjoint_need, forward_need

pytestmark = pytest.mark.gpu


def test_slabs_equal_the_whole_image(torch_cuda):
    torch = torch_cuda
    N, S = 300, 128
    gen = torch.Generator(device="cuda").manual_seed(3)
    plan = srk.SrkPlan(N, N, 0, 1.0, 1, spectra_M=1024, tile_M=S)
    plan.set_adj_convention(srk.SRK_ADJ_TRUE)
    plan.set_kernel(torch.full((1, 1), 0.75, device="cuda"), torch.full((1, 1), -0.5, device="cuda"))
    f, g, df, dg, v, ux, uy = (torch.randn((N, N), device="cuda", generator=gen) for _ in range(7))
    whole = [torch.zeros((N, N), device="cuda") for _ in range(4)]
    srk.srkForwardOaS(g, f, None, None, N, N, 0, 1.0, None, whole[0], plan)
    srk.shrinkageTangentOaS(f, g, df, dg, None, None, N, N, 0, 1.0, None, whole[1], plan)
    srk.adjointSRK(v, ux, uy, f, None, None, N, N, 0, 1.0, None, whole[2], whole[3], plan)
    got = [torch.full((N, N), float("nan"), device="cuda") for _ in range(4)]

    def halo(x, need, c0):
        buf = torch.full((need[1] - need[0] + 8, N), float("nan"), device="cuda")
        buf[4:4 + need[1] - need[0]] = x[need[0]:need[1]]
        return buf[4 + c0 - need[0]:]

    for c0, c1 in ((0, 128), (128, 256), (256, 300)):
        hf, hg, hdf, hdg = (halo(x, forward_need(c0, c1, N, 0), c0) for x in (f, g, df, dg))
        srk.srkForwardOaSSlab(hg, hf, None, None, N, 0, 1.0, c0, c1, None, got[0][c0:], plan)
        srk.shrinkageTangentOaSSlab(hf, hg, hdf, hdg, None, None, N, 0, 1.0, c0, c1, None, got[1][c0:], plan)
        hv = [halo(x, adjoint_need(c0, c1, N, 0), c0) for x in (v, ux, uy)]
        hI = halo(f, (max(c0 - 1, 0), min(c1 + 1, N)), c0)
        srk.adjointSRKSlab(*hv, hI, None, None, N, 0, 1.0, c0, c1, None, got[2][c0:], got[3][c0:], plan)
    plan.sync()
    for a, b in zip(whole, got):
        assert torch.isfinite(b).all() and (a - b).abs().max() <= 2e-5 * a.abs().max()
    plan.destroy()
