"""Scratch for ragged batches and slabs: they cover the adjoint geometry by
overlapping tiles even where a whole image is one tile of its own, so a plan
must hold the work tiles of one image's general tiling at once."""
import numpy as np
import pytest

import shrinkage_full_tests_b200 as srk
from oracle import oracle as O
from tests.gpu_util import dev, host
from tests.helpers import fields, kernel, rel_max_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile,N,KW", [(128, 100, 31), (256, 256, 61), (512, 512, 61)])
def test_one_image_in_one_chunk(torch_cuda, tile, N, KW):
    torch = torch_cuda
    e = (KW - 1) // 2
    W, S = N - 2 * e, tile - 2 * e
    Kx, Ky = kernel(KW)
    plan = srk.SrkPlan(N, W, e, 1.0, 1, spectra_M=1024, tile_M=tile)
    plan.set_kernel(dev(Kx, torch), dev(Ky, torch))
    plan.set_adj_convention(srk.SRK_ADJ_TRUE)
    tiles = -(-N // S)
    assert plan.info()["chunk_wt"] == max(1, (tiles * tiles + 1) // 2)
    f, g = fields(N, 2, N)
    v = np.random.default_rng(N).standard_normal((W, W)).astype(np.float32)
    _, ux, uy = O.forward(g, f, Kx, Ky, e, 1.0, return_u=True)
    a, b = (torch.full((N * N,), float("nan"), device="cuda") for _ in range(2))
    args = [dev(np.ascontiguousarray(x, np.float32).reshape(-1), torch) for x in (v, ux, uy, f)]
    srk.adjointSRKRagged(*args, None, None, [N], e, 1.0, None, a, b, plan)
    assert plan.info()["last_launches"] == 3
    plan.sync()
    want = O.adj_wrt_E(v, f, Kx, Ky, e, 1.0, "true")
    assert rel_max_err(host(b).reshape(N, N), want) < 2e-5
    plan.destroy()
