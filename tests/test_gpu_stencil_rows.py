"""The stencil of dL/df on small images: strips of 32 rows per warp where the
window is odd (single rows), pairs of rows where it is even, marches of four
columns from u and v.  Sizes around the blocks' 128 and 256 rows, both parities
of the erosion, against the FP64 oracle.

Tolerance: an output is half the sum of two differences of products u * v, five
roundings deep: 5 * 2^-24 of the four products, at most 2 max|u v| after the
half, so 10 * 2^-24 max|u v|."""
import numpy as np
import pytest

import shrinkage_full_tests_b200 as srk
from oracle import oracle as O
from tests.gpu_util import dev, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("e", [1, 2, 15])
@pytest.mark.parametrize("N", [35, 63, 64, 127, 128, 129, 255, 257, 511])
def test_small_images(torch_cuda, N, e):
    torch = torch_cuda
    W = N - 2 * e
    rng = np.random.default_rng(N * 100 + e)
    v, ux, uy = (rng.standard_normal((W, W)).astype(np.float32) for _ in range(3))
    f = rng.standard_normal((N, N)).astype(np.float32)
    plan = srk.SrkPlan(N, W, e, 1.0, 1, spectra_M=1024)
    plan.set_kernel(*(torch.zeros((2 * e + 1, 2 * e + 1), device="cuda") for _ in range(2)))
    a, b = (torch.full((N, N), float("nan"), device="cuda") for _ in range(2))
    srk.adjointSRK(*(dev(x, torch) for x in (v, ux, uy, f)), None, None, N, W, e, 1.0, None, a, b, plan)
    plan.sync()
    scale = max(np.abs(ux * v).max(), np.abs(uy * v).max())
    assert np.abs(host(a) - O.adj_wrt_I(*(x.astype(np.float64) for x in (v, ux, uy)), N, e)).max() <= 10 * 2.0 ** -24 * scale
    plan.destroy()
