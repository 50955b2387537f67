"""The engine's passes where their routes change: bulk column copies or
plain loads (N and the tile origins in 16-byte pieces, aligned images),
paired or single stores (parity of N and the erosion), tiles cut by the image
edge, every tile size, pointers off every alignment.  All operators against
the FP64 oracle.

Tolerance: two transforms along each axis, at most 4 log2(512) = 36 radix-2
levels of three roundings each, 36 * 3 * 2^-24 = 6.5e-6 of the result's
scale; a factor 3 between the largest and the typical value: 2e-5."""
import numpy as np
import pytest

import shrinkage_full_tests_b200 as srk
from oracle import oracle as O
from tests.helpers import fields, rel_max_err
from tests.gpu_util import dev, host

pytestmark = pytest.mark.gpu
TOL = 2e-5


def shifted(a, torch, shift):
    """a on the device, its first element `shift` elements past an allocation."""
    a = np.ascontiguousarray(a, np.float32)
    buf = torch.full((a.size + shift,), float("nan"), device="cuda")
    buf[shift:].copy_(torch.from_numpy(a.reshape(-1)))
    return buf[shift:].view(a.shape)


@pytest.mark.parametrize("shift", [0, 1, 2])
@pytest.mark.parametrize("tile,N,KW", [
    (128, 122, 3), (128, 124, 9), (128, 301, 15), (128, 302, 17),
    (256, 254, 31), (256, 256, 61), (256, 450, 61), (256, 463, 33),
    (512, 512, 31), (512, 510, 61), (512, 516, 63), (512, 905, 61), (512, 908, 61)])
def test_every_route(torch_cuda, tile, N, KW, shift):
    torch = torch_cuda
    e = (KW - 1) // 2
    W = N - 2 * e
    rng = np.random.default_rng(1000 * N + KW)
    Kx, Ky = (rng.standard_normal((KW, KW)).astype(np.float32) / KW for _ in range(2))
    f, g = fields(N, 2, 400 + N)
    df, dg = [(1e-2 * rng.standard_normal((N, N))).astype(np.float32) for _ in range(2)]
    v, dv = [rng.standard_normal((W, W)).astype(np.float32) for _ in range(2)]
    plan = srk.SrkPlan(N, W, e, 1.0, 1, spectra_M=tile, tile_M=tile)
    plan.set_kernel(dev(Kx, torch), dev(Ky, torch))
    t = {k: shifted(a, torch, shift) for k, a in dict(f=f, g=g, df=df, dg=dg, v=v, dv=dv).items()}

    def out(n):
        return shifted(np.full((n, n), np.nan), torch, shift)

    R, ux, uy, dh = out(W), out(W), out(W), out(W)
    srk.srkForwardOaS(t["g"], t["f"], None, None, N, W, e, 1.0, None, R, plan, ux, uy)
    srk.shrinkageTangentOaS(t["f"], t["g"], t["df"], t["dg"], None, None, N, W, e, 1.0, None, dh, plan)
    dI, dE, lf, lg = out(N), out(N), out(N), out(N)
    srk.adjointSRK(t["v"], ux, uy, t["f"], None, None, N, W, e, 1.0, None, dI, dE, plan)
    srk.shrinkageTangentAdjointOaS(t["f"], t["g"], t["df"], t["dg"], t["v"], t["dv"], None, None, N, W, e, 1.0, None,
                                   lf, lg, plan)
    plan.sync()
    oR, oux, ouy = O.forward(g, f, Kx, Ky, e, 1.0, return_u=True)
    of, og = O.tangent_adjoint(f, g, df, dg, v, dv, Kx, Ky, e, 1.0)
    for name, x, ref in [("R", R, oR), ("ux", ux, oux), ("uy", uy, ouy),
                         ("dh", dh, O.tangent(f, g, df, dg, Kx, Ky, e, 1.0)),
                         ("dLdI", dI, O.adj_wrt_I(v, host(ux), host(uy), N, e)),
                         ("dLdE", dE, O.adj_wrt_E(v, f, Kx, Ky, e, 1.0)),
                         ("dLam_f", lf, of), ("dLam_g", lg, og)]:
        assert rel_max_err(host(x), ref) < TOL, name


@pytest.mark.parametrize("dt", ["float16", "bfloat16"])
@pytest.mark.parametrize("tile,N,KW,B", [(128, 200, 15, 3), (256, 252, 31, 2), (256, 250, 61, 3), (512, 512, 61, 3),
                                         (512, 517, 31, 2)])
def test_storage_types_equal_the_fp32_routes(torch_cuda, tile, N, KW, B, dt):
    """2-byte storage only changes loads and stores: the result is the FP32
    plan's on the same (rounded) images, rounded once."""
    torch = torch_cuda
    e = (KW - 1) // 2
    W = N - 2 * e
    rng = np.random.default_rng(N + KW)
    K = [dev(rng.standard_normal((KW, KW)).astype(np.float32) / KW, torch) for _ in range(2)]
    T = getattr(torch, dt)
    f, g = (dev(np.stack(fields(N, B, s + N)), torch).to(T) for s in (600, 700))
    v = dev(rng.standard_normal((B, W, W)).astype(np.float32), torch).to(T)
    res = []
    for sdt, S in ((srk.SRK_F32, torch.float32), ({"float16": srk.SRK_F16, "bfloat16": srk.SRK_BF16}[dt], T)):
        plan = srk.SrkPlan(N, W, e, 1.0, B, spectra_M=tile, dtype=sdt, tile_M=tile)
        plan.set_kernel(*K)
        a = [x.to(S).contiguous() for x in (f, g, v)]
        h = torch.full((B, W, W), float("nan"), device="cuda", dtype=S)
        df, dg = (torch.full((B, N, N), float("nan"), device="cuda", dtype=S) for _ in range(2))
        srk.forward(a[0], a[1], B, h, plan)
        srk.vjp(a[2], a[0], a[1], B, df, dg, plan)
        plan.sync()
        res.append([x.to(T) for x in (h, df, dg)])
    for x, y in zip(*res):
        assert torch.equal(x, y)


@pytest.mark.parametrize("conv", [srk.SRK_ADJ_REFERENCE, srk.SRK_ADJ_TRUE])
@pytest.mark.parametrize("tile,N,KW", [(128, 128, 1), (128, 128, 3), (128, 101, 33), (128, 128, 113), (256, 256, 61),
                                       (256, 255, 31), (256, 200, 121), (512, 512, 121), (512, 509, 31)])
def test_adjoint_of_an_image_within_one_tile(torch_cuda, tile, N, KW, conv):
    """N <= tile: the adjoint with respect to g runs as one circular tile per
    image, up to N = tile, where the outputs fill the transform; against the
    oracle and against the overlapping tiles of a ragged call."""
    torch = torch_cuda
    e = (KW - 1) // 2
    W = N - 2 * e
    rng = np.random.default_rng(N + KW)
    Kx, Ky = (rng.standard_normal((KW, KW)).astype(np.float32) / KW for _ in range(2))
    B = 3
    f = np.stack(fields(N, B, 50 + N))
    v = rng.standard_normal((B, W, W)).astype(np.float32)
    plan = srk.SrkPlan(N, W, e, 1.0, B, spectra_M=tile, tile_M=tile)
    plan.set_adj_convention(conv)
    plan.set_kernel(dev(Kx, torch), dev(Ky, torch))
    fd, vd = dev(f, torch), dev(v, torch)
    u = torch.zeros((B, W, W), device="cuda")
    dI, dE, rE = (torch.full((B, N, N), float("nan"), device="cuda") for _ in range(3))
    for b in range(B):
        srk.adjointSRK(vd[b], u[b], u[b], fd[b], None, None, N, W, e, 1.0, None, dI[b], dE[b], plan)
    srk.adjointSRKRagged(vd, u, u, fd, None, None, [N] * B, e, 1.0, None, dI, rE, plan)
    plan.sync()
    name = "true" if conv == srk.SRK_ADJ_TRUE else "reference"
    for b in range(B):
        ref = O.adj_wrt_E(v[b], f[b], Kx, Ky, e, 1.0, name)
        assert rel_max_err(host(dE[b]), ref) < TOL
        assert rel_max_err(host(rE[b]), ref) < TOL


@pytest.mark.parametrize("tile,N,KW", [(128, 128, 15), (128, 304, 15), (128, 304, 33), (256, 256, 31), (256, 464, 31),
                                       (512, 512, 63), (512, 912, 31), (512, 912, 61)])
def test_aligned_forms(torch_cuda, tile, N, KW):
    """Images in 16-byte columns take kernels that know it and the parity of
    the first row (odd and even erosion); every operator, one tile and
    several, against the oracle, and 2-byte storage against FP32."""
    test_every_route(torch_cuda, tile, N, KW, 0)
    test_storage_types_equal_the_fp32_routes(torch_cuda, tile, N, KW, 2, "float16")


@pytest.mark.parametrize("tile,N,KW,B", [(128, 127, 3, 3), (128, 301, 33, 2), (256, 255, 61, 3), (512, 509, 121, 2),
                                         (512, 905, 31, 1)])
def test_odd_columns_of_two_byte_storage(torch_cuda, tile, N, KW, B):
    """Odd N, 2-byte storage: windows from the words around each column, whose
    alignment changes from column to column and from image to image."""
    for dt in ("float16", "bfloat16"):
        test_storage_types_equal_the_fp32_routes(torch_cuda, tile, N, KW, B, dt)
