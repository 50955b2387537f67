"""Workloads of the resist-shrinkage operator, as programs call it.

Each case is one use of a public entry point of shrinkage_full_tests_b200 at
the sizes its configurations, tests and benchmark run: single images (the
latency of one call), training batches, the save-for-backward step, the
derivative operators on large images, ragged batches of mixed N, FP32 and
FP16 / BF16 storage, even and odd N, tile sizes 128, 256 and 512.

Fields of a case: `op` (below), `N` (largest image of a ragged batch), `KW`
(kernel width, erosion = (KW - 1) / 2), `B` (images), `dtype` (storage),
`dx`, and `rows`: 1 pins the tensor-core schedule the autotuner picks for
FP16 storage at tile 512 (pinned, so that no timing decides what runs).

  train    srkTrainingForward (E = I, as the training driver calls it)
  oas      srkForwardOaS of one image, f != g
  step     forward + vjp, the save-for-backward training step
  adjoint  adjointSRK (given v, ux, uy)
  tangent  shrinkageTangentOaS
  tanadj   shrinkageTangentAdjointOaS
  ragged   adjointSRKRagged: sizes between N/8 and N

Inputs: Gaussian random fields of correlation length 8 px scaled to [0, 1],
N(0, 1) cotangents, directions of 1e-2 N(0, 1), the Bessel-K1 x Blackman
Green's tensor of 1/gamma = 30 nm.
"""
import math

import torch

import shrinkage_full_tests_b200 as srk

_TORCH = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
_SRK = {"f32": srk.SRK_F32, "f16": srk.SRK_F16, "bf16": srk.SRK_BF16}


def _case(name, op, N, KW, B=1, dtype="f32", dx=4.0, rows=0):
    return {"name": name, "op": op, "N": N, "KW": KW, "B": B, "dtype": dtype, "dx": dx, "rows": rows}


def listed():
    return [
        # one small image: a solver or a viewer calling the operator image by image
        _case("oas_n256_kw31", "oas", 256, 31),
        # calibration over a batch of small clips whose size is what the layout gave
        _case("train_b64_n333_kw31", "train", 333, 31, B=64),
        # the training batch at the smaller of the two configured image sizes
        _case("train_b3000_n256_kw61", "train", 256, 61, B=3000, dx=10.0),
        # the headline training batch
        _case("train_b5000_n512_kw121", "train", 512, 121, B=5000),
        # the same images stored as FP16, on the schedule tuned for that storage
        _case("train_b1000_n512_kw121_f16", "train", 512, 121, B=1000, dtype="f16", rows=1),
        # one optimiser step: forward and both gradients of a batch
        _case("step_b256_n512_kw61", "step", 512, 61, B=256),
        # gradients of one full-size image, the reference's adjoint contract
        _case("adjoint_n4096_kw61", "adjoint", 4096, 61),
        # the same at half storage and the widest kernel
        _case("adjoint_n2048_kw121_f16", "adjoint", 2048, 121, dtype="f16"),
        # directional derivative of a large image
        _case("tangent_n4096_kw121", "tangent", 4096, 121),
        # second-order product of a large image, narrow kernel, BF16 storage
        _case("tanadj_n4096_kw31_bf16", "tanadj", 4096, 31, dtype="bf16"),
        # a full-chip field in one call
        _case("oas_n16384_kw121", "oas", 16384, 121),
        # gradients of clips of many sizes in one call
        _case("ragged_b16_n4096_kw61", "ragged", 4096, 61, B=16),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: sizes spread over their logarithm, odd ones included;
    at most 2^28 image pixels in all (the largest listed case has 1.3e9)."""
    op = rng.choice(["train", "train", "oas", "step", "adjoint", "tangent", "tanadj", "ragged"])
    KW = rng.choice([31, 61, 121, 2 * rng.randint(7, 60) + 1])
    dtype = rng.choice(["f32", "f32", "f32", "f16", "bf16"])
    rows = 0
    if op in ("train", "step"):
        N = rng.choice([256, 512, _log_int(rng, max(160, KW + 40), 1100)])
        B = _log_int(rng, 1, max(1, min(4000, (1 << 27 if op == "step" else 1 << 28) // (N * N))))
        if op == "train" and N == 512 and dtype != "f32":
            rows = rng.randint(0, 1)
    elif op == "ragged":
        # the ragged entry points take float buffers
        N, B, dtype = _log_int(rng, 1024, 4096), rng.randint(2, 16), "f32"
    else:
        N, B = rng.choice([1024, 2048, 4096, 8192, _log_int(rng, 256, 8192)]), 1
    return {"op": op, "N": N, "KW": KW, "B": B, "dtype": dtype, "dx": rng.choice([4.0, 10.0]), "rows": rows}


# ---- inputs (from the seed alone) -------------------------------------------
def _green(KW, dx):
    """Gx, Gy (KW x KW, [column][row]) of 1/gamma = 30 nm, radial Blackman
    window of radius erosion * dx, centre 0; evaluated in 64 bits."""
    c, gamma = (KW - 1) // 2, 1.0 / 30.0
    x = (torch.arange(KW, dtype=torch.float64) - c) * dx
    X, Y = x[:, None].expand(KW, KW), x[None, :].expand(KW, KW)
    r = torch.sqrt(X * X + Y * Y)
    s = torch.clamp(r / (c * dx), max=1.0)
    w = 0.42 + 0.5 * torch.cos(math.pi * s) + 0.08 * torch.cos(2 * math.pi * s)
    w = torch.where(r <= c * dx, w, torch.zeros_like(w))
    rs = torch.where(r > 0, r, torch.ones_like(r))
    m = gamma / (2 * math.pi) * torch.special.modified_bessel_k1(gamma * rs) * w / rs
    m[c, c] = 0.0
    return (X * m).float().contiguous().cuda(), (Y * m).float().contiguous().cuda()


def _grf(gen, B, N, dtype, ell=8.0):
    """B Gaussian random fields [B][N][N], each scaled to [0, 1]."""
    out = torch.empty((B, N, N), device="cuda", dtype=_TORCH[dtype])
    k = torch.fft.fftfreq(N, device="cuda")
    h = torch.exp(-0.5 * (math.pi * ell) ** 2 * (k[:, None] ** 2 + k[None, : N // 2 + 1] ** 2))
    step = max(1, (1 << 26) // (N * N))
    for b in range(0, B, step):
        n = min(step, B - b)
        z = torch.randn((n, N, N), device="cuda", generator=gen)
        z = torch.fft.irfft2(torch.fft.rfft2(z) * h, s=(N, N))
        lo, hi = z.amin((1, 2), keepdim=True), z.amax((1, 2), keepdim=True)
        out[b : b + n] = (z - lo) / (hi - lo)
    return out


def _randn(gen, B, n, dtype, scale=1.0):
    out = torch.empty((B, n, n), device="cuda", dtype=_TORCH[dtype])
    step = max(1, (1 << 27) // (n * n))
    for b in range(0, B, step):
        m = min(step, B - b)
        out[b : b + m] = torch.randn((m, n, n), device="cuda", generator=gen) * scale
    return out


def _sizes(case):
    """Image sizes of a ragged batch, between N/8 (at least the kernel and a
    few pixels) and N; the largest is N."""
    lo = max(case["N"] // 8, case["KW"] + 9)
    return [case["N"]] + [lo + (i * 2654435761 % 4093) * (case["N"] - lo) // 4093 for i in range(1, case["B"])]


def _inputs(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    op, N, B, dt = case["op"], case["N"], case["B"], case["dtype"]
    W = N - case["KW"] + 1
    Kx, Ky = _green(case["KW"], case["dx"])
    d = {"Kx": Kx, "Ky": Ky}
    if op == "train":
        d["E"] = _grf(gen, B, N, dt)
    elif op == "oas":
        d["E"], d["I"] = _grf(gen, 1, N, dt)[0], _grf(gen, 1, N, dt)[0]
    elif op == "step":
        d["f"], d["g"], d["v"] = _grf(gen, B, N, dt), _grf(gen, B, N, dt), _randn(gen, B, W, dt)
    elif op == "ragged":
        for k in ("I", "v", "ux", "uy"):
            d[k] = []
        for n in _sizes(case):
            w = n - case["KW"] + 1
            E, I = _grf(gen, 1, n, dt)[0], _grf(gen, 1, n, dt)[0]
            ux, uy = _conv(E, Kx, Ky, case["dx"])
            d["I"].append(I)
            d["v"].append(_randn(gen, 1, w, dt)[0])
            d["ux"].append(ux.to(_TORCH[dt]))
            d["uy"].append(uy.to(_TORCH[dt]))
    else:
        f, g = _grf(gen, 1, N, dt)[0], _grf(gen, 1, N, dt)[0]
        if op == "adjoint":
            ux, uy = _conv(g, Kx, Ky, case["dx"])
            d["I"], d["v"] = f, _randn(gen, 1, W, dt)[0]
            d["ux"], d["uy"] = ux.to(_TORCH[dt]), uy.to(_TORCH[dt])
        else:
            d["f"], d["g"] = f, g
            d["df"], d["dg"] = _randn(gen, 1, N, dt, 1e-2)[0], _randn(gen, 1, N, dt, 1e-2)[0]
            if op == "tanadj":
                d["lam"], d["dlam"] = _randn(gen, 1, W, dt)[0], _randn(gen, 1, W, dt, 1e-2)[0]
    return d


# ---- what a program keeps, and one pass -------------------------------------
def prepare(case, seed):
    d = _inputs(case, seed)
    op, N, KW, B, dx, dt = case["op"], case["N"], case["KW"], case["B"], case["dx"], case["dtype"]
    e = (KW - 1) // 2
    W = N - 2 * e
    batch = B if op in ("train", "step") else 1
    # the training forward takes spectra at its own size; odd sizes (no such
    # spectrum) and the save-for-backward calls bind the kernel on the plan
    spatial = op == "step" or (op == "train" and N % 2 == 1)
    M = N if op == "train" and not spatial else 1024
    plan = srk.SrkPlan(N, W, e, dx, batch, spectra_M=M, dtype=_SRK[dt], tile_M=512 if case["rows"] else 0)
    if case["rows"]:
        plan.set_schedule(srk.SRK_SCHEDULE_TENSOR_ROWS)
    s = {"case": case, "plan": plan, "e": e, "W": W, "GX": None, "GY": None}
    if spatial:
        plan.set_kernel(d["Kx"], d["Ky"])
    else:
        for k, K in (("GX", d["Kx"]), ("GY", d["Ky"])):
            s[k] = torch.empty((M, M // 2 + 1), device="cuda", dtype=torch.complex64)
            srk.srkPrecomputeKernelFreq(K, KW, KW, M, s[k])
        plan.import_spectra(s["GX"], s["GY"])
    t = _TORCH[dt]
    if op == "ragged":
        s["Ns"] = _sizes(case)
        for k in ("I", "v", "ux", "uy"):
            s[k] = torch.cat([x.reshape(-1) for x in d[k]])
        s["out"] = [torch.empty(sum(n * n for n in s["Ns"]), device="cuda", dtype=t) for _ in range(2)]
    else:
        s.update({k: v for k, v in d.items() if k not in ("Kx", "Ky")})
        shape = {"train": [(B, W, W)], "oas": [(W, W)], "step": [(B, W, W), (B, N, N), (B, N, N)],
                 "adjoint": [(N, N)] * 2, "tangent": [(W, W)], "tanadj": [(N, N)] * 2}[op]
        s["out"] = [torch.empty(x, device="cuda", dtype=t) for x in shape]
    return s


def run(s):
    c, p, out, GX, GY = s["case"], s["plan"], s["out"], s["GX"], s["GY"]
    op, N, W, e, dx = c["op"], c["N"], s["W"], s["e"], c["dx"]
    if op == "train":
        srk.srkTrainingForward(s["E"], s["E"], GX, GY, N, W, e, dx, c["B"], None, out[0], p)
    elif op == "oas":
        srk.srkForwardOaS(s["E"], s["I"], GX, GY, N, W, e, dx, None, out[0], p)
    elif op == "step":
        srk.forward(s["f"], s["g"], c["B"], out[0], p)
        srk.vjp(s["v"], s["f"], s["g"], c["B"], out[1], out[2], p)
    elif op == "adjoint":
        srk.adjointSRK(s["v"], s["ux"], s["uy"], s["I"], GX, GY, N, W, e, dx, None, out[0], out[1], p)
    elif op == "tangent":
        srk.shrinkageTangentOaS(s["f"], s["g"], s["df"], s["dg"], GX, GY, N, W, e, dx, None, out[0], p)
    elif op == "tanadj":
        srk.shrinkageTangentAdjointOaS(s["f"], s["g"], s["df"], s["dg"], s["lam"], s["dlam"], GX, GY, N, W, e, dx,
                                       None, out[0], out[1], p)
    else:
        srk.adjointSRKRagged(s["v"], s["ux"], s["uy"], s["I"], GX, GY, s["Ns"], e, dx, None, out[0], out[1], p)
    return out


# ---- what a pass cannot do without ------------------------------------------
def work(case):
    """Bytes: every input read and every output written once.  Flops: one
    forward and two inverse real 2-D FFTs per convolved field (two forward
    and one inverse for the adjoint), 2.5 n log2 n each, and the pointwise
    products and differences."""
    op, KW = case["op"], case["KW"]
    sz = 4 if case["dtype"] == "f32" else 2
    Ns = _sizes(case) if op == "ragged" else [case["N"]] * case["B"]
    by = fl = 0.0
    for N in Ns:
        n, w = float(N * N), float((N - KW + 1) ** 2)
        fft = 2.5 * n * math.log2(n)
        nn, ww, ffts = {"train": (1, 1, 3), "oas": (2, 1, 3), "step": (4, 2, 9), "adjoint": (3, 3, 3),
                        "ragged": (3, 3, 3), "tangent": (4, 1, 6), "tanadj": (6, 2, 9)}[op]
        by += sz * (nn * n + ww * w)
        fl += ffts * (fft + 6 * n) + 8 * n
    return {"bytes": by, "flops": fl}


# ---- the same in 64 bits ----------------------------------------------------
def _spectra(Kx, Ky, P):
    """Spectra of the centred kernels on a P x P periodic grid."""
    KW = Kx.shape[0]
    c = (KW - 1) // 2
    out = []
    for K in (Kx, Ky):
        z = torch.zeros((P, P), device="cuda", dtype=torch.float64)
        z[:KW, :KW] = K.double()
        out.append(torch.fft.rfft2(torch.roll(z, (-c, -c), (0, 1))))
    return out


def _good(n):
    """Smallest even 2-3-5-smooth number >= n."""
    n += n & 1
    while True:
        m = n
        for q in (2, 3, 5):
            while m % q == 0:
                m //= q
        if m == 1:
            return n
        n += 2


def _conv(E, Kx, Ky, dx):
    """dx^2 conv(E, G) on the valid window (the last two dimensions), 64 bits."""
    N, e = E.shape[-1], (Kx.shape[0] - 1) // 2
    P = _good(N)
    F = torch.fft.rfft2(E.double(), s=(P, P))
    out = []
    for G in _spectra(Kx, Ky, P):
        out.append(torch.fft.irfft2(F * G, s=(P, P))[..., e : N - e, e : N - e] * dx ** 2)
    return out


def _grads(f, e):
    """Central differences (columns, rows) on the valid window, erosion >= 1."""
    f, N = f.double(), f.shape[-1]
    c = slice(e, N - e)
    return ((f[..., e + 1 : N - e + 1, c] - f[..., e - 1 : N - e - 1, c]) * 0.5,
            (f[..., c, e + 1 : N - e + 1] - f[..., c, e - 1 : N - e - 1]) * 0.5)


def _diff_t(wx, wy, e):
    """Transposed central differences of the valid window's wx, wy, N x N."""
    wx, wy = (torch.nn.functional.pad(w, (e, e, e, e)) for w in (wx, wy))
    out = torch.zeros_like(wx)
    out[..., 1:, :] += 0.5 * wx[..., :-1, :]
    out[..., :-1, :] -= 0.5 * wx[..., 1:, :]
    out[..., :, 1:] += 0.5 * wy[..., :, :-1]
    out[..., :, :-1] -= 0.5 * wy[..., :, 1:]
    return out


def _adj_g(hx, hy, Kx, Ky, dx, true_adjoint):
    """dx^2 (G * h) on the full N x N image, h zero outside its valid window;
    the exact adjoint correlates with G, the reference's convolves."""
    e = (Kx.shape[0] - 1) // 2
    N = hx.shape[-1] + 2 * e
    P = _good(N + 2 * e)
    Gx, Gy = _spectra(Kx, Ky, P)
    if true_adjoint:
        Gx, Gy = Gx.conj(), Gy.conj()
    hx, hy = (torch.nn.functional.pad(h, (e, e, e, e)) for h in (hx, hy))
    F = torch.fft.rfft2(hx, s=(P, P)) * Gx + torch.fft.rfft2(hy, s=(P, P)) * Gy
    return torch.fft.irfft2(F, s=(P, P))[..., :N, :N] * dx ** 2


def _fwd(f, g, Kx, Ky, dx):
    ux, uy = _conv(g, Kx, Ky, dx)
    fx, fy = _grads(f, (Kx.shape[0] - 1) // 2)
    return ux * fx + uy * fy


def _adj(v, ux, uy, f, Kx, Ky, dx, true_adjoint):
    e = (Kx.shape[0] - 1) // 2
    fx, fy = _grads(f, e)
    v = v.double()
    return (_diff_t(ux.double() * v, uy.double() * v, e), _adj_g(v * fx, v * fy, Kx, Ky, dx, true_adjoint))


def exact(case, seed):
    d = _inputs(case, seed)
    op, B, dx, Kx, Ky = case["op"], case["B"], case["dx"], d["Kx"], d["Ky"]
    e = (case["KW"] - 1) // 2
    if op == "oas":
        return [_fwd(d["I"], d["E"], Kx, Ky, dx)]
    if op == "adjoint":
        return list(_adj(d["v"], d["ux"], d["uy"], d["I"], Kx, Ky, dx, False))
    if op == "ragged":
        both = [_adj(d["v"][b], d["ux"][b], d["uy"][b], d["I"][b], Kx, Ky, dx, False) for b in range(B)]
        return [torch.cat([x[k].reshape(-1) for x in both]) for k in (0, 1)]
    if op in ("tangent", "tanadj"):
        ux, uy = _conv(d["g"], Kx, Ky, dx)
        dux, duy = _conv(d["dg"], Kx, Ky, dx)
        fx, fy = _grads(d["f"], e)
        dfx, dfy = _grads(d["df"], e)
        if op == "tangent":
            return [dux * fx + duy * fy + ux * dfx + uy * dfy]
        lam, dlam = d["lam"].double(), d["dlam"].double()
        return [_diff_t(dlam * ux + lam * dux, dlam * uy + lam * duy, e),
                _adj_g(dlam * fx + lam * dfx, dlam * fy + lam * dfy, Kx, Ky, dx, False)]
    # batches, a few images at a time
    N = case["N"]
    W = N - 2 * e
    sizes = [W] if op == "train" else [W, N, N]
    out = [torch.empty((B, n, n), device="cuda", dtype=torch.float64) for n in sizes]
    step = max(1, (1 << 24) // (N * N))
    for b in range(0, B, step):
        q = slice(b, min(B, b + step))
        if op == "train":
            out[0][q] = _fwd(d["E"][q], d["E"][q], Kx, Ky, dx)
            continue
        f, g, v = d["f"][q], d["g"][q], d["v"][q]
        ux, uy = _conv(g, Kx, Ky, dx)
        fx, fy = _grads(f, e)
        out[0][q] = ux * fx + uy * fy
        out[1][q], out[2][q] = _adj(v, ux, uy, f, Kx, Ky, dx, True)
    return out
