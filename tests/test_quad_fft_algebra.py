"""CPU check of the algebra and the index ranges behind the engine's
transforms (csrc/fft_quad.cuh, csrc/engine.cuh): the two flow graphs, the
exchange's addresses and banks, the scratch blocks and the gradient windows."""
import numpy as np
import pytest

SIZES = [128, 256, 512]


def quad(M):
    R = 8 if M == 128 else 16
    J = M // R
    return R, J, J // 2


def twiddle(M, p, lane, k):
    return np.exp(-2j * np.pi * ((2 * p + lane) * k) / M)


def dft(n):
    return np.exp(-2j * np.pi * np.outer(np.arange(n), np.arange(n)) / n)


def dit(x, M, inv):
    """pairs -> singles: radix-R butterflies of j, twiddle, lane combine."""
    R, J, H = quad(M)
    c = (lambda v: np.conj(v)) if inv else (lambda v: v)
    y = np.einsum("kr,rj->jk", c(dft(R)), x.reshape(R, J))  # y[j][k]
    X = np.empty(M, complex)
    for k in range(R):
        z = np.array([[y[2 * p + l, k] * c(twiddle(M, p, l, k)) for l in (0, 1)] for p in range(H)])
        e, o = (c(dft(H)) @ z[:, l] for l in (0, 1))
        w = c(np.exp(-2j * np.pi * np.arange(H) / J))
        X[k + R * np.arange(H)] = e + w * o
        X[k + R * (np.arange(H) + H)] = e - w * o
    return X


def dif(X, M, inv):
    """singles -> pairs: lane split, radix-J/2 butterflies, twiddle, radix R."""
    R, J, H = quad(M)
    c = (lambda v: np.conj(v)) if inv else (lambda v: v)
    ex = np.empty((J, R), complex)
    for k in range(R):
        a, b = X[k + R * np.arange(H)], X[k + R * (np.arange(H) + H)]
        w = c(np.exp(-2j * np.pi * np.arange(H) / J))
        even, odd = c(dft(H)) @ (a + b), c(dft(H)) @ ((a - b) * w)
        for p in range(H):
            ex[2 * p, k] = even[p] * c(twiddle(M, p, 0, k))
            ex[2 * p + 1, k] = odd[p] * c(twiddle(M, p, 1, k))
    return (c(dft(R)) @ ex.T).reshape(M)  # x[j + J r]


@pytest.mark.parametrize("M", SIZES)
@pytest.mark.parametrize("inv", [False, True])
def test_flow_graphs_are_the_dft(M, inv):
    rng = np.random.default_rng(M)
    x = rng.standard_normal(M) + 1j * rng.standard_normal(M)
    ref = np.fft.ifft(x) * M if inv else np.fft.fft(x)
    for f in (dit, dif):
        assert np.abs(f(x, M, inv) - ref).max() < 1e-11 * np.abs(ref).max()


@pytest.mark.parametrize("M", SIZES)
def test_generated_twiddles(M):
    """Quads past the fourth come from products with W^(8k) and W^(16k)."""
    R, J, H = quad(M)
    for k in range(R):
        t = [np.array([twiddle(M, p, l, k) for l in (0, 1)]) for p in range(4)]
        s = 4
        while s < H:
            t += [t[p] * twiddle(M, s, 0, k) for p in range(s)]
            s *= 2
        assert len(t) == H
        for p in range(H):
            assert np.abs(t[p] - [twiddle(M, p, l, k) for l in (0, 1)]).max() < 1e-14


@pytest.mark.parametrize("M", SIZES)
def test_exchange_addresses(M):
    R, J, H = quad(M)
    RP, LP = R + 1, H * (R + 1) + 2
    cells = {line * LP + p * RP + k for line in range(4) for p in range(H) for k in range(R)}
    assert len(cells) == 4 * H * R and max(cells) < 4 * LP  # no overlap, inside
    for q0 in range(0, H, 2):  # the quarter-warps: two rows (writes) or columns (reads) of four lines
        write = {(line * LP + q * RP) % 8 for q in (q0, q0 + 1) for line in range(4)}
        read = {(line * LP + q) % 8 for q in (q0, q0 + 1) for line in range(4)}
        assert len(write) == 8 and len(read) == 8


@pytest.mark.parametrize("M", SIZES)
def test_scratch_blocks_and_windows(M):
    R, J, H = quad(M)
    ex_bytes, buf_bytes, lead = 64 * (H * (R + 1) + 2), 32 * M, 2 * M
    for e in range(0, M // 2 - 3):
        S = M - 2 * e
        xa, P = e & ~3, (S + 7) & ~7
        assert (e + S - 1 - xa) // 4 < P // 4              # engine layout: last valid column's block
        assert (S + (e - xa) + 3) // 4 <= P // 4           # blocks P3 reads
        for size, pitch in ((4, (S + 28) // 32 * 32 + 8), (2, (S + 56) // 64 * 64 + 16)):
            assert pitch * size % 16 == 0
            assert (pitch * size // 4) % 32 == 8           # pair reads of a half-warp on distinct banks
            epc = 16 // size
            for off in range(epc):                         # first window row in its 16-byte piece
                n = off + S + 2
                assert (n + epc - 1) // epc * epc <= pitch
                # rows 0 .. M-1 of the tile, with their neighbours, stay inside the group's memory
                lo, hi = off + 1 - e, off + 1 - e + M - 1
                assert lo * size >= -lead
                for col, first, last in ((0, lo, hi), (1, lo - 1, hi + 1), (5, lo, hi)):
                    assert (col * pitch + first) * size >= -lead
                    assert lead + (col * pitch + last + 1) * size <= ex_bytes
                    assert (col * pitch + last + 1) * size <= buf_bytes
