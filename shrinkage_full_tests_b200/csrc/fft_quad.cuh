// fft_quad.cuh — complex FFTs of length M (128, 256, 512), four lines at a
// time by a group of one or two warps, in packed FP32 pairs (sm_100a).
//
// M = R * J.  With n = j + J r (j < J, r < R) and K = k + R m (k < R, m < J)
//   X[K] = sum_j W_M^(j k) W_J^(j m) [ sum_r W_R^(r k) x[j + J r] ],
// so a transform is J butterflies of radix R, a twiddle, and R butterflies
// of radix J, with one exchange between them.  A line has TPL = J / 2
// threads.  Two distributions of a line over its threads:
//   pairs   thread q holds x[2q + l + J r], l = 0, 1: the operands of the
//           butterflies j = 2q and 2q + 1, as packed pairs (lane l) of real
//           and imaginary parts;
//   singles thread k holds X[k + R m] for its KPT values of k (k = q + TPL i).
// fft_dit goes from pairs to singles, fft_dif (the transposed flow graph)
// from singles to pairs; either direction of the transform (INV conjugates
// every twiddle).  A product in the frequency domain therefore runs between
// a dif and a dit with its operands in packed pairs, and neither transform
// reorders anything.
//
// Why this shape.  The passes are bound by instruction issue and by the
// shared-memory pipe before they are bound by HBM, so the transform is made
// of packed FP32 instructions (add / mul / fma .f32x2: two results per issue
// slot) and of as few exchanges as the registers allow: 32 values per thread
// need one exchange where 8 values per thread need two.  Every butterfly but
// the last stage of the radix-J ones pairs two butterflies with the same
// twiddle structure ("vertical", packed); that last stage combines the two
// lanes of a pair and is scalar, which is also where complex values change
// between (re, im) order in memory and packed pairs, for free.
// Per 512-point transform: about 230 warp instructions of arithmetic and 24
// shared-memory accesses, against about 600 and 130 for three radix-8 passes
// of scalar code over 64 threads.
//
// The exchange moves 16-byte quads (re0, re1, im0, im1): quad (p, k) of a
// line holds butterflies j = 2p, 2p + 1 at output k.  Row pitch R + 1 quads
// and line pitch = 2 (mod 8) quads put the eight quads of every quarter-warp
// (two rows or two columns of four lines) on distinct banks, for writes and
// reads alike.
//
// Lanes: thread t of a group is (q = t / 4, line = t % 4), so a warp holds
// 8 consecutive indices of 4 lines: accesses to an array blocked by four
// lines ([line / 4][index][line % 4]) are contiguous.
//
// All arithmetic uses explicit roundings (no contraction), so every kernel
// that inlines a transform computes bit-identical results.
#pragma once
#include <cuda_runtime.h>

namespace srk {

// ---- packed pairs ------------------------------------------------------------
using pk = unsigned long long;  // two floats: lane 0 in the low word
__device__ __forceinline__ pk pk_make(float a, float b) {
  pk r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ pk pk_dup(float a) { return pk_make(a, a); }
__device__ __forceinline__ float pk_lo(pk v) {
  float a, b;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
  return a;
}
__device__ __forceinline__ float pk_hi(pk v) {
  float a, b;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
  return b;
}
__device__ __forceinline__ pk pk_add(pk a, pk b) {
  pk r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ pk pk_mul(pk a, pk b) {
  pk r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ pk pk_fma(pk a, pk b, pk c) {
  pk r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ pk pk_sub(pk a, pk b) {
  pk r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// Sign change; the assembler folds it into the packed instruction that uses it.
__device__ __forceinline__ pk pk_neg(pk a) { return pk_make(-pk_lo(a), -pk_hi(a)); }
// a*b + c*d with one fixed rounding sequence (dot2 of scalars, per lane)
__device__ __forceinline__ pk pk_dot2(pk a, pk b, pk c, pk d) { return pk_fma(a, b, pk_mul(c, d)); }

// A pair of complex values.
struct cpk {
  pk re, im;
};
__device__ __forceinline__ cpk cpk_load(const float4& v) { return cpk{pk_make(v.x, v.y), pk_make(v.z, v.w)}; }
__device__ __forceinline__ float4 cpk_quad(const cpk& c) {
  return make_float4(pk_lo(c.re), pk_hi(c.re), pk_lo(c.im), pk_hi(c.im));
}
// a * w, or a * conj(w)
template <bool CONJ>
__device__ __forceinline__ cpk cpk_mul(const cpk& a, const cpk& w) {
  if constexpr (CONJ)
    return cpk{pk_fma(a.re, w.re, pk_mul(a.im, w.im)), pk_fma(a.im, w.re, pk_neg(pk_mul(a.re, w.im)))};
  else
    return cpk{pk_fma(a.re, w.re, pk_neg(pk_mul(a.im, w.im))), pk_fma(a.im, w.re, pk_mul(a.re, w.im))};
}

// ---- constants -----------------------------------------------------------------
// cos(pi k / 16), k = 0 .. 8
__host__ __device__ constexpr double cos16(int k) {
  return k == 0   ? 1.0
         : k == 1 ? 0.98078528040323044913
         : k == 2 ? 0.92387953251128675613
         : k == 3 ? 0.83146961230254523708
         : k == 4 ? 0.70710678118654752440
         : k == 5 ? 0.55557023301960222474
         : k == 6 ? 0.38268343236508977173
         : k == 7 ? 0.19509032201612826785
                  : 0.0;
}
// cos / sin(2 pi k / 32), 0 <= k < 16
__host__ __device__ constexpr double cos32(int k) { return k <= 8 ? cos16(k) : -cos16(16 - k); }
__host__ __device__ constexpr double sin32(int k) { return k <= 8 ? cos16(8 - k) : cos16(k - 8); }

template <bool NEG>
__device__ __forceinline__ pk pk_const(double v) {
  const pk p = pk_dup((float)v);
  return NEG ? pk_neg(p) : p;
}

// ---- packed butterflies -----------------------------------------------------------
// a = e + W o, b = e - W o with W = exp(-+ 2 pi i m / 16), 0 <= m < 8 (minus:
// forward).  W o = c (x + T y) + i c (y - T x) up to signs and a swap, T =
// tan(pi / 8): four fused steps per result pair, no separate product.
template <int m, bool INV>
__device__ __forceinline__ void pk_butterfly(const cpk& e, const cpk& o, cpk& a, cpk& b) {
  const pk x = o.re, y = o.im;
  if constexpr (m == 0) {
    a = cpk{pk_add(e.re, x), pk_add(e.im, y)};
    b = cpk{pk_sub(e.re, x), pk_sub(e.im, y)};
  } else if constexpr (m == 4) {
    const cpk p{pk_add(e.re, y), pk_sub(e.im, x)}, n{pk_sub(e.re, y), pk_add(e.im, x)};  // e -+ i o
    a = INV ? n : p;
    b = INV ? p : n;
  } else {
    constexpr bool diag = m == 2 || m == 6;
    constexpr double T = diag ? 1.0 : 0.41421356237309504880;                       // tan(pi/8)
    constexpr double C = diag ? 0.70710678118654752440 : 0.92387953251128675613;  // cos(pi/4), cos(pi/8)
    // theta = pi m / 8; forward W o = (x c + y s) + i (y c - x s), inverse with -s
    constexpr bool swap = m == 3 || m == 5;  // |sin| > |cos|
    constexpr double sc = m < 4 ? 1.0 : -1.0;  // sign of cos
    constexpr double ss = INV ? -1.0 : 1.0;    // sign of the sine term
    pk u, v;      // W o = +-C u +- i C v
    bool nu, nv;  // the signs
    if constexpr (!swap) {
      // re = sc C (x + (ss sc T) y), im = sc C (y - (ss sc T) x)
      u = diag ? (ss * sc > 0 ? pk_add(x, y) : pk_sub(x, y)) : pk_fma(pk_const<ss * sc < 0>(T), y, x);
      v = diag ? (ss * sc > 0 ? pk_sub(y, x) : pk_add(y, x)) : pk_fma(pk_const<(ss * sc > 0)>(T), x, y);
      nu = nv = sc < 0;
    } else {
      // re = ss C (y + (ss sc T) x), im = -ss C (x - (ss sc T) y)
      u = pk_fma(pk_const<ss * sc < 0>(T), x, y);
      v = pk_fma(pk_const<(ss * sc > 0)>(T), y, x);
      nu = ss < 0;
      nv = ss > 0;
    }
    const pk cp = pk_const<false>(C), cn = pk_const<true>(C);
    a = cpk{pk_fma(nu ? cn : cp, u, e.re), pk_fma(nv ? cn : cp, v, e.im)};
    b = cpk{pk_fma(nu ? cp : cn, u, e.re), pk_fma(nv ? cp : cn, v, e.im)};
  }
}

// In-register R-point DFT of both lanes (natural order in and out), radix-2
// decimation in time applied recursively.
template <int R, bool INV>
struct PkDft {
  template <int K>
  __device__ __forceinline__ static void combine(cpk* a, const cpk* e, const cpk* o) {
    if constexpr (K < R / 2) {
      pk_butterfly<(16 / R) * K, INV>(e[K], o[K], a[K], a[K + R / 2]);
      combine<K + 1>(a, e, o);
    }
  }
  __device__ __forceinline__ static void run(cpk* a) {
    cpk e[R / 2], o[R / 2];
#pragma unroll
    for (int i = 0; i < R / 2; ++i) { e[i] = a[2 * i]; o[i] = a[2 * i + 1]; }
    PkDft<R / 2, INV>::run(e);
    PkDft<R / 2, INV>::run(o);
    combine<0>(a, e, o);
  }
};
template <bool INV>
struct PkDft<1, INV> {
  __device__ __forceinline__ static void run(cpk*) {}
};

// Scalar combine of the two lanes (E, O) of a pair: X0 = E + W O, X1 = E - W O,
// W = exp(-+ 2 pi i k / 32), 0 <= k < 16.
template <int k, bool INV>
__device__ __forceinline__ void lane_combine(const cpk& z, float2& X0, float2& X1) {
  const float ex = pk_lo(z.re), ey = pk_lo(z.im), x = pk_hi(z.re), y = pk_hi(z.im);
  if constexpr (k == 0) {
    X0 = make_float2(__fadd_rn(ex, x), __fadd_rn(ey, y));
    X1 = make_float2(__fsub_rn(ex, x), __fsub_rn(ey, y));
  } else if constexpr (k == 8) {
    const float2 p = make_float2(__fadd_rn(ex, y), __fsub_rn(ey, x));
    const float2 n = make_float2(__fsub_rn(ex, y), __fadd_rn(ey, x));
    X0 = INV ? n : p;
    X1 = INV ? p : n;
  } else {
    constexpr double c = cos32(k), s = INV ? -sin32(k) : sin32(k);
    constexpr bool big_c = k < 4 || k > 12 || k == 4 || k == 12;
    constexpr double T = big_c ? s / c : c / s;
    constexpr float cu = (float)(big_c ? c : s), cv = (float)(big_c ? c : -s);
    const float u = big_c ? __fmaf_rn((float)T, y, x) : __fmaf_rn((float)T, x, y);
    const float v = big_c ? __fmaf_rn((float)-T, x, y) : __fmaf_rn((float)-T, y, x);
    X0 = make_float2(__fmaf_rn(cu, u, ex), __fmaf_rn(cv, v, ey));
    X1 = make_float2(__fmaf_rn(-cu, u, ex), __fmaf_rn(-cv, v, ey));
  }
}
// The transposed step: lane 0 = X0 + X1, lane 1 = (X0 - X1) W.
template <int k, bool INV>
__device__ __forceinline__ cpk lane_split(const float2& X0, const float2& X1) {
  const float ax = __fadd_rn(X0.x, X1.x), ay = __fadd_rn(X0.y, X1.y);
  const float x = __fsub_rn(X0.x, X1.x), y = __fsub_rn(X0.y, X1.y);
  if constexpr (k == 0) {
    return cpk{pk_make(ax, x), pk_make(ay, y)};
  } else if constexpr (k == 8) {
    return INV ? cpk{pk_make(ax, -y), pk_make(ay, x)} : cpk{pk_make(ax, y), pk_make(ay, -x)};
  } else {
    constexpr double c = cos32(k), s = INV ? -sin32(k) : sin32(k);
    constexpr bool big_c = k < 4 || k > 12 || k == 4 || k == 12;
    constexpr double T = big_c ? s / c : c / s;
    constexpr float cu = (float)(big_c ? c : s), cv = (float)(big_c ? c : -s);
    const float u = big_c ? __fmaf_rn((float)T, y, x) : __fmaf_rn((float)T, x, y);
    const float v = big_c ? __fmaf_rn((float)-T, x, y) : __fmaf_rn((float)-T, y, x);
    return cpk{pk_make(ax, __fmul_rn(cu, u)), pk_make(ay, __fmul_rn(cv, v))};
  }
}

// ---- transform geometry --------------------------------------------------------------
constexpr int kLines = 4;  // lines per group
template <int M>
struct Quad {
  static_assert(M == 128 || M == 256 || M == 512, "unsupported FFT length");
  static constexpr int R = M == 128 ? 8 : 16;   // radix of the pairs side
  static constexpr int J = M / R;               // radix of the singles side (16 or 32)
  static constexpr int TPL = J / 2;             // threads per line
  static constexpr int KPT = R / TPL;           // values of k per thread
  static constexpr int GT = TPL * kLines;       // threads per group
  static constexpr int VPT = KPT * J;           // complex values per thread
  static constexpr int RP = R + 1;              // exchange row pitch (quads)
  static constexpr int LP = (J / 2) * RP + 2;   // exchange line pitch (quads)
  static constexpr int XQ = kLines * LP;        // quads of one group's exchange
  static constexpr int TWQ = (J / 2) * R;       // twiddle quads (p, k)
  static_assert(RP % 8 == 1 && LP % 8 == 2, "exchange pitches");
  static_assert(R % TPL == 0 || TPL % R == 0, "geometry");
  static_assert(KPT >= 1 && VPT == R * 2, "values per thread");
};

// Barrier over the threads of a group: a warp, or the whole block (a group
// of two warps is its block's only one).
template <int M>
__device__ __forceinline__ void group_sync() {
  if constexpr (Quad<M>::GT == 32)
    __syncwarp();
  else
    __syncthreads();
}

// One thread's place in its group and the group's shared memory.
struct QuadThread {
  int q, line;
};
template <int M>
__device__ __forceinline__ QuadThread quad_thread() {
  const int t = threadIdx.x % Quad<M>::GT;
  return QuadThread{t >> 2, t & 3};
}

// Twiddle quads W_M^(j k): (re, re, im, im) of j = 2p, 2p + 1.  The forward
// values; the inverse conjugates.
__device__ __forceinline__ cpk tw_quad(const float4* __restrict__ tw, int i) { return cpk_load(__ldg(tw + i)); }

// All twiddle quads of one k: four from the table, the others by products with
// W^(8k) and W^(16k) (lane 0 of quads 4 and 8), at most two roundings each.
// A table read serves only 8 distinct quads per warp (its four lines share
// them) but costs the four wavefronts of any 16-byte access, and the passes
// are short of shared-memory / L1 bandwidth, not of arithmetic.
template <int M>
__device__ __forceinline__ void tw_all(const float4* __restrict__ tw, int k, cpk (&t)[Quad<M>::J / 2]) {
  using Q = Quad<M>;
#pragma unroll
  for (int p = 0; p < 4; ++p) t[p] = tw_quad(tw, p * Q::R + k);
#pragma unroll
  for (int s = 4; s < Q::J / 2; s *= 2) {
    const float* f = reinterpret_cast<const float*>(tw + s * Q::R + k);
    const cpk u{pk_dup(__ldg(f)), pk_dup(__ldg(f + 2))};
#pragma unroll
    for (int p = 0; p < s; ++p) t[p + s] = cpk_mul<false>(t[p], u);
  }
}

template <int J, bool INV, int K = 0>
__device__ __forceinline__ void lane_combine_all(const cpk (&z)[J / 2], float2* X) {
  if constexpr (K < J / 2) {
    lane_combine<(32 / J) * K, INV>(z[K], X[K], X[K + J / 2]);
    lane_combine_all<J, INV, K + 1>(z, X);
  }
}
template <int J, bool INV, int K = 0>
__device__ __forceinline__ void lane_split_all(const float2* X, cpk (&z)[J / 2]) {
  if constexpr (K < J / 2) {
    z[K] = lane_split<(32 / J) * K, INV>(X[K], X[K + J / 2]);
    lane_split_all<J, INV, K + 1>(X, z);
  }
}

// pairs -> singles: a[r] = x[2q + l + J r] in, X[i J + m] = X[k_i + R m] out,
// k_i = q + TPL i.  ex: the group's exchange quads.
template <int M, bool INV>
__device__ __forceinline__ void fft_dit(cpk (&a)[Quad<M>::R], float2 (&X)[Quad<M>::VPT], float4* __restrict__ ex,
                                        const float4* __restrict__ tw, const QuadThread& t) {
  using Q = Quad<M>;
  PkDft<Q::R, INV>::run(a);
  group_sync<M>();  // the exchange may still be read from its previous use
  float4* wr = ex + t.line * Q::LP + t.q * Q::RP;
#pragma unroll
  for (int k = 0; k < Q::R; ++k) wr[k] = cpk_quad(a[k]);
  group_sync<M>();
#pragma unroll
  for (int i = 0; i < Q::KPT; ++i) {
    const int k = t.q + Q::TPL * i;
    const float4* rd = ex + t.line * Q::LP + k;
    cpk z[Q::J / 2], w[Q::J / 2];
    tw_all<M>(tw, k, w);
#pragma unroll
    for (int p = 0; p < Q::J / 2; ++p) z[p] = cpk_mul<INV>(cpk_load(rd[p * Q::RP]), w[p]);
    PkDft<Q::J / 2, INV>::run(z);
    lane_combine_all<Q::J, INV>(z, X + i * Q::J);
  }
}

// singles -> pairs, up to the last radix-R butterflies: their operands are in
// a; fft_dif_finish runs them.  Between the two the exchange is free again
// once the group has synchronised.  mid() runs between the group's first
// synchronisation (every thread is past the loads of its X) and the exchange.
template <int M, bool INV, typename F>
__device__ __forceinline__ void fft_dif_begin(const float2 (&X)[Quad<M>::VPT], cpk (&a)[Quad<M>::R],
                                              float4* __restrict__ ex, const float4* __restrict__ tw,
                                              const QuadThread& t, F&& mid) {
  using Q = Quad<M>;
  cpk z[Q::KPT][Q::J / 2];
#pragma unroll
  for (int i = 0; i < Q::KPT; ++i) {
    const int k = t.q + Q::TPL * i;
    lane_split_all<Q::J, INV>(X + i * Q::J, z[i]);
    PkDft<Q::J / 2, INV>::run(z[i]);
    cpk w[Q::J / 2];
    tw_all<M>(tw, k, w);
#pragma unroll
    for (int p = 0; p < Q::J / 2; ++p) z[i][p] = cpk_mul<INV>(z[i][p], w[p]);
  }
  group_sync<M>();  // the exchange may still be read from its previous use
  mid();
#pragma unroll
  for (int i = 0; i < Q::KPT; ++i) {
    float4* wr = ex + t.line * Q::LP + t.q + Q::TPL * i;
#pragma unroll
    for (int p = 0; p < Q::J / 2; ++p) wr[p * Q::RP] = cpk_quad(z[i][p]);
  }
  group_sync<M>();
  const float4* rd = ex + t.line * Q::LP + t.q * Q::RP;
#pragma unroll
  for (int k = 0; k < Q::R; ++k) a[k] = cpk_load(rd[k]);
}
template <int M, bool INV>
__device__ __forceinline__ void fft_dif_begin(const float2 (&X)[Quad<M>::VPT], cpk (&a)[Quad<M>::R],
                                              float4* __restrict__ ex, const float4* __restrict__ tw,
                                              const QuadThread& t) {
  fft_dif_begin<M, INV>(X, a, ex, tw, t, [] {});
}
template <int M, bool INV>
__device__ __forceinline__ void fft_dif_finish(cpk (&a)[Quad<M>::R]) {
  PkDft<Quad<M>::R, INV>::run(a);
}

}  // namespace srk
