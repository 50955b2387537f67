// engine.cuh — overlap-and-save (OaS) FFT convolution engine for the
// resist-shrinkage operator and its derivatives.
//
// Terminology
//   image      N x N, column-major buf[col*N + row] ("x" = column, "y" = row)
//   tile       M x M window of the (virtual) input image at origin
//              (tx*S, ty*S); its valid outputs are local x,y in [e, e+S)
//   work tile  (WT) one complex M x M field pair processed together:
//              either two real tiles packed as re/im (forward-type ops), the
//              base and tangent field of one tile (JVP-type ops), or two
//              packed tiles with two fields each (adjoint-type ops).
//
// One WT goes through three passes whose intermediates live in a scratch
// buffer (8-byte complex, blocked by four lines so that both the pass that
// writes and the pass that reads touch whole 128-byte pieces straight from
// registers, see fft_quad.cuh for the lane order):
//   P1  per column x: load the field(s) (the op's loader computes them on
//       the fly: image values, or v*df/dx products for the adjoint), FFT
//       along y                          -> S1[wt][k][ky/4][x][ky%4]
//   P2  per row ky: FFT along x, spectral map with the kernel spectra (Gx,
//       Gy; conjugated for a true adjoint), inverse FFT along kx, keep the
//       valid columns                    -> S2[wt][l][(x-xa)/4][ky][x%4]
//   P3  per valid column: inverse FFT along ky, then the op's epilogue
//       (central differences of f, combine, store) — conv(g,Gx), conv(g,Gy)
//       never leave registers.
// xa = e rounded down to a multiple of four (s2_first).
//
// A group of one (M = 128, 256) or two (M = 512) warps transforms four lines
// with 32 (M = 128: 16) complex values per thread.  Its inputs (columns,
// spectra, blocks of S1 and S2, image windows) arrive in shared memory by
// bulk copies, which free the group's exchange and one more buffer hold in
// turn; results are stored from registers.  A second field (P2's Z*Gy, P3's
// and the adjoint's second field) stays in registers: at 168 registers and
// 12 warps per SM that costs less than its round trip through shared memory
// at a higher occupancy, since the packed transforms have 16 independent
// chains per thread.
//
// The reference performs the same linear "valid" convolution with cufftDX
// tiles (srk_forward.cuh:354-423) or whole-image cuFFT
// (training/srk_training_forward.cuh:175-241); with KW <= 2e+1 there is no
// circular wrap-around in either, so all of them equal
//     u[o] = dx^2 * sum_d E[o+e-d] * G[c+d]
// (adjoint/main_adjoint.cu:70-90) up to rounding.
#pragma once
#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <cuda_bf16.h>
#include <cstdint>
#include <type_traits>
#include "fft_quad.cuh"
#include "tc.cuh"
#include "tile_cols.h"

// CTAs of kThreads threads per SM the kernels are compiled for (register cap
// 65536 / (kThreads n), in steps of 8): 8 -> 128 registers, 6 -> 168.
#ifndef SRK_P1_MIN_BLOCKS
#define SRK_P1_MIN_BLOCKS 8
#endif
#ifndef SRK_P1_ADJ_MIN_BLOCKS
#define SRK_P1_ADJ_MIN_BLOCKS 6
#endif
#ifndef SRK_P2_MIN_BLOCKS
#define SRK_P2_MIN_BLOCKS 6
#endif
#ifndef SRK_P3_MIN_BLOCKS
#define SRK_P3_MIN_BLOCKS 6
#endif
#ifndef SRK_P3_ADJ_MIN_BLOCKS
#define SRK_P3_ADJ_MIN_BLOCKS 8
#endif
// M = 128 has half the values per thread: every pass fits 128 registers.
#ifndef SRK_SMALL_MIN_BLOCKS
#define SRK_SMALL_MIN_BLOCKS 8
#endif

namespace srk {

constexpr int kThreads = 64;

enum Op : int {
  OP_FWD = 0,       // R = ux*df/dx + uy*df/dy (pairs of tiles); optional ux/uy
  OP_VJP_F = 1,     // wx = ux*v, wy = uy*v (pairs of tiles) for dL/df
  OP_JVP = 2,       // dh from g + i*dg (one tile per WT)
  OP_TANADJ_F = 3,  // wx = dlam*ux_g + lam*ux_dg, wy likewise (one tile per WT)
  OP_ADJ = 4,       // dL/dg (full N x N) from hx + i*hy fields (pairs of tiles)
};

template <int OP> struct OpTraits;
template <> struct OpTraits<OP_FWD>      { static constexpr int K = 1, L = 2; static constexpr bool PAIRS = true; };
template <> struct OpTraits<OP_VJP_F>    { static constexpr int K = 1, L = 2; static constexpr bool PAIRS = true; };
template <> struct OpTraits<OP_JVP>      { static constexpr int K = 1, L = 2; static constexpr bool PAIRS = false; };
template <> struct OpTraits<OP_TANADJ_F> { static constexpr int K = 1, L = 2; static constexpr bool PAIRS = false; };
template <> struct OpTraits<OP_ADJ>      { static constexpr int K = 2, L = 1; static constexpr bool PAIRS = true; };

// One image of a ragged batch: its size and where it starts in the
// concatenated N-sized and W-sized batch arrays (elements).  A column slab
// of one image is a one-image table whose offsets are negative (the
// caller's pointers address the slab's first column) and whose stencil
// blocks cover only the pixel columns [cx0, cx1).
struct RagImage {
  long long on, ow;
  int N, W;
  int blk0;      // first block of this image in the ragged stencil launch
  int cx0, cx1;  // pixel columns of the N x N output the stencil writes
  int pad;
};

// Tile geometry of one launch.  A uniform batch tiles every image alike
// (tile u -> image u / TT); a ragged batch of images of different N lists
// its tiles in `rtile` (image, x0, y0) and its images in `rimg`.
struct Geom {
  int M;      // FFT tile size
  int e;      // first valid local output of a tile (the erosion, or 0: see adj_geom)
  int S;      // valid outputs per tile per axis
  int org;    // origin of the first tile in virtual coordinates (uniform batch)
  int T;      // tiles per axis (uniform batch)
  int Nin;    // virtual input size (N for forward-type, N + 2e for adjoint)
  int Wout;   // output size (W for forward-type, N for adjoint)
  int TT;     // T*T
  int U;      // tiles in the whole batch
  int N, W;   // image and valid-output size (uniform batch)
  int wout_n; // outputs are N x N (adjoint-type) rather than W x W
  const int4* __restrict__ rtile;      // ragged: tile -> (image, x0, y0, 0); else nullptr
  const RagImage* __restrict__ rimg;   // ragged: per-image sizes and offsets
  unsigned int* err;                   // error word of the bounded waits (may be nullptr)
};

// Operand pointers.  All images are column-major; batch strides are
// N*N for N-sized images and W*W for W-sized ones.
struct OpArgs {
  const void* E;    // convolved field g            [B][N][N]
  const void* I;    // differentiated field f       [B][N][N]
  const void* dE;   // tangent of g                 [B][N][N]
  const void* dI;   // tangent of f                 [B][N][N]
  const void* v;    // cotangent (lambda_h)         [B][W][W]
  const void* dv;   // tangent of the cotangent     [B][W][W]
  void* out0;       // R | dh | wx | dL/dg
  void* out1;       // wy
  void* out_ux;     // optional ux (OP_FWD)
  void* out_uy;     // optional uy (OP_FWD)
  int N, W, e;
};

// ---- storage types --------------------------------------------------------
template <typename T> __device__ __forceinline__ float ldf(const T* p, long long i);
template <> __device__ __forceinline__ float ldf<float>(const float* p, long long i) { return __ldg(p + i); }
template <> __device__ __forceinline__ float ldf<__half>(const __half* p, long long i) { return __half2float(p[i]); }
template <> __device__ __forceinline__ float ldf<__nv_bfloat16>(const __nv_bfloat16* p, long long i) {
  return __bfloat162float(p[i]);
}
template <typename T> __device__ __forceinline__ void stf(T* p, long long i, float v);
template <> __device__ __forceinline__ void stf<float>(float* p, long long i, float v) { p[i] = v; }
template <> __device__ __forceinline__ void stf<__half>(__half* p, long long i, float v) { p[i] = __float2half_rn(v); }
template <> __device__ __forceinline__ void stf<__nv_bfloat16>(__nv_bfloat16* p, long long i, float v) {
  p[i] = __float2bfloat16_rn(v);
}

// a*b + c*d with one fixed rounding sequence (pk_dot2 of scalars).
__device__ __forceinline__ float dot2(float a, float b, float c, float d) { return __fmaf_rn(a, b, __fmul_rn(c, d)); }

struct TileRef {
  int b, x0, y0;     // image index and tile origin in virtual input coordinates
  bool live;
  int N, W, Wout;    // this image's size, valid-output size and output size
  long long on, ow;  // offset of this image in N-sized / W-sized batch arrays
};
__device__ __forceinline__ TileRef tile_of(const Geom& g, int u) {
  TileRef t;
  t.live = u < g.U;
  const int uu = t.live ? u : 0;
  if (g.rtile) {
    const int4 q = g.rtile[uu];
    const RagImage im = g.rimg[q.x];
    t.b = q.x;
    t.x0 = q.y;
    t.y0 = q.z;
    t.N = im.N;
    t.W = im.W;
    t.on = im.on;
    t.ow = im.ow;
  } else {
    if (g.TT == 1) {  // one tile per image (tile size >= image): no divisions
      t.b = uu;
      t.x0 = g.org;
      t.y0 = g.org;
    } else {
      t.b = uu / g.TT;
      const int r = uu - t.b * g.TT;
      const int tx = r / g.T, ty = r - (r / g.T) * g.T;
      t.x0 = tx * g.S;
      t.y0 = ty * g.S;
    }
    t.N = g.N;
    t.W = g.W;
    t.on = (long long)t.b * g.N * g.N;
    t.ow = (long long)t.b * g.W * g.W;
  }
  t.Wout = g.wout_n ? t.N : t.W;
  return t;
}

// ---- blocks, groups and scratch layout -----------------------------------------
// A CTA of kThreads threads holds groups_of<M>() groups of four lines.
template <int M>
__host__ __device__ constexpr int groups_of() { return kThreads / Quad<M>::GT; }
template <int M>
__host__ __device__ constexpr int unit_lines() { return kLines * groups_of<M>(); }
// First column of S2: the valid columns start at x = e; the blocks of four
// start at a multiple of four so that P2's stores cover whole blocks.
__host__ __device__ inline int s2_first(int e) { return e & ~3; }
// Columns of S2, a multiple of 8.  With S = M - 2e (M a multiple of 8),
// S mod 8 = -2e mod 8, so (S + 7) & ~7 >= S + e % 4: xa .. e + S - 1 fits.
__host__ __device__ inline int s2_pitch(int S) { return (S + 7) & ~7; }
// Blocks of four columns that hold a valid one, first valid column xa + off.
__host__ __device__ inline int s2_blocks(int S, int off) { return (S + off + kLines - 1) / kLines; }

// Scratch of one work tile: S1 [K fields] of M x M, then S2 [L fields] of
// s2_pitch(S) x M (float2).
template <int M, int OP>
__host__ __device__ constexpr size_t s1_elems() { return (size_t)OpTraits<OP>::K * M * M; }
template <int M, int OP>
__host__ __device__ inline size_t wt_elems(int S) {
  return s1_elems<M, OP>() + (size_t)OpTraits<OP>::L * M * s2_pitch(S);
}

// Engine layout of a kernel spectrum: quads of two neighbouring kx (re, re,
// im, im), blocked by four rows ky like S1, so P2 multiplies packed pairs
// read as contiguous 16-byte quads.  Index of Re G(ky, kx) in floats; Im is
// two floats further.
__host__ __device__ inline size_t spec_index(int M, int ky, int kx) {
  return 4 * (((size_t)(ky >> 2) * (M / 2) + (kx >> 1)) * 4 + (ky & 3)) + (kx & 1);
}

// ---- a group's shared memory and bulk copies ----------------------------------------
// Inputs that are contiguous runs (image columns, S1 and S2 blocks, spectra)
// arrive by bulk copies (cp.async.bulk, the TMA engine) into shared memory:
// the copies need no registers and no L1 lines while in flight.  Loads
// straight to registers did: at two to three exchanges of 17 KB per SM's
// free L1 the lines in flight, not HBM, bounded the passes (P1 at M = 512
// moved 5.5 TB/s against 6.2 with bulk copies).
//   exchange  Quad<M>::XQ quads; also the landing zone of the first input
//   buffer    one block of four lines (4 M complex values): the second input,
//             the spectra, or a gradient window
//   barriers  two mbarriers
// A wait whose copy never comes ends the thread (wait): nothing is made from
// the missing data and, without the leader, no further copy is issued.  The
// call's outputs are incomplete, which the error word tells the host.
template <int M>
__host__ __device__ constexpr size_t exch_bytes() { return sizeof(float4) * (size_t)Quad<M>::XQ; }
template <int M>
__host__ __device__ constexpr size_t block_bytes() { return sizeof(float2) * (size_t)kLines * M; }
template <int M, bool BUF>
__host__ __device__ constexpr size_t group_bytes() { return exch_bytes<M>() + (BUF ? block_bytes<M>() : 0) + 16; }
// Polls before a wait gives up: the second half of them is the wait for a copy
// that may still land in the block's memory.
constexpr unsigned long long kBulkWaitLimit = 1ull << 23;
constexpr unsigned kStopSite = 20;  // what a thread that gave up a wait writes to the error word
// The last two quads of the exchange are used by no line (Quad<M>::LP) and
// what lands in the exchange ends before them: a thread that gives up a wait
// sets this word, for the code whose other threads go on.
template <int M>
__host__ __device__ constexpr size_t landing_bytes() { return exch_bytes<M>() - 2 * sizeof(float4); }
template <int M>
__device__ __forceinline__ unsigned* stop_word(void* group_memory) {
  return reinterpret_cast<unsigned*>(static_cast<float4*>(group_memory) + Quad<M>::XQ - 1);
}

template <int M>
struct GroupMem {
  QuadThread t;
  float4* ex;
  unsigned char* buf;
  uint64_t* bar;       // two barriers
  unsigned parity;     // bit i: the phase barrier i waits for next
  unsigned int* err;   // error word (device or mapped host memory, may be nullptr)
  __device__ __forceinline__ bool leader() const { return threadIdx.x % Quad<M>::GT == 0; }
  // Copies may be issued into memory that the group has used before.
  __device__ __forceinline__ void open() const {
    tc::fence_async_smem();
    group_sync<M>();
  }
  // One contiguous run by the leader.
  __device__ __forceinline__ void fetch(int i, void* dst, const void* src, unsigned bytes) const {
    if (leader()) {
      tc::mbar_expect_tx(bar + i, bytes);
      tc::bulk_g2s(dst, src, bytes, bar + i);
    }
  }
  __device__ __forceinline__ void wait(int i, unsigned long long limit = kBulkWaitLimit) {
    tc::leave_unless<kStopSite>(tc::mbar_wait(bar + i, parity >> i & 1u, limit), err, stop_word<M>(ex));
    parity ^= 1u << i;
  }
};
// Carves the group's part out of the block's shared memory and initialises
// its barriers (once per kernel).
template <int M, bool BUF>
__device__ __forceinline__ GroupMem<M> group_mem(unsigned char* sm, unsigned int* err) {
  GroupMem<M> g;
  unsigned char* p = sm + threadIdx.x / Quad<M>::GT * group_bytes<M, BUF>();
  g.t = quad_thread<M>();
  g.ex = reinterpret_cast<float4*>(p);
  g.buf = BUF ? p + exch_bytes<M>() : nullptr;
  g.bar = reinterpret_cast<uint64_t*>(p + group_bytes<M, BUF>() - 16);
  g.parity = 0;
  g.err = err;
  if (g.leader()) {
    tc::mbar_init(g.bar, 1);
    tc::mbar_init(g.bar + 1, 1);
    *stop_word<M>(g.ex) = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  return g;
}

// ---- loaders ------------------------------------------------------------------------
// Shared-memory image values: one, and an aligned pair.
template <typename T> __device__ __forceinline__ float swin(const T* p);
template <> __device__ __forceinline__ float swin<float>(const float* p) { return *p; }
template <> __device__ __forceinline__ float swin<__half>(const __half* p) { return __half2float(*p); }
template <> __device__ __forceinline__ float swin<__nv_bfloat16>(const __nv_bfloat16* p) { return __bfloat162float(*p); }
template <typename T> __device__ __forceinline__ pk swin2(const T* p);
template <> __device__ __forceinline__ pk swin2<float>(const float* p) {
  return *reinterpret_cast<const unsigned long long*>(p);
}
template <> __device__ __forceinline__ pk swin2<__half>(const __half* p) {
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(p));
  return pk_make(f.x, f.y);
}
template <> __device__ __forceinline__ pk swin2<__nv_bfloat16>(const __nv_bfloat16* p) {
  const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p));
  return pk_make(f.x, f.y);
}

// One value and an aligned pair under a predicate (zero without it): a
// predicated load, not a branch around one.  Ordinary loads that stay behind
// grid_wait (volatile, memory clobber): what they read may be stored by the
// kernel before, which still runs when a dependent launch's blocks start, so
// the read-only path (ld.global.nc) does not serve.
__device__ __forceinline__ unsigned short ldp16(const void* p, bool on) {
  unsigned short v;
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\tmov.b16 %0, 0;\n\t@q ld.global.b16 %0, [%1];\n\t}"
               : "=h"(v) : "l"(p), "r"((unsigned)on) : "memory");
  return v;
}
__device__ __forceinline__ unsigned ldp32(const void* p, bool on) {
  unsigned v;
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\tmov.b32 %0, 0;\n\t@q ld.global.b32 %0, [%1];\n\t}"
               : "=r"(v) : "l"(p), "r"((unsigned)on) : "memory");
  return v;
}
__device__ __forceinline__ pk ldp64(const void* p, bool on) {
  pk v;
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\tmov.b64 %0, 0;\n\t@q ld.global.b64 %0, [%1];\n\t}"
               : "=l"(v) : "l"(p), "r"((unsigned)on) : "memory");
  return v;
}
template <typename T> __device__ __forceinline__ float ldp(const T* p, bool on);
template <> __device__ __forceinline__ float ldp<float>(const float* p, bool on) { return __uint_as_float(ldp32(p, on)); }
template <> __device__ __forceinline__ float ldp<__half>(const __half* p, bool on) {
  return __half2float(__ushort_as_half(ldp16(p, on)));
}
template <> __device__ __forceinline__ float ldp<__nv_bfloat16>(const __nv_bfloat16* p, bool on) {
  return __bfloat162float(__ushort_as_bfloat16(ldp16(p, on)));
}
// Two consecutive values as a packed pair; VEC: one aligned access under `lo`.
template <bool VEC, typename T>
__device__ __forceinline__ pk ld2(const T* __restrict__ p, long long i, bool lo, bool hi) {
  if constexpr (!VEC) {
    return pk_make(ldp(p + i, lo), ldp(p + i + 1, hi));
  } else if constexpr (sizeof(T) == 4) {
    return ldp64(p + i, lo);
  } else {
    const unsigned u = ldp32(p + i, lo);
    if constexpr (std::is_same<T, __half>::value) {
      const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&u));
      return pk_make(f.x, f.y);
    } else {
      const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u));
      return pk_make(f.x, f.y);
    }
  }
}
template <bool VEC, typename T>
__device__ __forceinline__ void st2(T* __restrict__ p, long long i, pk v, bool lo, bool hi) {
  if constexpr (VEC) {
    if (!lo) return;
    if constexpr (sizeof(T) == 4)
      *reinterpret_cast<unsigned long long*>(p + i) = v;
    else if constexpr (std::is_same<T, __half>::value)
      *reinterpret_cast<__half2*>(p + i) = __floats2half2_rn(pk_lo(v), pk_hi(v));
    else
      *reinterpret_cast<__nv_bfloat162*>(p + i) = __floats2bfloat162_rn(pk_lo(v), pk_hi(v));
  } else {
    if (lo) stf(p, i, pk_lo(v));
    if (hi) stf(p, i + 1, pk_hi(v));
  }
}
template <typename T>
__device__ __forceinline__ bool pair_aligned(const T* p) {
  return (reinterpret_cast<uintptr_t>(p) & (2 * sizeof(T) - 1)) == 0;
}

// Column x of one real tile of image `img` (forward-type ops) in the pairs
// distribution: out[r] = rows 2q, 2q + 1 (+ J r), zero outside the image.
// Tile origins are even (multiples of the even tile stride), so with even N
// and an aligned image every pair is one aligned access, wholly inside or
// wholly outside.
template <int M, typename T>
__device__ __forceinline__ void load_tile_column(const T* __restrict__ img, const TileRef& t, int x, int q,
                                                 pk (&out)[Quad<M>::R]) {
  constexpr int R = Quad<M>::R, J = Quad<M>::J;
  const int N = t.N;
  const int gx = t.x0 + x;
  if (!t.live || gx >= N) {
#pragma unroll
    for (int r = 0; r < R; ++r) out[r] = 0ull;
    return;
  }
  const T* base = img + t.on;
  const T* col = base + (long long)gx * N + t.y0 + 2 * q;
  const int rows = N - t.y0 - 2 * q;  // rows available from this thread's first element on
  if (!(N & 1) && pair_aligned(base)) {
    if (N - t.y0 >= M) {
#pragma unroll
      for (int r = 0; r < R; ++r) out[r] = ld2<true>(col, J * r, true, true);
    } else {
#pragma unroll
      for (int r = 0; r < R; ++r) out[r] = ld2<true>(col, J * r, J * r < rows, true);
    }
  } else {
#pragma unroll
    for (int r = 0; r < R; ++r) out[r] = ld2<false>(col, J * r, J * r < rows, J * r + 1 < rows);
  }
}

// The four columns 4 blk .. of the two real tiles of a single-field op, by
// bulk copies: column c of tile h lands at element (4 h + c) column pitches,
// a pitch of 8 (mod 32) words so that the pair reads are free of bank
// conflicts.  Needs 16-byte pieces: N and the tile origin multiples of 16
// bytes and an aligned image (else false, and nothing is issued).
template <int M, typename T>
__host__ __device__ constexpr int bulk_pitch() { return M + 32 / (int)sizeof(T); }
template <int M, typename T>
__device__ __forceinline__ bool load_columns_bulk(const T* const (&img)[2], const TileRef (&tr)[2], int blk,
                                                  GroupMem<M>& gm, cpk (&z)[Quad<M>::R]) {
  constexpr int R = Quad<M>::R, J = Quad<M>::J;
  constexpr int CP = bulk_pitch<M, T>();
  constexpr int EPC = 16 / (int)sizeof(T);
  static_assert(8 * CP * sizeof(T) <= landing_bytes<M>() && block_bytes<M>() <= landing_bytes<M>(), "the columns land in the exchange");
  T* st = reinterpret_cast<T*>(gm.ex);
  int rows[2], cols[2];
  bool ok = true;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int N = tr[h].N;
    rows[h] = max(0, min(M, N - tr[h].y0));
    cols[h] = tr[h].live ? max(0, min(kLines, N - tr[h].x0 - blk * kLines)) : 0;
    ok = ok && N % EPC == 0 && tr[h].y0 % EPC == 0 && (reinterpret_cast<uintptr_t>(img[h] + tr[h].on) & 15) == 0;
  }
  if (!ok) return false;
  gm.open();
  if (gm.leader()) {
    tc::mbar_expect_tx(gm.bar, (unsigned)((cols[0] * rows[0] + cols[1] * rows[1]) * sizeof(T)));
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const T* src = img[h] + tr[h].on + (long long)(tr[h].x0 + blk * kLines) * tr[h].N + tr[h].y0;
      for (int c = 0; c < (rows[h] ? cols[h] : 0); ++c, src += tr[h].N)
        tc::bulk_g2s(st + (kLines * h + c) * CP, src, (unsigned)(rows[h] * sizeof(T)), gm.bar);
    }
  }
  gm.wait(0);
  const T* c0 = st + gm.t.line * CP + 2 * gm.t.q;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int y = 2 * gm.t.q + J * r;
    z[r].re = gm.t.line < cols[0] && y < rows[0] ? swin2(c0 + J * r) : 0ull;
    z[r].im = gm.t.line < cols[1] && y < rows[1] ? swin2(c0 + kLines * CP + J * r) : 0ull;
  }
  return true;
}

// The field(s) of a single-field op at tile column x: the two tiles of a
// pair, or g and dg of one tile, as re / im.
template <int M, int OP, typename T>
__device__ __forceinline__ void load_column(const OpArgs& a, const Geom& g, int w, int blk, GroupMem<M>& gm,
                                            cpk (&z)[Quad<M>::R]) {
  constexpr int R = Quad<M>::R;
  constexpr bool PAIRS = OpTraits<OP>::PAIRS;
  static_assert(OpTraits<OP>::K == 1, "single-field ops");
  const TileRef tr[2] = {tile_of(g, PAIRS ? 2 * w : w), tile_of(g, PAIRS ? 2 * w + 1 : w)};
  const T* const img[2] = {static_cast<const T*>(a.E), static_cast<const T*>(PAIRS ? a.E : a.dE)};
  if (load_columns_bulk<M, T>(img, tr, blk, gm, z)) return;
  const int x = blk * kLines + gm.t.line;
  pk re[R], im[R];
  load_tile_column<M, T>(img[0], tr[0], x, gm.t.q, re);
  load_tile_column<M, T>(img[1], tr[1], x, gm.t.q, im);
#pragma unroll
  for (int r = 0; r < R; ++r) z[r] = cpk{re[r], im[r]};
}

// ---- image windows --------------------------------------------------------------------
// Columns of an image in shared memory, raw storage values: window column c
// <-> image column gx0 + c, element i <-> image row gya + i; out-of-image
// elements are zero (the central-difference rule).  The four columns of a
// group need the columns and rows around them for the central differences:
// kWinCols columns.  gya is the first row wanted rounded down to a multiple
// of the 16-byte chunk (at least of 2): a pair of rows (y, y + 1) of an even
// image row is one aligned access.  Column pitch: 8 (mod 32) 4-byte words, so
// the pair reads of a half-warp (four indices of four lines) fall on
// distinct banks.
constexpr int kWinCols = kLines + 2;
// Pitch that holds S + 2 rows from any start inside a chunk.
template <typename T>
__host__ __device__ constexpr int win_pitch(int S) {
  return sizeof(T) == 4 ? (S + 5 + 23) / 32 * 32 + 8 : (S + 9 + 47) / 64 * 64 + 16;
}
template <int M, typename T>
__host__ __device__ constexpr size_t win_bytes() { return (size_t)kWinCols * win_pitch<T>(M) * sizeof(T); }
// Bytes before a window that reads of the rows above the first output reach:
// less than e <= M / 2 elements.
template <int M>
__host__ __device__ constexpr size_t win_lead() { return 2 * (size_t)M; }

// What a launch knows of the images that its blocks stage: nothing; or that
// every column starts on 16 bytes, the erosion is at least 1 and the first row
// that a thread works on is even / odd in every tile (P3: even also means that
// every pair of outputs is one aligned store); or that N is odd (element-wise
// windows, single stores) and the erosion at least 1.  The kernels of the known
// forms hold neither the copies in other pieces nor the other stores and, of
// the 16-byte forms, the other parity.  The passes are short of instruction
// cache and registers, so the paths not taken cost: P3 of 150 image pairs at
// M = 512 177 -> 149 us (erosion 60), 241 -> 198 (15); of 600 at M = 256
// 179 -> 153 and 220 -> 189; forward of 100 images of 511, KW 31: 206 -> 193.
enum Form : int { kAny = 0, kEven = 1, kOdd = 2, kOddN = 3 };
__host__ __device__ constexpr bool rows16_form(int form) { return form == kEven || form == kOdd; }

// An issued window: `at` is the image row of element 0; the caller waits for
// it with window_wait.
struct Window {
  int at;
  bool bulk;   // copied by the TMA engine, on the group's barrier
  bool sync;   // elements written by the threads
};

// Elements [0, n) of the nc columns that bulk copies or window_pieces do not
// write (outside the image, or needed by no valid output): zero.  Columns c0 .. c1 - 1, elements r0 .. r1 - 1
// lie in the image.  Returns whether there are any.
template <int M, typename T>
__device__ __forceinline__ bool window_zero(int nc, int n, int c0, int c1, int r0, int r1, int HP, T* __restrict__ win) {
  constexpr int GT = Quad<M>::GT;
  const int t = threadIdx.x % GT;
  if (c1 - c0 == nc && r1 - r0 == n) return false;
  for (int c = 0; c < nc; ++c) {
    const bool in = c >= c0 && c < c1;
    for (int k = t; k < n; k += GT)
      if (!in || k < r0 || k >= r1) win[c * HP + k] = T(0.f);
  }
  return true;
}

// Columns [c0, c1) and elements [r0, r1) (whole pieces) of a window in
// asynchronous pieces of BYTES; 2: through registers, a batch of loads in
// flight, in aligned words (forward of 100 FP16 images of 511, KW 31: 262 us
// with single values, 195 so).  A column's asynchronous copies have no loop or
// address arithmetic between them, for the group's few warps wait on their
// issue and not on the memory (adjoint of one odd-N image, FP32, N = 257 to 1501:
// 3 % less device time); not in the last pass at M = 512, whose registers that
// takes (forward of one image of 777, KW 121: 20 -> 24 us).  The words come by
// predicated loads in the tangent-adjoint's first pass (one odd-N FP16 image, N =
// 257 to 1501: 3 % less); in the adjoint's they cost 1 %, in the last pass 4 %.
enum WindowUser : int { kLastPass = 0, kFirstPass = 1, kFirstPassTan = 2 };
template <int M, typename T, int BYTES, int USER>
__device__ __forceinline__ void window_pieces(const T* __restrict__ src, int N, int c0, int c1, int r0, int r1, int HP,
                                              T* __restrict__ win) {
  constexpr int E = BYTES / (int)sizeof(T) ? BYTES / (int)sizeof(T) : 1;
  constexpr int GT = Quad<M>::GT;
  const int t = threadIdx.x % GT;
  if constexpr (BYTES > 2) {
    const int k0 = r0 + E * t;
#pragma unroll 1
    for (int c = c0; c < c1; ++c) {
      const T* p = src + (long long)c * N + k0;
      unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(win + c * HP + k0));
      auto copy = [&](int i) {
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(d + i * BYTES * GT), "l"(p + i * E * GT),
                     "n"(BYTES)
                     : "memory");
      };
      if constexpr (USER != kLastPass || M < 512) {
#pragma unroll
        for (int i = 0; i < (win_pitch<T>(M) + E * GT - 1) / (E * GT); ++i)
          if (k0 + i * E * GT < r1) copy(i);
      } else {
#pragma unroll 4
        for (int k = k0; k < r1; k += E * GT, p += E * GT, d += BYTES * GT) copy(0);
      }
    }
  } else {
    // Four elements per thread and column from the aligned words around them,
    // where these lie wholly inside the column's elements; the up to four at
    // either end of a column one by one, each by a thread of its own.
    static_assert(win_pitch<T>(M) % 4 == 0, "8-byte stores");
    const int K0 = r0 & -4;
    const unsigned odd0 = (unsigned)(reinterpret_cast<uintptr_t>(src) >> 1);
    auto shift = [&](int c) { return (int)((odd0 + (unsigned)(c * N)) & 1); };  // of column c against the words
    constexpr int ENDS = (8 * kWinCols + GT - 1) / GT;
    T ev[ENDS];
    int ek[ENDS];  // window element, or -1
#pragma unroll
    for (int i = 0; i < ENDS; ++i) {
      const int j = (t + i * GT) & 7, c = (t + i * GT) >> 3, s = shift(c);
      const int first = min(K0 - s >= r0 ? K0 : K0 + 4, r1);             // the words begin
      const int last = max(K0 + ((r1 - s - K0) >> 2) * 4, first);        // and end here
      const int k = j < 4 ? r0 + j : last + j - 4;
      const bool on = c >= c0 && c < c1 && (j < 4 ? k < first : k < r1);
      ek[i] = on ? c * HP + k : -1;
      if (on) ev[i] = src[(long long)c * N + k];
    }
#pragma unroll 1
    for (int k = K0 + 4 * t; k < r1; k += 4 * GT) {
      unsigned w[kWinCols][3];
#pragma unroll
      for (int c = 0; c < kWinCols; ++c) {
        const int s = shift(c);
        const unsigned* q = reinterpret_cast<const unsigned*>(src + (long long)c * N + k - s);
        const bool on = c >= c0 && c < c1 && k - s >= r0 && k + 4 + s <= r1;
        if constexpr (USER == kFirstPassTan) {
          w[c][0] = ldp32(q, on);
          w[c][1] = ldp32(q + 1, on);
          w[c][2] = ldp32(q + 2, on && s);
        } else if (on) {
          w[c][0] = q[0];
          w[c][1] = q[1];
          if (s) w[c][2] = q[2];
        }
      }
#pragma unroll
      for (int c = 0; c < kWinCols; ++c) {
        const int s = shift(c);
        if (c >= c0 && c < c1 && k - s >= r0 && k + 4 + s <= r1)
          *reinterpret_cast<uint2*>(win + c * HP + k) =
              make_uint2(__funnelshift_r(w[c][0], w[c][1], 16 * s), __funnelshift_r(w[c][1], w[c][2], 16 * s));
      }
    }
#pragma unroll
    for (int i = 0; i < ENDS; ++i)
      if (ek[i] >= 0) win[ek[i]] = ev[i];
  }
}

// Starts the copy of nc (at most the group's threads) columns from gx0, of
// them those of `need`, and nr rows from gy0 of the N x N image at img (any of
// them outside the image; not live: nothing) on the group's barrier i.  edge: elements outside the image
// become zero; else they keep whatever the memory held (with erosion >= 1
// only values that are never stored read them, and zeroing them was the
// longest step of a tile at the image's edge).  One bulk copy per column where
// every 16-byte chunk lies wholly inside or outside the image (N a multiple
// of the chunk, an aligned image): a loop of 16-byte cp.async over the
// threads cost P3 and the adjoint's P1 several hundred instructions.  Else
// the threads copy the largest pieces that N and the image allow.  The group
// is past gm.open().  FORM: what the launch knows of the images (Form).
template <int M, int FORM, int USER, typename T>
__device__ __forceinline__ Window issue_window(const T* __restrict__ img, int N, bool live, int gx0, int nc, ColSpan need,
                                               int gy0, int nr, int HP, T* __restrict__ win, bool edge,
                                               const GroupMem<M>& gm, int i) {
  constexpr int EPC = 16 / (int)sizeof(T);
  constexpr int GT = Quad<M>::GT;
  static_assert(kWinCols <= GT, "one thread per column");
  const int t = threadIdx.x % GT;
  const int mis = (int)(reinterpret_cast<uintptr_t>(img) & 15) | (N * (int)sizeof(T));  // alignment of every column
  const int bytes = FORM == kOddN ? (int)sizeof(T) : FORM != kAny || !(mis & 15) ? 16 : !(mis & 7) ? 8 : !(mis & 3) ? 4 : 2;  // the piece that it allows
  const int E = max(bytes / (int)sizeof(T), 1);
  Window w;
  w.bulk = FORM != kOddN && live && bytes == 16;
  w.at = gy0 & -max(E, 2);
  w.sync = live && !w.bulk;
  if (!live) return w;  // (nothing reads the window of a dead tile)
  // whole pieces; elements r0 .. r1 - 1 and columns c0 .. c1 - 1 lie in the image
  const int n = (gy0 - w.at + nr + E - 1) & -E;
  const int r0 = max(0, -w.at), r1 = max(r0, min(n, N - w.at));
  const ColSpan cs = clip_span(need, gx0, N);
  const int c0 = cs.lo, c1 = cs.hi;
  const T* src = img + (long long)gx0 * N + w.at;  // (dereferenced inside the image only)
  if constexpr (FORM == kOddN) {
    window_pieces<M, T, (int)sizeof(T), USER>(src, N, c0, c1, r0, r1, HP, win);
    return w;
  }
  if (w.bulk) {
    const unsigned len = (unsigned)((r1 - r0) * sizeof(T));
    if (t == 0) tc::mbar_expect_tx(gm.bar + i, (unsigned)(c1 - c0) * len);
    __syncwarp();
    if (t >= c0 && t < c1 && len) tc::bulk_g2s(win + t * HP + r0, src + (long long)t * N + r0, len, gm.bar + i);
    if constexpr (FORM != kAny) return w;
  } else if (bytes == 8) {
    window_pieces<M, T, 8, USER>(src, N, c0, c1, r0, r1, HP, win);
  } else if (bytes == 4) {
    window_pieces<M, T, 4, USER>(src, N, c0, c1, r0, r1, HP, win);
  } else {
    window_pieces<M, T, 2, USER>(src, N, c0, c1, r0, r1, HP, win);
  }
  if (edge) w.sync |= window_zero<M, T>(nc, n, c0, c1, r0, r1, HP, win);
  return w;
}
// The window has arrived for every thread of the group (group-uniform).
template <int FORM, int M>
__device__ __forceinline__ void window_wait(const Window& w, GroupMem<M>& gm, int i) {
  if (FORM != kOddN && w.bulk)
    gm.wait(i);
  else if (!rows16_form(FORM))
    asm volatile("cp.async.wait_all;\n" ::: "memory");
  if (!rows16_form(FORM) && w.sync) group_sync<M>();
}

// This thread's column of one tile in a W- or N-sized array: rows y = 2q + l
// + J r of the tile column lie in the array for 0 <= rel + l + J r < cnt.
struct OutCol {
  bool on;        // the column lies in the array
  unsigned cnt;   // rows
  int rel;        // row 2q relative to the first
  long long off;  // element offset of row 2q in the batch array
};
// Adjoint-type fields h_x = v * df/dx, h_y = v * df/dy on the valid window,
// zero elsewhere (or dv * df/dx + v * d(df)/dx for the tangent-adjoint).
// Virtual coordinates are shifted by +e so that the full N x N output is the
// valid part of the convolution of the zero-extended (N + 2e)^2 field
// (srk_adj_load_tile, adjoint/srk_adjoint.cuh:169-200).
//
// Twice the central differences of a staged image at the pair of rows `row`,
// row + 1 of window column 1 (win: the column left of this thread's).  ODD:
// `row` is odd, the row pairs around it are aligned.
template <bool ODD, typename T>
__device__ __forceinline__ void diff2(const T* __restrict__ win, int HP, int row, pk& gx, pk& gy) {
  const T* cm = win + row;
  const T* cc = cm + HP;
  const T* cp = cc + HP;
  if constexpr (ODD) {
    const pk lm = swin2(cm - 1), lp = swin2(cm + 1), rm = swin2(cp - 1), rp = swin2(cp + 1);
    gx = pk_sub(pk_make(pk_hi(rm), pk_lo(rp)), pk_make(pk_hi(lm), pk_lo(lp)));
    gy = pk_sub(swin2(cc + 1), swin2(cc - 1));
  } else {
    gx = pk_sub(swin2(cp), swin2(cm));
    const pk c = swin2(cc);
    gy = pk_make(__fsub_rn(pk_hi(c), swin(cc - 1)), __fsub_rn(swin(cc + 2), pk_lo(c)));
  }
}

// v / 2 (the differences' factor; halving is exact) at this thread's rows of
// the valid-window column o, zero outside.
template <int M, typename T>
__device__ __forceinline__ void load_cotangent(const T* __restrict__ v, const TileRef& t, const OutCol& o,
                                               pk (&vv)[Quad<M>::R]) {
  constexpr int R = Quad<M>::R, J = Quad<M>::J;
  const pk half = pk_dup(0.5f);
  if (!((t.W | o.rel) & 1) && pair_aligned(v + t.ow)) {
#pragma unroll
    for (int r = 0; r < R; ++r)
      vv[r] = ld2<true>(v + o.off, J * r, o.on && (unsigned)(o.rel + J * r) < o.cnt, true);
  } else {
#pragma unroll
    for (int r = 0; r < R; ++r)
      vv[r] = ld2<false>(v + o.off, J * r, o.on && (unsigned)(o.rel + J * r) < o.cnt,
                         o.on && (unsigned)(o.rel + J * r + 1) < o.cnt);
  }
#pragma unroll
  for (int r = 0; r < R; ++r) vv[r] = pk_mul(vv[r], half);
}

// One tile's h_x, h_y in the re (LANE 0) or im (LANE 1) parts: v * gradient
// of the window wf, or (TAN) dv * gradient of wf + v * gradient of wd.  MASK:
// some of the group's values lie outside the valid window.
template <int M, typename T, bool TAN, int LANE, bool ODD, bool MASK>
__device__ __forceinline__ void adj_fields(const pk (&vv)[Quad<M>::R], const pk (&dv)[Quad<M>::R], const OutCol& o,
                                           const T* __restrict__ wf, const T* __restrict__ wd, int row,
                                           cpk (&hx)[Quad<M>::R], cpk (&hy)[Quad<M>::R]) {
  constexpr int R = Quad<M>::R, J = Quad<M>::J, HP = win_pitch<T>(M);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = J * r;
    pk gx, gy;
    diff2<ODD>(wf, HP, row + i, gx, gy);
    if constexpr (TAN) {
      pk dgx, dgy;
      diff2<ODD>(wd, HP, row + i, dgx, dgy);
      gx = pk_dot2(dv[r], gx, vv[r], dgx);
      gy = pk_dot2(dv[r], gy, vv[r], dgy);
    } else {
      gx = pk_mul(vv[r], gx);
      gy = pk_mul(vv[r], gy);
    }
    if constexpr (MASK) {
      // outside the valid window exactly zero, whatever the image holds there
      const bool lo = o.on && (unsigned)(o.rel + i) < o.cnt, hi = o.on && (unsigned)(o.rel + i + 1) < o.cnt;
      gx = pk_make(lo ? pk_lo(gx) : 0.f, hi ? pk_hi(gx) : 0.f);
      gy = pk_make(lo ? pk_lo(gy) : 0.f, hi ? pk_hi(gy) : 0.f);
    }
    (LANE ? hx[r].im : hx[r].re) = gx;
    (LANE ? hy[r].im : hy[r].re) = gy;
  }
}
template <int M, typename T, bool TAN, int LANE, int FORM>
__device__ __forceinline__ void adj_lane(const GroupMem<M>& gm, bool cols, const pk (&vv)[Quad<M>::R],
                                         const pk (&dv)[Quad<M>::R], const OutCol& o,
                                         const T* __restrict__ wf, const T* __restrict__ wd, int row,
                                         cpk (&hx)[Quad<M>::R], cpk (&hy)[Quad<M>::R]) {
  const int y0 = o.rel - 2 * gm.t.q;  // first tile row in the valid window (group-uniform, like `inside`)
  const bool inside = cols && y0 >= 0 && y0 + M <= (int)o.cnt;
  const bool odd = rows16_form(FORM) ? FORM == kOdd : row & 1;
  if (!inside) {
    if (odd)
      adj_fields<M, T, TAN, LANE, true, true>(vv, dv, o, wf, wd, row, hx, hy);
    else
      adj_fields<M, T, TAN, LANE, false, true>(vv, dv, o, wf, wd, row, hx, hy);
  } else if (odd) {
    adj_fields<M, T, TAN, LANE, true, false>(vv, dv, o, wf, wd, row, hx, hy);
  } else {
    adj_fields<M, T, TAN, LANE, false, false>(vv, dv, o, wf, wd, row, hx, hy);
  }
}

// h_x, h_y of the group's columns for both tiles of the pair.  Two windows at
// a time, in the exchange and the buffer: f of both tiles, or f and df of one
// tile after the other; the cotangents are loaded while they arrive.
template <int M, typename T, bool TAN, int FORM>
__device__ __forceinline__ void load_adj(const OpArgs& a, const Geom& g, int w, int blk, GroupMem<M>& gm,
                                         cpk (&hx)[Quad<M>::R], cpk (&hy)[Quad<M>::R]) {
  constexpr int HP = win_pitch<T>(M);
  static_assert(win_bytes<M, T>() <= landing_bytes<M>() && win_bytes<M, T>() <= block_bytes<M>(), "window size");
  const int x = blk * kLines + gm.t.line, q2 = 2 * gm.t.q;
  T* const w0 = reinterpret_cast<T*>(gm.ex);
  T* const w1 = reinterpret_cast<T*>(gm.buf);
  auto column = [&](const TileRef& t) {  // this thread's column of the tile in the valid window
    const int ox = t.x0 + x - 2 * a.e;
    OutCol o;
    o.on = t.live && (unsigned)ox < (unsigned)t.W;
    o.cnt = (unsigned)t.W;
    o.rel = t.y0 - 2 * a.e + q2;
    o.off = t.ow + (long long)ox * t.W + o.rel;
    return o;
  };
  auto stage = [&](const TileRef& t, const void* img, int i) {
    return issue_window<M, FORM, TAN ? kFirstPassTan : kFirstPass>(
        static_cast<const T*>(img) + t.on, t.N, t.live, t.x0 + blk * kLines - a.e - 1, kWinCols, ColSpan{0, kWinCols},
        t.y0 - a.e - 1, M + 2, HP, i ? w1 : w0, a.e < 1, gm, i);
  };
  auto inside = [&](const TileRef& t) {  // every column of the group lies in the valid window
    const int ox = t.x0 + blk * kLines - 2 * a.e;
    return t.live && ox >= 0 && ox + kLines <= t.W;
  };
  auto row = [&](const TileRef& t, const Window& wn) { return t.y0 - a.e + q2 - wn.at; };  // this thread's first row
  gm.open();
  const T* const f0 = w0 + gm.t.line * HP;
  const T* const f1 = w1 + gm.t.line * HP;
  if constexpr (TAN) {
    // One copy of the code for both tiles: the first tile's fields arrive in the
    // im parts and move to the re parts when the second's take their place.
    // The pass is short of instruction cache, most of all in the calls of a few
    // blocks: tangent-adjoint of N >= 2047 1 - 3 % faster, FP16 of N <= 1022 up to 8 %.
#pragma unroll
    for (int r = 0; r < Quad<M>::R; ++r) hx[r] = hy[r] = cpk{0ull, 0ull};
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
      const TileRef th = tile_of(g, 2 * w + h);
      const OutCol o = column(th);
      pk vv[Quad<M>::R], dv[Quad<M>::R];
      if (h) gm.open();  // the windows are read
      const Window f = stage(th, a.I, 0), d = stage(th, a.dI, 1);
      load_cotangent<M, T>(static_cast<const T*>(a.v), th, o, vv);
      load_cotangent<M, T>(static_cast<const T*>(a.dv), th, o, dv);
      window_wait<FORM>(f, gm, 0);
      window_wait<FORM>(d, gm, 1);
#pragma unroll
      for (int r = 0; r < Quad<M>::R; ++r) {
        hx[r].re = hx[r].im;
        hy[r].re = hy[r].im;
      }
      adj_lane<M, T, true, 1, FORM>(gm, inside(th), vv, dv, o, f0, f1, row(th, f), hx, hy);
    }
  } else {
    const TileRef tr[2] = {tile_of(g, 2 * w), tile_of(g, 2 * w + 1)};
    const OutCol o0 = column(tr[0]), o1 = column(tr[1]);
    pk v0[Quad<M>::R], v1[Quad<M>::R];
    const Window f = stage(tr[0], a.I, 0), s = stage(tr[1], a.I, 1);
    load_cotangent<M, T>(static_cast<const T*>(a.v), tr[0], o0, v0);
    load_cotangent<M, T>(static_cast<const T*>(a.v), tr[1], o1, v1);
    window_wait<FORM>(f, gm, 0);
    window_wait<FORM>(s, gm, 1);
    adj_lane<M, T, false, 0, FORM>(gm, inside(tr[0]), v0, v0, o0, f0, f0, row(tr[0], f), hx, hy);
    adj_lane<M, T, false, 1, FORM>(gm, inside(tr[1]), v1, v1, o1, f1, f1, row(tr[1], s), hx, hy);
  }
}

// ---- P1 ------------------------------------------------------------------------------------
// The transform of column x (ky = k_i + R m) -> S1[ky/4][x][ky%4].
template <int M>
__device__ __forceinline__ void p1_store(const float2 (&X)[Quad<M>::VPT], float2* __restrict__ S1k, int x, int q) {
  using Q = Quad<M>;
#pragma unroll
  for (int i = 0; i < Q::KPT; ++i) {
    const int k = q + Q::TPL * i;
    float2* dst = S1k + (size_t)(k >> 2) * (4 * M) + x * 4 + (k & 3);
#pragma unroll
    for (int m = 0; m < Q::J; ++m) __stcg(dst + (size_t)m * (Q::R / 4) * (4 * M), X[i * Q::J + m]);
  }
}

// P1: the group transforms columns 4 blk .. 4 blk + 3 of every field along y.
// OP_ADJ: TAN when dv and df are given.
template <int M, int OP, typename T, bool TAN = false, int FORM = kAny>
__device__ __forceinline__ void phase1(const OpArgs& a, const Geom& g, int w, int blk, float2* __restrict__ S1,
                                       GroupMem<M>& gm, const float4* __restrict__ tw) {
  using Q = Quad<M>;
  const QuadThread t = gm.t;
  const int x = blk * kLines + t.line;
  float2 X[Q::VPT];
  if constexpr (OP == OP_ADJ) {
    // both fields from one pass over the inputs; h_y waits in registers
    cpk hx[Q::R], hy[Q::R];
    load_adj<M, T, TAN, FORM>(a, g, w, blk, gm, hx, hy);
    // one copy of the transform: the pass is short of instruction cache
    // (adjoint N = 4096, KW = 61: 262 -> 242 us with P2's)
#pragma unroll 1
    for (int k = 0; k < 2; ++k) {
      fft_dit<M, false>(hx, X, gm.ex, tw, t);
      p1_store<M>(X, S1 + (size_t)k * M * M, x, t.q);
#pragma unroll
      for (int r = 0; r < Q::R; ++r) hx[r] = hy[r];
    }
  } else {
    cpk z[Q::R];
    load_column<M, OP, T>(a, g, w, blk, gm, z);
    fft_dit<M, false>(z, X, gm.ex, tw, t);
    p1_store<M>(X, S1, x, t.q);
  }
}

// ---- P2 ------------------------------------------------------------------------------------
// P2: rows ky = 4 blk .. 4 blk + 3: FFT along x, spectral map, inverse, keep
// the valid columns.
// The spectra are older than the pass before: ready() is called between their
// fetch and that of S1.
template <int M, int OP, typename F>
__device__ __forceinline__ void phase2(const float2* __restrict__ S1, float2* __restrict__ S2,
                                       const float4* __restrict__ Gx, const float4* __restrict__ Gy, int conjG,
                                       const Geom& g, int blk, GroupMem<M>& gm, const float4* __restrict__ tw,
                                       F&& ready) {
  using Q = Quad<M>;
  constexpr int K = OpTraits<OP>::K;
  constexpr unsigned BB = (unsigned)block_bytes<M>();
  const QuadThread t = gm.t;
  const int S = g.S, e = g.e, P = s2_pitch(S), xa = s2_first(e);
  const size_t row = (size_t)blk * (kLines * M);  // complex values before this block of rows
  const float4* gb = reinterpret_cast<const float4*>(gm.buf);
  // row ky of a staged S1 block: x = k_i + R m
  auto load = [&](const void* blkmem, float2 (&X)[Q::VPT]) {
    const float2* src = static_cast<const float2*>(blkmem) + t.line + 4 * t.q;
#pragma unroll
    for (int i = 0; i < Q::KPT; ++i)
#pragma unroll
      for (int m = 0; m < Q::J; ++m) X[i * Q::J + m] = src[4 * (Q::TPL * i + Q::R * m)];
  };
  // staged spectrum quad of kx = 2q, 2q + 1 (+ J r): quad 4 (q + J r / 2) + line of the block
  auto spec = [&](int r) {
    cpk v = cpk_load(gb[4 * t.q + t.line + r * (2 * Q::J)]);
    if (K == 2 && conjG) v.im = pk_neg(v.im);
    return v;
  };
  auto emit = [&](const float2 (&X)[Q::VPT], int l) {
    float2* dst0 = S2 + (size_t)l * M * P + (size_t)(blk * kLines + t.line) * 4;
#pragma unroll
    for (int i = 0; i < Q::KPT; ++i) {
      const int k = t.q + Q::TPL * i;
      float2* dst = dst0 + ((k >> 2) - (xa >> 2)) * (4 * M) + (k & 3);
#pragma unroll
      for (int m = 0; m < Q::J; ++m)
        if ((unsigned)(k + Q::R * m - e) < (unsigned)S) __stcg(dst + m * (Q::R / 4) * (4 * M), X[i * Q::J + m]);
    }
  };
  float2 X[Q::VPT];
  cpk z[Q::R], b[Q::R];
  gm.open();
  gm.fetch(1, gm.buf, Gx + row / 2, BB);
  ready();
  gm.fetch(0, gm.ex, S1 + row, BB);
  if constexpr (K == 1) {
    gm.wait(0);
    load(gm.ex, X);
    fft_dif_begin<M, false>(X, z, gm.ex, tw, t);
    fft_dif_finish<M, false>(z);
    // (one copy of the inverse at M = 512: 171 -> 167 us per 150 work tiles;
    // at M = 256 it spills, 159 -> 163 per 600)
#pragma unroll (M == 512 ? 1 : 2)
    for (int l = 0; l < 2; ++l) {
      gm.wait(1);
#pragma unroll
      for (int r = 0; r < Q::R; ++r) b[r] = cpk_mul<false>(z[r], spec(r));
      if (l == 0) {
        gm.open();
        gm.fetch(1, gm.buf, Gy + row / 2, BB);  // in flight during the first inverse
      }
      fft_dit<M, true>(b, X, gm.ex, tw, t);
      emit(X, l);
    }
  } else {
#pragma unroll
    for (int r = 0; r < Q::R; ++r) b[r] = cpk{0ull, 0ull};
#pragma unroll 1
    for (int k = 0; k < 2; ++k) {
      gm.wait(0);
      load(gm.ex, X);
      fft_dif_begin<M, false>(X, z, gm.ex, tw, t);
      if (k == 0) {
        gm.open();  // the exchange is read: the second field takes its place
        gm.fetch(0, gm.ex, S1 + (size_t)M * M + row, BB);
      }
      fft_dif_finish<M, false>(z);
      gm.wait(1);
#pragma unroll
      for (int r = 0; r < Q::R; ++r) {
        const cpk c = cpk_mul<false>(z[r], spec(r));
        b[r] = cpk{pk_add(b[r].re, c.re), pk_add(b[r].im, c.im)};
      }
      if (k == 0) {
        gm.open();
        gm.fetch(1, gm.buf, Gy + row / 2, BB);  // in flight during the second transform
      }
    }
    fft_dit<M, true>(b, X, gm.ex, tw, t);
    emit(X, 0);
  }
}

// ---- P3 ------------------------------------------------------------------------------------
template <int OP>
__host__ __device__ constexpr bool grad_op() { return OP == OP_FWD || OP == OP_JVP; }
// Operators whose epilogue multiplies by cotangents (W-sized images).
template <int OP>
__host__ __device__ constexpr bool cot_op() { return OP == OP_VJP_F || OP == OP_TANADJ_F; }
// Shared memory of a block in each pass (P1 of the single-field ops has one
// landing zone, P3 of the adjoint one field).
template <int OP>
__host__ __device__ constexpr bool p1_buf() { return OP == OP_ADJ; }
template <int M, int OP>
__host__ __device__ constexpr size_t p1_smem_bytes() { return groups_of<M>() * group_bytes<M, p1_buf<OP>()>(); }
template <int M>
__host__ __device__ constexpr size_t p2_smem_bytes() { return groups_of<M>() * group_bytes<M, true>(); }
template <int OP>
__host__ __device__ constexpr bool p3_buf() { return OpTraits<OP>::L == 2; }
template <int M, int OP>
__host__ __device__ constexpr size_t p3_smem_bytes() { return groups_of<M>() * group_bytes<M, p3_buf<OP>()>(); }

// Virtual coordinates are output coordinates + the erosion.
template <int M>
__device__ __forceinline__ OutCol out_col(const Geom& g, int erosion, const TileRef& tr, int x, int q, bool nsized) {
  OutCol o;
  const int ox = tr.x0 + x - erosion, oy = tr.y0 + g.e - erosion;  // output column, first valid output row
  o.on = tr.live && x >= g.e && x < g.e + g.S && ox < tr.Wout;
  o.cnt = (unsigned)max(0, min(g.S, tr.Wout - oy));
  o.rel = 2 * q - g.e;
  o.off = (nsized ? tr.on + (long long)ox * tr.N : tr.ow + (long long)ox * tr.W) + oy + o.rel;
  return o;
}
// Every pair of rows is one aligned access, wholly valid or wholly not (the
// first valid output row of a tile is even).
__device__ __forceinline__ bool out_even(const Geom& g, const TileRef& tr) { return !((g.e | tr.Wout) & 1); }

// Forward / tangent epilogue, round h, with the central differences read
// from the staged window.  FWD: round h finishes image h of the pair.  JVP:
// round 0 (window = f) leaves the f terms in u0.im, round 1 (window = df)
// adds the df terms.
template <int M, int OP, typename T, bool VEC>
__device__ __forceinline__ void grad_round(const OpArgs& a, const OutCol& o, int line, int q, int h, int row0,
                                           const T* __restrict__ win, int HP, cpk (&u0)[Quad<M>::R],
                                           const cpk (&u1)[Quad<M>::R]) {
  constexpr int R = Quad<M>::R, J = Quad<M>::J;
  // row0: window element of tile row 2q
  const T* cm = win + line * HP + row0;  // image column gx - 1
  const T* cc = cm + HP;                 // gx
  const T* cp = cc + HP;                 // gx + 1
  T* __restrict__ out = static_cast<T*>(a.out0) + o.off;
  T* __restrict__ UX = a.out_ux ? static_cast<T*>(a.out_ux) + o.off : nullptr;
  T* __restrict__ UY = a.out_uy ? static_cast<T*>(a.out_uy) + o.off : nullptr;
  const pk half = pk_dup(0.5f);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = J * r;
    const bool lo = (unsigned)(o.rel + i) < o.cnt;
    const bool hi = VEC ? lo : (unsigned)(o.rel + i + 1) < o.cnt;
    // every row is computed (no branch between the shared-memory reads of
    // the rows); rows outside the outputs read neighbouring shared memory
    // (win_lead) and are not stored
    const pk dx = pk_sub(swin2(cp + i), swin2(cm + i));
    const pk c = swin2(cc + i);
    const pk dy = pk_make(__fsub_rn(pk_hi(c), swin(cc + i - 1)), __fsub_rn(swin(cc + i + 2), pk_lo(c)));
    // the differences' factor 1/2 is applied once, at the end: halving is exact
    if constexpr (OP == OP_FWD) {
      const pk ux = h ? u0[r].im : u0[r].re, uy = h ? u1[r].im : u1[r].re;
      if (UX) st2<VEC>(UX, i, ux, lo, hi);
      if (UY) st2<VEC>(UY, i, uy, lo, hi);
      st2<VEC>(out, i, pk_mul(pk_dot2(ux, dx, uy, dy), half), lo, hi);
    } else {
      // srk_tangent_combine (tan_tanadj/srk_tangent.cuh:28-52):
      // dh = Im(zx) fx + Im(zy) fy + Re(zx) dfx + Re(zy) dfy
      if (h == 0)
        u0[r].im = pk_dot2(u0[r].im, dx, u1[r].im, dy);
      else
        st2<VEC>(out, i, pk_mul(pk_fma(u1[r].re, dy, pk_fma(u0[r].re, dx, u0[r].im)), half), lo, hi);
    }
  }
}

// Epilogue of the cotangent ops, from the staged window(s) of the cotangent
// (element `row` = tile row 2q of this line's column).  VJP (f): w = u * v of
// image h; tangent-adjoint (f): w = dlam * Re + lam * Im.  ODD: row is odd.
template <int M, int OP, typename T, bool VEC, bool ODD>
__device__ __forceinline__ void cot_epilogue(const OpArgs& a, const OutCol& o, int h, const T* __restrict__ v,
                                             const T* __restrict__ dv, const cpk (&u0)[Quad<M>::R],
                                             const cpk (&u1)[Quad<M>::R]) {
  constexpr int R = Quad<M>::R, J = Quad<M>::J;
  float* __restrict__ WX = static_cast<float*>(a.out0) + o.off;
  float* __restrict__ WY = static_cast<float*>(a.out1) + o.off;
  auto pair = [](const T* p) { return ODD ? pk_make(swin(p), swin(p + 1)) : swin2(p); };
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = J * r;
    const bool lo = (unsigned)(o.rel + i) < o.cnt;
    const bool hi = VEC ? lo : (unsigned)(o.rel + i + 1) < o.cnt;
    const pk vv = pair(v + i);
    pk wx, wy;
    if constexpr (OP == OP_VJP_F) {
      wx = pk_mul(h ? u0[r].im : u0[r].re, vv);
      wy = pk_mul(h ? u1[r].im : u1[r].re, vv);
    } else {
      const pk dd = pair(dv + i);
      wx = pk_dot2(dd, u0[r].re, vv, u0[r].im);
      wy = pk_dot2(dd, u1[r].re, vv, u1[r].im);
    }
    st2<VEC>(WX, i, wx, lo, hi);
    st2<VEC>(WY, i, wy, lo, hi);
  }
}

// Epilogue of the adjoint: the full N x N output of image h.
template <int M, typename T, bool VEC>
__device__ __forceinline__ void adj_epilogue(const OpArgs& a, const OutCol& o, int h, const cpk (&u)[Quad<M>::R]) {
  constexpr int R = Quad<M>::R, J = Quad<M>::J;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = J * r;
    const bool lo = (unsigned)(o.rel + i) < o.cnt;
    const bool hi = VEC ? lo : (unsigned)(o.rel + i + 1) < o.cnt;
    st2<VEC>(static_cast<T*>(a.out0) + o.off, i, h ? u[r].im : u[r].re, lo, hi);
  }
}

// S2 layouts P3 reads: the engine's, first column xa = s2_first(e), or the
// tensor-core row pass's (hybrid.cu): first column e, the lines of column
// block b rotated by b.
enum S2Layout : int { kS2Engine = 0, kS2Rotated = 1 };

// P3: columns 4 blk .. of S2: inverse FFT along ky, epilogue.
template <int M, int OP, typename T, int S2L = kS2Engine, int FORM = kAny>
__device__ __forceinline__ void phase3(const float2* __restrict__ S2, const OpArgs& a, const Geom& g, int w, int blk,
                                       GroupMem<M>& gm, const float4* __restrict__ tw) {
  using Q = Quad<M>;
  constexpr int L = OpTraits<OP>::L;
  constexpr bool GRAD = grad_op<OP>(), WIN = L == 2;
  static_assert(GRAD || cot_op<OP>() || L == 1, "two-field ops have windows");
  constexpr unsigned BB = (unsigned)block_bytes<M>();
  // rows below the last output reach less than e elements past a window
  static_assert(!WIN || (win_bytes<M, T>() + 2 * win_lead<M>() <= landing_bytes<M>() &&
                          win_bytes<M, T>() + win_lead<M>() <= block_bytes<M>()),
                "the windows reuse the buffer (behind the exchange) and the exchange");
  const QuadThread t = gm.t;
  const int P = s2_pitch(g.S);
  const int xg = (S2L == kS2Rotated ? g.e : s2_first(g.e)) + blk * kLines;  // the group's first tile column
  const int x = xg + t.line;
  auto tile_h = [&](int h) { return tile_of(g, OpTraits<OP>::PAIRS ? 2 * w + h : w); };
  // the windows take the place of the second field (once every thread has
  // read it) and of the last exchange: f (and df) around the group's columns,
  // or v (lam and dlam) at the group's output columns
  T* win[2] = {reinterpret_cast<T*>(gm.buf), reinterpret_cast<T*>(reinterpret_cast<unsigned char*>(gm.ex) + win_lead<M>())};
  Window wn[2];
  const int HP = win_pitch<T>(g.S);
  // a column slab's buffer holds only the columns that valid outputs read;
  // slabs come by tile tables, which are kAny, and images of the other forms
  // are whole (5000 images of 512, erosion 60, with the span in every form:
  // 7534 -> 7610 us)
  auto need = [&](int halo) {
    return FORM == kAny ? window_span(xg, g.e, g.S, halo) : ColSpan{0, kLines + 2 * halo};
  };
  auto window = [&](int h) {
    const TileRef tr = tile_h(h);
    if constexpr (GRAD) {
      const T* img = static_cast<const T*>(OP == OP_FWD || h == 0 ? a.I : a.dI) + tr.on;
      wn[h] = issue_window<M, FORM, kLastPass>(img, tr.N, tr.live, tr.x0 + xg - 1, kWinCols, need(1),
                                 tr.y0 + g.e - 1, g.S + 2, HP, win[h], a.e < 1, gm, 1 - h);
    } else {
      const T* img = static_cast<const T*>(OP == OP_VJP_F || h == 0 ? a.v : a.dv) + tr.ow;
      wn[h] = issue_window<M, FORM, kLastPass>(img, tr.W, tr.live, tr.x0 + xg - a.e, kLines, need(0), tr.y0, g.S, HP, win[h], false,
                                 gm, 1 - h);
    }
  };
  // column x of a staged S2 block: ky = k_i + R m
  auto load = [&](const void* blkmem, float2 (&X)[Q::VPT]) {
    const float2* src = static_cast<const float2*>(blkmem) + t.line;
#pragma unroll
    for (int i = 0; i < Q::KPT; ++i)
#pragma unroll
      for (int m = 0; m < Q::J; ++m) {
        const int ky = t.q + Q::TPL * i + Q::R * m;
        X[i * Q::J + m] = src[4 * (S2L == kS2Rotated ? (ky + blk) & (M - 1) : ky)];
      }
  };
  // One copy of the transform for both fields at M = 512, images in 16-byte
  // columns.  Forward of 150 work tiles 159 -> 148 us with pairs of stores, 208 ->
  // 198 with single ones (24 bytes of spills); the cotangent operators spill 24
  // bytes with one copy and 32 - 40 with two and take the same time (VJP of 64
  // images of 512, KW 61: 278.6 against 277.7 us, KW 121: 259.3 against 260.1).  At
  // M = 256 and 128 two copies are as fast or faster (153 against 156, 161 against
  // 162), and beside the copies in smaller pieces of kAny and kOddN one copy costs
  // more spills than it saves (177 against 181, 241 against 269).
  constexpr bool LOOP = M == 512 && rows16_form(FORM);
  float2 X[Q::VPT];
  cpk u0[Q::R], u1[Q::R];
  gm.open();
  gm.fetch(0, gm.ex, S2 + (size_t)blk * (kLines * M), BB);
  if constexpr (L == 2) gm.fetch(1, gm.buf, S2 + (size_t)M * P + (size_t)blk * (kLines * M), BB);
  if constexpr (L == 2 && LOOP) {
#pragma unroll 1
    for (int l = 0; l < 2; ++l) {
      gm.wait(l);
      load(l ? static_cast<const void*>(gm.buf) : gm.ex, X);
      tc::fence_async_smem();  // the buffer's next copy comes after these reads
      fft_dif_begin<M, true>(X, u1, gm.ex, tw, t, [&] {
        if (l) window(0);
      });
      if (l) {
        gm.open();  // the exchange is read: window 1 takes its place
        window(1);
      }
      fft_dif_finish<M, true>(u1);
      if (l == 0) {
#pragma unroll
        for (int r = 0; r < Q::R; ++r) u0[r] = u1[r];
      }
    }
  } else {
    gm.wait(0);
    load(gm.ex, X);
    fft_dif_begin<M, true>(X, u0, gm.ex, tw, t);
    if constexpr (L == 2) {
      fft_dif_finish<M, true>(u0);
      gm.wait(1);
      load(gm.buf, X);
      tc::fence_async_smem();  // the buffer's next copy comes after these reads
      fft_dif_begin<M, true>(X, u1, gm.ex, tw, t, [&] {
        window(0);
      });
      gm.open();  // the exchange is read: window 1 takes its place
      window(1);
      fft_dif_finish<M, true>(u1);
    }
  }
  if constexpr (WIN) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      window_wait<FORM>(wn[h], gm, 1 - h);
      if (OP == OP_TANADJ_F && h == 0) continue;  // both windows at once
      const TileRef tr = tile_h(h);
      const OutCol o = out_col<M>(g, a.e, tr, x, t.q, false);
      if (!o.on) continue;
      if constexpr (GRAD) {
        const int row0 = tr.y0 + 2 * t.q - wn[h].at;
        auto al = [&](const void* p) { return !p || pair_aligned(static_cast<const T*>(p) + tr.ow); };
        const bool vec = FORM == kAny ? out_even(g, tr) && al(a.out0) && al(a.out_ux) && al(a.out_uy) : FORM == kEven;
        if (vec)
          grad_round<M, OP, T, true>(a, o, t.line, t.q, h, row0, win[h], HP, u0, u1);
        else
          grad_round<M, OP, T, false>(a, o, t.line, t.q, h, row0, win[h], HP, u0, u1);
      } else {
        constexpr int H1 = OP == OP_TANADJ_F ? 0 : 1;  // the window of v
        const int hv = H1 ? h : 0;
        const int row = tr.y0 + o.rel - wn[hv].at, drow = tr.y0 + o.rel - wn[1].at;
        const T* v = win[hv] + t.line * HP + row;
        const T* dv = win[1] + t.line * HP + drow;
        const bool vec = FORM == kAny ? out_even(g, tr) && pair_aligned(static_cast<const float*>(a.out0) + tr.ow) &&
                                            pair_aligned(static_cast<const float*>(a.out1) + tr.ow)
                                      : FORM == kEven;
        const bool even = rows16_form(FORM) ? FORM == kEven : (row & 1) == 0;  // (both windows start at even rows)
        if (even && vec)
          cot_epilogue<M, OP, T, true, false>(a, o, h, v, dv, u0, u1);
        else if (even)
          cot_epilogue<M, OP, T, false, false>(a, o, h, v, dv, u0, u1);
        else
          cot_epilogue<M, OP, T, false, true>(a, o, h, v, dv, u0, u1);
      }
    }
  } else {
    fft_dif_finish<M, true>(u0);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const TileRef tr = tile_h(h);
      const OutCol o = out_col<M>(g, a.e, tr, x, t.q, true);
      if (!o.on) continue;
      if (FORM == kEven || (out_even(g, tr) && pair_aligned(static_cast<const T*>(a.out0) + tr.on)))
        adj_epilogue<M, T, true>(a, o, h, u0);
      else
        adj_epilogue<M, T, false>(a, o, h, u0);
    }
  }
}

// ---- three-launch schedule (one kernel per phase over a chunk of WTs) ------
// The kernels of one call run back to back on one stream by programmatic
// dependent launch: a kernel's blocks are placed while the last blocks of the
// one before finish, set up their barriers and wait there (grid_wait: every
// kernel before is complete and visible).  Every kernel waits before it lets
// the next one start (grid_next), so at most two kernels overlap and what a
// kernel does before its wait may use anything older than its predecessor.
// A no-op where the launch is an ordinary one.  Only tables that are older
// than the call (twiddles) are read through the read-only path.
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Index of this thread's group in its block.
template <int M>
__device__ __forceinline__ int group_index() { return threadIdx.x / Quad<M>::GT; }

// TAN (adjoint-type op of the tangent-adjoint, dv and df given) is chosen by
// the launch.
template <int M, int OP, typename T, bool TAN = false, int FORM = kAny>
__global__ void __launch_bounds__(kThreads, OP == OP_ADJ && M > 128 ? SRK_P1_ADJ_MIN_BLOCKS : SRK_P1_MIN_BLOCKS)
k_p1(OpArgs a, Geom g, const float4* __restrict__ tw, int w0, float2* __restrict__ scratch) {
  extern __shared__ __align__(16) unsigned char sm[];
  GroupMem<M> gm = group_mem<M, p1_buf<OP>()>(sm, g.err);
  const int wl = blockIdx.y;
  grid_wait();
  grid_next();
  phase1<M, OP, T, TAN, FORM>(a, g, w0 + wl, blockIdx.x * groups_of<M>() + group_index<M>(),
                        scratch + wl * wt_elems<M, OP>(g.S), gm, tw);
}

template <int M, int OP>
__global__ void __launch_bounds__(kThreads, M > 128 ? SRK_P2_MIN_BLOCKS : SRK_SMALL_MIN_BLOCKS)
k_p2(float2* __restrict__ scratch, const float4* __restrict__ Gx, const float4* __restrict__ Gy, int conjG, Geom g,
     const float4* __restrict__ tw) {
  extern __shared__ __align__(16) unsigned char sm[];
  GroupMem<M> gm = group_mem<M, true>(sm, g.err);
  float2* base = scratch + blockIdx.y * wt_elems<M, OP>(g.S);
  phase2<M, OP>(base, base + s1_elems<M, OP>(), Gx, Gy, conjG, g, blockIdx.x * groups_of<M>() + group_index<M>(), gm,
                tw, [] {
                  grid_wait();
                  grid_next();
                });
}

template <int M, int OP, typename T, int S2L = kS2Engine, int FORM = kAny>
__global__ void __launch_bounds__(kThreads, M == 128                ? SRK_SMALL_MIN_BLOCKS
                                           : OpTraits<OP>::L == 1 ? SRK_P3_ADJ_MIN_BLOCKS
                                                                  : SRK_P3_MIN_BLOCKS)
k_p3(float2* __restrict__ scratch, OpArgs a, Geom g, const float4* __restrict__ tw, int w0) {
  extern __shared__ __align__(16) unsigned char sm[];
  GroupMem<M> gm = group_mem<M, p3_buf<OP>()>(sm, g.err);
  const int wl = blockIdx.y;
  const int nblk = s2_blocks(g.S, S2L == kS2Rotated ? 0 : g.e - s2_first(g.e));
  const int blk = blockIdx.x * groups_of<M>() + group_index<M>();
  grid_wait();
  grid_next();
  if (blk < nblk)
    phase3<M, OP, T, S2L, FORM>(scratch + wl * wt_elems<M, OP>(g.S) + s1_elems<M, OP>(), a, g, w0 + wl, blk, gm, tw);
}

// Failure-path self test of the passes' waits: a group waits, with a short
// limit, for a copy that is never issued; `out` counts the threads that go on.
static __global__ void __launch_bounds__(kThreads)
k_copy_wait_selftest(unsigned int* err, unsigned long long limit, unsigned int* out) {
  extern __shared__ __align__(16) unsigned char sm[];
  GroupMem<512> gm = group_mem<512, false>(sm, err);
  gm.open();
  gm.wait(0, limit);
  gm.open();
  atomicAdd(out, 1u);
}

// ---- persistent schedule ---------------------------------------------------------
// One launch processes every WT.  Work is a ticket queue of rounds; round r
// holds the P1 units of WT r, the P2 units of WT r-lag and the P3 units of
// WT r-2*lag.  A WT's scratch lives in slot w mod nslot of a small ring that
// stays in L2.  Per-slot counters (monotonic over the slot's reuses) order
// the phases:
//   P1(w) needs c2[slot] >= gen*n2       (previous user's P2 done reading S1)
//   P2(w) needs c1[slot] >= (gen+1)*n1   (its S1 complete)
//           and c3[slot] >= gen*n3       (previous user's P3 done reading S2)
//   P3(w) needs c2[slot] >= (gen+1)*n2   (its S2 complete)
// S1 and S2 are stored by ordinary stores and fetched by bulk copies, which
// read global memory through the async proxy: the counters' release and
// acquire order ordinary accesses only, so every thread fences its stores
// before the release and the copying threads fence after the acquire
// (fence_async_global).  Between launches the kernel boundary does that.
// Every dependency points to a smaller ticket, and a ticket is only ever held
// by a running CTA (a CTA holds at most its current ticket and one
// prefetched larger one), so the smallest unfinished ticket can always
// proceed.  The lag and the ring size only decide how often a unit finds its
// dependency not yet met.  Waits are bounded anyway: a wait that exceeds
// `spin_limit` polls sets ctl->abort (with the place in ctl->where) and every
// CTA returns.
constexpr int kMaxSlots = 32;

struct Ctl {
  unsigned int ticket;
  unsigned int abort;
  unsigned int where;
  unsigned int pad;
  unsigned long long spins;  // polls that found a dependency unmet (diagnostic)
  unsigned int c1[kMaxSlots], c2[kMaxSlots], c3[kMaxSlots];
};

struct PersistParams {
  int lag;        // rounds between the phases of one WT
  int nslot;      // scratch ring slots (> lag)
  int prefetch;   // fetch the next ticket while running the current one
  int pad;
  unsigned long long spin_limit;
};

__device__ __forceinline__ unsigned int ld_acquire(const unsigned int* p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Thread-0 wait: returns false if the kernel must stop.
__device__ __forceinline__ bool wait_geq(const unsigned int* p, unsigned int target, unsigned long long limit,
                                         Ctl* ctl, unsigned int where, unsigned long long& spins) {
  unsigned long long it = 0;
  while (ld_acquire(p) < target) {
    if (ld_acquire(&ctl->abort)) return false;
    if (++it > limit) {
      atomicExch(&ctl->where, where);
      atomicExch(&ctl->abort, 1u);
      return false;
    }
    __nanosleep(32);
  }
  spins += it;
  return true;
}

template <int M, int OP, typename T>
__global__ void __launch_bounds__(kThreads, SRK_P2_MIN_BLOCKS)
k_persist(OpArgs a, Geom g, const float4* __restrict__ Gx, const float4* __restrict__ Gy, int conjG,
          const float4* __restrict__ tw, float2* __restrict__ scratch, int nwt, Ctl* ctl, PersistParams pp) {
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ int s_t[2];
  constexpr int NG = groups_of<M>();
  GroupMem<M> gm = group_mem<M, true>(sm, g.err);
  const int nblk = s2_blocks(g.S, g.e - s2_first(g.e));
  const int n1 = M / unit_lines<M>(), n2 = n1, n3 = (nblk + NG - 1) / NG;
  const int round = n1 + n2 + n3;
  const int lag = pp.lag, nslot = pp.nslot;
  const long long total = (long long)(nwt + 2 * lag) * round;
  const size_t slot_elems = wt_elems<M, OP>(g.S);
  unsigned long long spins = 0;
  if (threadIdx.x == 0) s_t[0] = (int)atomicAdd(&ctl->ticket, 1u);
  __syncthreads();
  int cur = s_t[0];
  while (cur < total) {
    unsigned int nxt = 0;
    if (threadIdx.x == 0 && pp.prefetch) nxt = atomicAdd(&ctl->ticket, 1u);
    const int r = cur / round, u = cur - (cur / round) * round;
    int phase, w, unit;
    if (u < n1) { phase = 1; w = r; unit = u; }
    else if (u < n1 + n2) { phase = 2; w = r - lag; unit = u - n1; }
    else { phase = 3; w = r - 2 * lag; unit = u - n1 - n2; }
    const bool live = (w >= 0 && w < nwt);
    const int slot = live ? w % nslot : 0;
    const unsigned int gen = live ? (unsigned int)(w / nslot) : 0u;
    if (threadIdx.x == 0) {
      bool ok = ld_acquire(&ctl->abort) == 0u;
      if (ok && live) {
        if (phase == 1) ok = wait_geq(&ctl->c2[slot], gen * n2, pp.spin_limit, ctl, 1, spins);
        else if (phase == 2) ok = wait_geq(&ctl->c1[slot], (gen + 1) * n1, pp.spin_limit, ctl, 2, spins) &&
                                  wait_geq(&ctl->c3[slot], gen * n3, pp.spin_limit, ctl, 3, spins);
        else ok = wait_geq(&ctl->c2[slot], (gen + 1) * n2, pp.spin_limit, ctl, 4, spins);
      }
      s_t[1] = ok ? 1 : 0;
    }
    __syncthreads();
    // a thread of this block that gave up a wait for a copy has left (perhaps
    // the one that draws the tickets): end the launch
    bool stopped = false;
#pragma unroll
    for (int i = 0; i < NG; ++i)
      stopped |= *const_cast<volatile unsigned*>(stop_word<M>(sm + i * group_bytes<M, true>())) != 0u;
    if (stopped) {
      atomicExch(&ctl->where, kStopSite);
      atomicExch(&ctl->abort, 1u);
    }
    if (!s_t[1] || stopped) break;
    if (live) {
      tc::fence_async_global();  // the copies come after the stores just acquired
      float2* base = scratch + (size_t)slot * slot_elems;
      const int blk = unit * NG + group_index<M>();
      if (phase == 1) {
        if (OP == OP_ADJ && a.dI != nullptr)
          phase1<M, OP, T, OP == OP_ADJ>(a, g, w, blk, base, gm, tw);
        else
          phase1<M, OP, T>(a, g, w, blk, base, gm, tw);
      } else if (phase == 2) {
        phase2<M, OP>(base, base + s1_elems<M, OP>(), Gx, Gy, conjG, g, blk, gm, tw, [] {});
      } else if (blk < nblk) {
        phase3<M, OP, T>(base + s1_elems<M, OP>(), a, g, w, blk, gm, tw);
      }
      tc::fence_async_global();  // this thread's scratch stores, before other blocks' copies
    }
    __syncthreads();  // every thread's scratch stores of this unit are issued
    if (threadIdx.x == 0) {
      if (live) {
        __threadfence();
        atomicAdd(phase == 1 ? &ctl->c1[slot] : phase == 2 ? &ctl->c2[slot] : &ctl->c3[slot], 1u);
      }
      s_t[0] = pp.prefetch ? (int)nxt : (int)atomicAdd(&ctl->ticket, 1u);
    }
    __syncthreads();
    cur = s_t[0];
  }
  if (threadIdx.x == 0 && spins) atomicAdd(&ctl->spins, spins);
}

// Bounded-wait self test: thread 0 of one CTA waits for a counter that
// nothing increments; the wait must give up and raise the abort flag.
static __global__ void k_wait_selftest(Ctl* ctl, unsigned long long spin_limit) {
  unsigned long long spins = 0;
  if (threadIdx.x == 0) wait_geq(&ctl->c1[0], 1u, spin_limit, ctl, 99, spins);
}

// dL/df = D_x^T(wx) + D_y^T(wy) on N x N, with wx, wy given on the W x W
// window (zero outside); adjoint of the central difference
// (adjointWrtI_kernel, adjoint/srk_adjoint.cuh:25-59).  With ux, uy, v
// given instead (the reference contract) w = u*v is formed on the fly.
// Every element is loaded once: a warp owns kStencilWarpRows rows and marches
// over the columns, CX per step with every load of a step in flight; the
// column neighbours of wx stay in registers, the row neighbours of wy come
// from the neighbouring lanes (the first and last lane load one row more).
// With one row per lane the march is bound by instruction issue (N = 4096:
// 58 us FP32, the same at FP16 storage), so a lane owns a pair of rows, one
// aligned access each, where the window's rows allow (W even, aligned
// arrays; the pairs start at even window rows), and single rows in strips of
// 32 elsewhere (`rows` per warp).  N = 4096 from u and v: 62 us with blocks that loaded
// every neighbour, 47 us (5.6 TB/s) so, FP16 38; B = 256, N = 512 from wx,
// wy: 141 -> 108 us (6.3 TB/s).  16 columns a block: 32 and 64 measured 3 to
// 10 % slower (fewer blocks in flight), 8 for small images.
constexpr int kStencilThreads = 128;
constexpr int kStencilWarpRows = 64;
constexpr int kStencilCols = 16;  // columns of a block
// Row blocks of an image: pairs start at even window rows, one row above the
// image for odd erosion.
__host__ __device__ inline int stencil_row_blocks(int N, int e, int rows = kStencilWarpRows) {
  return (N + (e & 1) + kStencilThreads / 32 * rows - 1) / (kStencilThreads / 32 * rows);
}

template <bool PAIR>
struct StencilVal;  // a lane's value(s): one float or a packed pair
template <>
struct StencilVal<false> {
  using V = float;
  template <typename T>
  static __device__ __forceinline__ V load(const T* p, bool on) { return ldp(p, on); }
  static __device__ __forceinline__ V mul(V a, V b) { return __fmul_rn(a, b); }
  static __device__ __forceinline__ V sub(V a, V b) { return __fsub_rn(a, b); }
  static __device__ __forceinline__ V add(V a, V b) { return __fadd_rn(a, b); }
  static __device__ __forceinline__ V half() { return 0.5f; }
  // rows above and below, h: the edge lanes' halo value
  static __device__ __forceinline__ void neighbours(V y, float h, int lane, V& up, V& dn) {
    up = __shfl_up_sync(0xffffffffu, y, 1);
    dn = __shfl_down_sync(0xffffffffu, y, 1);
    if (lane == 0) up = h;
    if (lane == 31) dn = h;
  }
};
template <>
struct StencilVal<true> {
  using V = pk;
  template <typename T>
  static __device__ __forceinline__ V load(const T* p, bool on) { return ld2<true>(p, 0, on, on); }
  static __device__ __forceinline__ V mul(V a, V b) { return pk_mul(a, b); }
  static __device__ __forceinline__ V sub(V a, V b) { return pk_sub(a, b); }
  static __device__ __forceinline__ V add(V a, V b) { return pk_add(a, b); }
  static __device__ __forceinline__ V half() { return pk_dup(0.5f); }
  static __device__ __forceinline__ void neighbours(V y, float h, int lane, V& up, V& dn) {
    float u = __shfl_up_sync(0xffffffffu, pk_hi(y), 1), d = __shfl_down_sync(0xffffffffu, pk_lo(y), 1);
    if (lane == 0) u = h;
    if (lane == 31) d = h;
    up = pk_make(u, pk_lo(y));
    dn = pk_make(pk_hi(y), d);
  }
};

// Columns [gx0, gx1) of the lane's row gy (PAIR: rows gy, gy + 1).
template <typename T, bool FROM_U, bool PAIR>
__device__ __forceinline__ void adj_wrt_f_strip(const float* __restrict__ wx, const float* __restrict__ wy,
                                                const T* __restrict__ v, const T* __restrict__ ux,
                                                const T* __restrict__ uy, long long wo, long long oo, int N, int W,
                                                int e, int gx0, int gx1, int gy, T* __restrict__ out) {
  using O = StencilVal<PAIR>;
  using V = typename O::V;
  constexpr int CX = FROM_U ? 4 : 8;  // 8 loads a step with two arrays, 4 with three (47 us; 54 with 8)
  const int lane = threadIdx.x & 31;
  const int oy = gy - e;  // the lane's (first) row in the window; PAIR: even, W even
  const int hd = lane == 0 ? -1 : PAIR ? 2 : 1;
  const bool rin = (unsigned)oy < (unsigned)W, hin = (lane == 0 || lane == 31) && (unsigned)(oy + hd) < (unsigned)W;
  const long long base = wo + oy;
  int c = gx0 - e;  // window column of the first output
  // window columns read: up to that of gx1 (a slab's arrays end there)
  const int cend = gx1 - e;
  auto in = [&](int k) { return (unsigned)k < (unsigned)W && k <= cend; };
  auto load_x = [&](int k, V& vk) -> V {
    const bool on = rin && in(k);
    const long long i = base + (long long)k * W;
    if constexpr (FROM_U) {
      vk = O::load(v + i, on);
      return O::mul(O::load(ux + i, on), vk);
    } else {
      return O::load(wx + i, on);
    }
  };
  const bool o0 = (unsigned)gy < (unsigned)N, o1 = PAIR && (unsigned)(gy + 1) < (unsigned)N;
  const bool opair = PAIR && o0 && o1 && !((N | gy) & 1) && pair_aligned(out + oo);
  V vc{};  // v at column c (FROM_U)
  V xm = load_x(c - 1, vc), x0 = load_x(c, vc);
  for (int gx = gx0; gx < gx1; gx += CX, c += CX) {
    V xn[CX], vn[CX], y[CX];
    float h[CX];
#pragma unroll
    for (int j = 0; j < CX; ++j) {
      xn[j] = load_x(c + 1 + j, vn[j]);
      const bool cin = in(c + j) && c + j < cend;
      const long long i = base + (long long)(c + j) * W;
      if constexpr (FROM_U) {
        y[j] = O::load(uy + i, rin && cin);
        h[j] = __fmul_rn(ldp(uy + i + hd, hin && cin), ldp(v + i + hd, hin && cin));
      } else {
        y[j] = O::load(wy + i, rin && cin);
        h[j] = ldp(wy + i + hd, hin && cin);
      }
    }
#pragma unroll
    for (int j = 0; j < CX; ++j) {
      if constexpr (FROM_U) y[j] = O::mul(y[j], j ? vn[j - 1] : vc);
      V up, dn;
      O::neighbours(y[j], h[j], lane, up, dn);
      const V left = j == 0 ? xm : j == 1 ? x0 : xn[j - 2];
      const V r = O::add(O::mul(O::sub(left, xn[j]), O::half()), O::mul(O::sub(up, dn), O::half()));
      if (gx + j < gx1) {
        T* __restrict__ p = out + oo + (long long)(gx + j) * N + gy;
        if constexpr (PAIR) {
          if (opair)
            st2<true>(p, 0, r, true, true);
          else
            st2<false>(p, 0, r, o0, o1);
        } else if (o0) {
          stf(p, 0, r);
        }
      }
    }
    xm = xn[CX - 2];
    x0 = xn[CX - 1];
    if constexpr (FROM_U) vc = vn[CX - 1];
  }
}
// Columns [gx0, gx1) of row block rb of one image.
template <typename T, bool FROM_U>
__device__ __forceinline__ void adj_wrt_f_block(const float* __restrict__ wx, const float* __restrict__ wy,
                                                const T* __restrict__ v, const T* __restrict__ ux,
                                                const T* __restrict__ uy, long long wo, long long oo, int N, int W,
                                                int e, int gx0, int gx1, int rb, int rows, T* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const int r0 = (rb * (kStencilThreads / 32) + (threadIdx.x >> 5)) * rows - (e & 1);  // the warp's first row
  if (r0 >= N) return;
  bool pair = !(W & 1);
  if constexpr (FROM_U)
    pair = pair && pair_aligned(v + wo) && pair_aligned(ux + wo) && pair_aligned(uy + wo);
  else
    pair = pair && pair_aligned(wx + wo) && pair_aligned(wy + wo);
  if (pair) {
    adj_wrt_f_strip<T, FROM_U, true>(wx, wy, v, ux, uy, wo, oo, N, W, e, gx0, gx1, r0 + 2 * lane, out);
  } else {
#pragma unroll 1
    for (int s = 0; s < rows; s += 32)
      adj_wrt_f_strip<T, FROM_U, false>(wx, wy, v, ux, uy, wo, oo, N, W, e, gx0, gx1, r0 + s + lane, out);
  }
}

// Uniform batch: grid (row blocks, columns / cols, B).
template <typename T, bool FROM_U>
__global__ void __launch_bounds__(kStencilThreads)
k_adj_wrt_f(const float* __restrict__ wx, const float* __restrict__ wy, const T* __restrict__ v,
            const T* __restrict__ ux, const T* __restrict__ uy, int N, int W, int e, int cols, int rows,
            T* __restrict__ out) {
  const int gx0 = blockIdx.y * cols;
  const int b = blockIdx.z;
  grid_wait();
  grid_next();
  adj_wrt_f_block<T, FROM_U>(wx, wy, v, ux, uy, (long long)b * W * W, (long long)b * N * N, N, W, e, gx0,
                             min(gx0 + cols, N), blockIdx.x, rows, out);
}

// The same for a ragged batch or a column slab over the pixel columns
// [cx0, cx1) of each image, the blocks of image b starting at rimg[b].blk0.
template <typename T, bool FROM_U>
__global__ void __launch_bounds__(kStencilThreads)
k_adj_wrt_f_rag(const float* __restrict__ wx, const float* __restrict__ wy, const T* __restrict__ v,
                const T* __restrict__ ux, const T* __restrict__ uy, const RagImage* __restrict__ rimg, int B, int e,
                T* __restrict__ out) {
  grid_wait();
  grid_next();
  int lo = 0, hi = B - 1;
  const int blk = blockIdx.x;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (rimg[mid].blk0 <= blk) lo = mid; else hi = mid - 1;
  }
  const RagImage im = rimg[lo];
  const int nby = stencil_row_blocks(im.N, e);
  const int k = blk - im.blk0;
  const int gx0 = im.cx0 + (k / nby) * kStencilCols;
  adj_wrt_f_block<T, FROM_U>(wx, wy, v, ux, uy, im.ow, im.on, im.N, im.W, e, gx0, min(gx0 + kStencilCols, im.cx1),
                             k % nby, kStencilWarpRows, out);
}

}  // namespace srk
