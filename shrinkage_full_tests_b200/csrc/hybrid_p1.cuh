// hybrid_p1.cuh — the column pass (P1) of the tensor-core row schedule
// (SRK_SCHEDULE_TENSOR_ROWS): the same column FFT along y as the engine's P1
// at M = 512, but its output is written as FP16 planes, one per (ky, part),
// in the layout the tensor-core row pass (hybrid.cu) reads with TMA:
//   planes[((ky * 2 + part) * c + wl) * M + x]      (part 0 = re, 1 = im),
// c = work tiles in the chunk, wl = work tile within the chunk.  Each CTA
// transforms 8 consecutive columns (two groups of four), stages their values
// [ky][part][8] in shared memory and writes them with TMA stores (one
// 16-byte piece per (ky, part) plane row).  Used for the pair ops (OP_FWD,
// OP_VJP_F: two images per work tile) where the column DFT of
// hybrid_p1g.cuh does not apply, and by the refit pass.
#pragma once
#include <cuda.h>

#include "engine.cuh"
#include "hybrid_scale.cuh"
#include "internal.h"
#include "tc.cuh"

namespace srk {

// Shared memory of k_p1h / k_p1h_refit, all dynamic (static __shared__
// variables would move the dynamic block off the 128-byte boundary the TMA
// stores need): the engine's phase layout, the FP16 staging block
// [M][2][kP1hCols], then the refit's work list (P1hAux).
// 8 columns per CTA (16 bytes per (ky, part)): measured 0.66 ms per 500 work
// tiles against 0.81 ms with 16 columns (whole 32-byte sectors, but 3 CTAs
// per SM and twice the transforms per line).
constexpr int kP1hCols = 8;
constexpr int kP1hThreads = kP1hCols / kLines * Quad<kHybM>::GT;
// Byte offset of the staging block (128-byte aligned: the source of TMA stores).
__host__ __device__ constexpr size_t p1h_stage_offset() { return (kP1hCols / kLines * group_bytes<kHybM, false>() + 127) / 128 * 128; }
struct P1hAux {
  int cnt[kP1hThreads / 32];  // refit: flagged work tiles per warp
  int list[kP1hThreads];      // refit: the flagged work tiles of one group
};
__host__ __device__ constexpr size_t p1h_aux_offset() {
  return p1h_stage_offset() + (size_t)kHybM * 2 * kP1hCols * sizeof(__half);
}
__host__ __device__ constexpr size_t p1h_smem_bytes() { return p1h_aux_offset() + sizeof(P1hAux); }
// Planes written per TMA store (box {8 columns, 1 work tile, kP1hBox planes}).
constexpr int kP1hBox = 256;

// The column pass of the kP1hCols columns kP1hCols * xb .. of work tile wl
// (w = w0 + wl): FFTs along y, values times sp rounded to FP16 and staged
// [plane = 2 ky + part][8 columns], written by TMA stores (box {8 columns, 1
// work tile, kP1hBox planes}: the TMA engine writes the 1024 16-byte row
// pieces the threads would otherwise scatter).  Block-uniform arguments; the
// twiddle quads are tw.  With zmax given, each warp folds the max |Z| of its
// unscaled values into zmax[wl] (one atomic per warp, float bits).  Ends with
// the stores complete and the block synchronised (the staging block may be
// reused).
template <int OP, typename T>
__device__ __forceinline__ void p1h_cols(const CUtensorMap* pmap, const OpArgs& a, const Geom& g, unsigned char* sm,
                                         GroupMem<kHybM>& gm, const float4* __restrict__ tw, int w0, int wl, int xb,
                                         float sp, unsigned int* zmax, unsigned int* err) {
  constexpr int M = kHybM;
  using Q = Quad<M>;
  constexpr int NU = kP1hCols / kLines;  // groups of four columns per CTA
  static_assert(kP1hThreads == NU * Q::GT && Q::KPT == 1, "one group of four columns per group of threads");
  const QuadThread t = gm.t;
  const int u = group_index<M>();
  __half* st = reinterpret_cast<__half*>(sm + p1h_stage_offset());
  const int w = w0 + wl;
  cpk z[Q::R];
  float2 X[Q::VPT];
  load_column<M, OP, T>(a, g, w, xb * NU + u, gm, z);
  fft_dit<M, false>(z, X, gm.ex, tw, t);
  float m = 0.f;
#pragma unroll
  for (int i = 0; i < Q::J; ++i) {
    const int ky = t.q + Q::R * i;
    m = fmaxf(m, fmaxf(fabsf(X[i].x), fabsf(X[i].y)));
    st[(ky * 2 + 0) * kP1hCols + u * kLines + t.line] = __float2half_rn(X[i].x * sp);
    st[(ky * 2 + 1) * kP1hCols + u * kLines + t.line] = __float2half_rn(X[i].y * sp);
  }
  if (zmax) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0 && m > 0.f) atomicMax(zmax + wl, __float_as_uint(m));
  }
  tc::fence_async_smem();
  __syncthreads();
  if (threadIdx.x == 0) {
    bool stopped = false;  // a group whose columns never came has left: the planes keep what they held
    for (int i = 0; i < NU; ++i)
      stopped |= *const_cast<volatile unsigned*>(stop_word<M>(sm + i * group_bytes<M, false>())) != 0u;
    if (stopped) {
      // nothing to store
    } else if ((tc::smem_u32(st) & 127u) == 0) {
      for (int p0 = 0; p0 < 2 * M; p0 += kP1hBox) tc::tma_store_3d(pmap, xb * kP1hCols, wl, p0, st + p0 * kP1hCols);
      tc::bulk_commit();
    } else {
      atomicCAS(err, 0u, 15u);  // the TMA source must sit on 128 bytes: record, store nothing
    }
    tc::bulk_wait_all();
  }
  __syncthreads();
}

// First column pass of a chunk: every work tile's planes at scale 1, and
// zmax[wl] = max |Z| of work tile wl (float bits; zeroed before the launch).
// Grid (M / kP1hCols, c).
template <int OP, typename T>
__global__ void __launch_bounds__(kP1hThreads, 4)
k_p1h(const __grid_constant__ CUtensorMap pmap, OpArgs a, Geom g, const float4* __restrict__ tw, int w0,
      unsigned int* __restrict__ zmax, unsigned int* err) {
  static_assert(OpTraits<OP>::K == 1, "single-field ops only");
  extern __shared__ __align__(128) unsigned char smh[];
  GroupMem<kHybM> gm = group_mem<kHybM, false>(smh, g.err);
  p1h_cols<OP, T>(&pmap, a, g, smh, gm, tw, w0, blockIdx.y, blockIdx.x, 1.f, zmax, err);
}

// Refit: the work tiles whose zmax lies outside the range kept at scale 1
// (plane_exp != 0) are transformed again, their planes written at scale
// 2^plane_exp.  Persistent over the (work tile, column block) units of the
// flagged work tiles, in order; every block scans zmax (c words) for them, so
// a chunk without such work tiles costs one short launch.
template <int OP, typename T>
__global__ void __launch_bounds__(kP1hThreads, 4)
k_p1h_refit(const __grid_constant__ CUtensorMap pmap, OpArgs a, Geom g, const float4* __restrict__ tw, int w0, int c,
            const unsigned int* __restrict__ zmax, unsigned int* err) {
  constexpr int NX = kHybM / kP1hCols;  // column blocks per work tile
  extern __shared__ __align__(128) unsigned char smh[];
  GroupMem<kHybM> gm = group_mem<kHybM, false>(smh, g.err);
  P1hAux* aux = reinterpret_cast<P1hAux*>(smh + p1h_aux_offset());
  int* cnt = aux->cnt;
  int* list = aux->list;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  long long rank0 = 0;  // flagged work tiles before this group of kP1hThreads
  for (int b0 = 0; b0 < c; b0 += kP1hThreads) {
    const int wl = b0 + threadIdx.x;
    const bool f = wl < c && plane_exp(__ldg(zmax + wl)) != 0;
    const unsigned bal = __ballot_sync(0xffffffffu, f);
    if (lane == 0) cnt[warp] = __popc(bal);
    __syncthreads();
    int before = 0, total = 0;
    for (int i = 0; i < kP1hThreads / 32; ++i) {
      before += i < warp ? cnt[i] : 0;
      total += cnt[i];
    }
    if (f) list[before + __popc(bal & ((1u << lane) - 1u))] = wl;
    __syncthreads();
    for (int k = 0; k < total; ++k) {
      const int wk = list[k];
      const float sp = ldexpf(1.f, plane_exp(__ldg(zmax + wk)));
      for (int xb = 0; xb < NX; ++xb) {
        if ((int)(((rank0 + k) * NX + xb) % gridDim.x) != (int)blockIdx.x) continue;
        p1h_cols<OP, T>(&pmap, a, g, smh, gm, tw, w0, wk, xb, sp, nullptr, err);
      }
    }
    rank0 += total;
    __syncthreads();  // cnt and list are rewritten by the next group
  }
}

}  // namespace srk
