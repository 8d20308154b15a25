// The decode step's packed matvecs for up to 16 fp32 activation rows per launch part (nb_chain_linear), and the embedding that
// opens the step (nb_chain_embed).  The reference runs the same products one fused matvec per linear with element-wise launches
// between them (inference/triton_kernel.py:240-256, inference/generate_torch.py:109-117).
//
// A step is a chain of dependent launches of a few microseconds, so what is between the products counts as much as they do:
//  * A linear's activations arrive as the two fp16 terms the tensor cores take, written by the launch before in the layout that
//    is read here (nb_chain.cuh), so staging them is a copy.  The launch before has also added its result to the residual stream
//    and multiplied it by the norm's weight; the norm's scale is one factor on this linear's sums, from the partial sums of
//    squares that the launch before left per row tile.  (Every CTA computing all of that for itself took 1.5 - 2 us a launch for
//    one row, and grew with the rows.)
//  * Weights do not depend on earlier launches: a CTA's share of them, one bulk copy per row tile, is requested before the
//    dependency wait, and the matrix two linears ahead is brought into L2.
//  * The units of a CTA are dealt to its warps in equal runs across its row tiles, so no warp waits at a tile's end; the parts of
//    a tile meet in shared memory behind one barrier.
//  * Where the staged rows do not fit beside the weights, a cluster of S CTAs shares its row tiles: every CTA takes K / S columns
//    of all of them and pushes its parts into the shared memory of the CTA that finishes the tile.
//  * Plain rows of up to 16 may come against the packed matrix itself (kRaw): what is written to it is what the next call reads, and
//    nothing has to be made or kept beside it.  Unpacking costs a unit about 55 clocks more than the copy's selector words, and the
//    products wait for all of a CTA's weights (2560 x 6912, 16 bf16 rows 11.3 us against 9.5 over the copy and 13.9 for nb_gemv;
//    2560 x 2560, 8 rows 5.8, 4.8, 7.8; 13824 x 2560, 16 fp32 rows 24.6, 21.3, 35.9).  With a barrier per tile and an arrival per copying
//    thread on it 12.7, 6.6.
//  * Column 2r + s of the MMAs carries term s of activation row r: one product covers four fp32 rows.
// Decode step of the 2.2B decoder with 12 layers (us), matvecs that stage the rows themselves -> this: 1 sequence 437 -> 384, 2:
// 539 -> 448, 8: 665 -> 498, 16 (a matvec over the packed bytes and launches between): 1523 -> 943 over the packed matrix, rows
// given plainly and normed before they are split (934 over the copy; 865 with terms, which keep fewer bits of small rows).  17 and
// more rows stay on the tcgen05 kernel (32: 1121, here 1460).  For one sequence a layer's 28 us are four times 1.3 us from the end of a launch
// to the next one's first dependent instruction, 12.5 us of products (66 clocks per unit and SM against 54 without copies; down
// projections wait for the 12 SMs with two tiles), 4.4 us of attention and the rest staging and sums.  Measured and not kept:
// 12 or 16 warps so that the next launch's CTA is resident early (391 -> 421, 442), clusters of 2 or 4 for balance (no
// difference: the cluster's barriers take what the balance gains).
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

#include "nb_chain.cuh"
#include "nb_common.cuh"
#include "nb_device.cuh"
#include "nb_host.h"
#include "nb_launch.cuh"

namespace nb {

constexpr int kCW = 24;                     // warps per CTA
constexpr int kCThreads = kCW * 32;
constexpr int kChainBulk = 128;             // 256-byte blocks of staged activations from which on they come as bulk copies: fewer wait
                                            // less as 16-byte ones, as bulk copies queue behind the weights' (a row of 2560 0.3 against
                                            // 1.5 us behind the launch before), many have too many instructions (8 rows of 2560: a
                                            // layer 41 -> 44 us)
constexpr int kChainTiles = 16;             // row tiles of a CTA in one launch
constexpr uint32_t kChainSpin = 1u << 22;

__device__ __forceinline__ bool chain_wait(uint64_t* bar, uint32_t parity, int* status) {
  for (uint32_t i = 0; i < kChainSpin; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  atomicExch(status, (int)NB_ERR_TIMEOUT);
  return false;
}

struct ChainParams {
  const uint8_t* w;           // stream layout, or (kRaw) the packed rows themselves
  const uint8_t* xt;          // activations as terms
  const float* ss;            // (M, ss_n) partial sums of squares of the rows in front of the norm (null: no norm)
  void* y;                    // NB_CHAIN_STORE: (M, N) of type y_dtype
  uint8_t* yt;                // the other two: terms of the next linear's activations (null: none)
  float* res;                 // NB_CHAIN_RESIDUAL: (M, N), updated in place
  const float* w_next;        // ... the next norm's weight; with x and ss that of the norm of the rows themselves
  float* ss_out;              // ... (M, N / 16) partial sums of squares of the new rows (null: none)
  const uint8_t* ahead;       // weights of the launch behind (null: none), `ahead_step` bytes per CTA
  int* status;
  unsigned ahead_bytes, ahead_step;
  const void* x;              // plain activations (M, K) of type x_dtype instead of the terms (null: none)
  int x_dtype, y_dtype;
  int N, bpr, M, mode, ss_n;
  float eps;
  int m_part, parts;          // activation rows per part of the launch, parts
  int clusters, lg_split;     // clusters of one part, of 2^lg_split CTAs each
  unsigned rcp_clusters, rcp_kc, rcp_kc1;     // ceil(2^32 / v) of the clusters, the smaller and the larger share of a row's blocks
  int tile0, n_tiles;         // row tiles of this launch
  int w_bytes, J;             // room for weights; partial results per tile and CTA
};
// What only packed rows need; the other kernels' launches do not carry it.
struct ChainRaw {
  const uint8_t* cb;          // codebooks of type cb_dtype, cb_block bytes per block
  int cb_dtype, cb_block;
  int idx_stride, cb_stride;  // bytes from row to row in shared memory
};
struct ChainCopy {};
template <bool kRaw> using ChainLayout = std::conditional_t<kRaw, ChainRaw, ChainCopy>;
// v / d for v * d < 2^32 (d == 1 has no 32-bit reciprocal)
__device__ __forceinline__ int div_rcp(int v, int d, unsigned rcp) { return d == 1 ? v : (int)__umulhi((unsigned)v, rcp); }

// 32 packed indices -> four selector words, nibble i of word j the index at position 8j + i: the order of the stream layout.
// Fields move apart half by half; what moves is picked by a mask and moved by a multiply-add.
template <int BITS> __device__ __forceinline__ void packed_selectors(const uint8_t* src, uint32_t (&U)[4]) {
  const uint32_t* w = reinterpret_cast<const uint32_t*>(src);
  if (BITS == 4) {
    const uint4 v = *reinterpret_cast<const uint4*>(src);
    U[0] = v.x; U[1] = v.y; U[2] = v.z; U[3] = v.w;
  } else if (BITS == 3) {
    const uint32_t w0 = w[0], w1 = w[1], w2 = w[2];
    U[0] = w0 & 0xFFFFFFu;
    U[1] = funnel_r(w0, w1, 24) & 0xFFFFFFu;
    U[2] = funnel_r(w1, w2, 16) & 0xFFFFFFu;
    U[3] = w2 >> 8;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      U[j] = mad_lo(U[j] & 0xFFF000u, 15u, U[j]);
      U[j] = mad_lo(U[j] & 0x0FC00FC0u, 3u, U[j]);
      U[j] += U[j] & 0x38383838u;
    }
  } else {
    const uint2 v = *reinterpret_cast<const uint2*>(src);
    U[0] = v.x & 0xFFFFu; U[1] = v.x >> 16; U[2] = v.y & 0xFFFFu; U[3] = v.y >> 16;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      U[j] = mad_lo(U[j] & 0xFF00u, 255u, U[j]);
      U[j] = mad_lo(U[j] & 0x00F000F0u, 15u, U[j]);
      U[j] = mad_lo(U[j] & 0x0C0C0C0Cu, 3u, U[j]);
    }
  }
}

// 16 rows x 128 weights against CG groups of eight columns.  kRaw: `ub` and `cb` are this lane's indices and codebook of row g, those
// of row g + 8 eight strides on.
template <int BITS, int CG, bool kRaw>
__device__ __forceinline__ void chain_unit(const ChainLayout<kRaw>& raw, const uint8_t* ub, const uint8_t* cb, const uint8_t* const (&x)[CG], int lane,
                                           const ByteShift& sm, uint32_t act, uint4 (&last)[1], float (&c)[CG == 1 ? 2 : CG][4]) {
  const int g = lane >> 2, t = lane & 3;
  uint32_t UA[4], UB[4], TA[BITS == 4 ? 8 : 4], TB[BITS == 4 ? 8 : 4];
  if constexpr (kRaw) {
    packed_selectors<BITS>(ub, UA);
    packed_selectors<BITS>(ub + 8 * raw.idx_stride, UB);
    make_table<BITS>(cb, raw.cb_dtype, true, TA);
    make_table<BITS>(cb + 8 * raw.cb_stride, raw.cb_dtype, true, TB);
  } else {
    unit_selectors(ub, lane, 0, UA);
    unit_selectors(ub, lane, 1, UB);
    unit_table<BITS>(ub, g, TA);
    unit_table<BITS>(ub, g + 8, TB);
  }
#pragma unroll
  for (int uu = 0; uu < 4; ++uu) {
    uint4 xq[CG];
#pragma unroll
    for (int j = 0; j + 1 < CG; ++j) xq[j] = *reinterpret_cast<const uint4*>(x[j] + ((uu ^ t ^ (g & 1)) << 4));
    lds_if(last[0], x[CG - 1] + ((uu ^ t ^ (g & 1)) << 4), act);
    xq[CG - 1] = last[0];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint32_t a0, a1, a2, a3;
      lookup4_pairs<BITS>(h ? UA[uu] >> 16 : UA[uu], TA, sm, a0, a2);
      lookup4_pairs<BITS>(h ? UB[uu] >> 16 : UB[uu], TB, sm, a1, a3);
#pragma unroll
      for (int j = 0; j < CG; ++j) mma_16816(c[CG == 1 ? h : j], a0, a1, a2, a3, h ? xq[j].z : xq[j].x, h ? xq[j].w : xq[j].y);
    }
  }
}

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ void st_cluster_f32(uint32_t local, uint32_t rank, float v) {
  uint32_t remote;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(remote), "f"(v) : "memory");
}

// 1 / rms of row `r` from its partial sums, by a whole warp, in a fixed order: the same bits in every CTA.
__device__ __forceinline__ float row_scale(const ChainParams& p, int r, int lane) {
  const float* sq = p.ss + (size_t)r * p.ss_n;
  float s = 0.f;
#pragma unroll 6
  for (int q = lane; q < p.ss_n; q += 32) s += __ldcg(sq + q);
  return 1.0f / sqrtf(warp_sum(s) / (float)(p.bpr * kBlock) + p.eps);
}

// Shared memory: the CTA's units, tile after tile (kRaw: a tile's 16 rows of indices, then of codebooks) | staged columns (XT m_part of kc_max * 256 bytes) | partial
// results [own tile][CTA][J][row][16] of the tiles this CTA finishes.
// kPlain: plain activations.  (As a run-time choice the code that converts and norms them, and the packed rows' parameters in every
// launch, cost launches whose rows are terms 0.2 us each: a step of the 2.2B decoder with 12 layers 398 us, now 384.)
template <int BITS, int CG, int XT, bool kCluster, bool kRaw, bool kPlain>
__global__ void __launch_bounds__(kCThreads, 1) chain_kernel(const ChainParams p, const ChainLayout<kRaw> raw) {
  constexpr int kUnit = StreamUnit<BITS>::kBytes;
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ uint64_t s_bar[kChainTiles], s_xbar;
  __shared__ float s_scale[16];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const ByteShift sm = byte_shift();
  const int lg = kCluster ? p.lg_split : 0, S = 1 << lg, rank = (int)blockIdx.x & (S - 1), cl = (int)blockIdx.x >> lg;
  const int part = p.parts == 1 ? 0 : cl % p.parts, ci = p.parts == 1 ? cl : cl / p.parts;
  const int T = div_rcp(p.n_tiles - ci + p.clusters - 1, p.clusters, p.rcp_clusters);      // tiles ci, ci + clusters, ..
  const int k0 = p.bpr * rank >> lg, kc = (p.bpr * (rank + 1) >> lg) - k0, kc_max = (p.bpr + S - 1) >> lg;
  // ---- the weights do not depend on the launch before: one copy per row tile
  if (tid == 0) {
    mbar_init(&s_xbar, 1);
    for (int i = 0; !kRaw && i < T; ++i) mbar_init(&s_bar[i], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    const uint8_t* src = p.w + ((size_t)(p.tile0 + ci) * p.bpr + k0) * kUnit;
    for (int i = 0; !kRaw && i < T; ++i) {
      mbar_arrive_expect_tx(&s_bar[i], (uint32_t)(kc * kUnit));
      bulk_g2s(smem + (size_t)i * kc * kUnit, src, (uint32_t)(kc * kUnit), &s_bar[i]);
      src += (size_t)p.clusters * p.bpr * kUnit;
    }
  }
  if constexpr (kRaw) {                                     // thread after thread takes the next piece of a row: indices, then codebooks
    const int idx_pieces = kc * BITS, cb_piece = raw.cb_block >= 16 ? 16 : 8, per_row = idx_pieces + kc * raw.cb_block / cb_piece;
    const int rows = kCThreads / per_row, rest = kCThreads - rows * per_row;
    int r = tid / per_row, c = tid - r * per_row;
    for (;;) {
      if (c >= per_row) { c -= per_row; ++r; }
      if (r >= 16 * T) break;
      const int i = r >> 4, row = r & 15, tile = p.tile0 + ci + i * p.clusters;
      const int n = p.mode == NB_CHAIN_SWIGLU ? tile * 8 + (row & 7) + (row & 8 ? p.N >> 1 : 0) : min(tile * 16 + row, p.N - 1);
      const size_t block = (size_t)(n * p.bpr + k0);
      uint8_t* dst = smem + i * 16 * (raw.idx_stride + raw.cb_stride);
      if (c < idx_pieces) {
        cp_async16(dst + row * raw.idx_stride + 16 * c, p.w + block * (16 * BITS) + 16 * c);
      } else {
        dst += 16 * raw.idx_stride + row * raw.cb_stride + cb_piece * (c - idx_pieces);
        const uint8_t* src = raw.cb + block * raw.cb_block + cb_piece * (c - idx_pieces);
        if (cb_piece == 16) cp_async16(dst, src);
        else cp_async8(dst, src);
      }
      r += rows;
      c += rest;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  const int row0 = part * p.m_part, m = min(p.m_part, p.M - row0);
  const unsigned rcp_kc = kc == kc_max ? p.rcp_kc1 : p.rcp_kc;
  const int U = T * kc;                                     // units of this CTA, tile after tile
  const int ua = U * warp / kCW, ub = U * (warp + 1) / kCW; // this warp's run
  uint8_t* x_s = smem + p.w_bytes;
  float* parts = reinterpret_cast<float*>(x_s + (size_t)XT * p.m_part * kc_max * 256);
  const int own = (T + S - 1 - rank) >> lg;                 // tiles rank, rank + S, .. of the cluster's are finished here
  const int slot = 16 * m;
  const int i_first = div_rcp(ua, kc, rcp_kc), kk_first = ua - i_first * kc;
  // the warp's first tile may have been begun by warps before it: their parts come first (later tiles it begins itself;
  // with fewer units than warps a warp has one unit or none, and a unit's place in its tile is the place of its part)
  const int j_first = U <= kCW ? kk_first : kk_first > 0 ? warp - (int)((unsigned)((i_first * kc + 1) * kCW - 1) / (unsigned)U) : 0;
  __syncthreads();
  if (kCluster) asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");      // this CTA runs: others may write to its shared memory
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;");

  const uint8_t* xt = p.xt + ((size_t)(2 * row0) * p.bpr + k0) * 256;
  const bool bulk = !kPlain && (kRaw || 2 * m * kc > kChainBulk);      // (a wait for 16-byte copies would be one for the weights')
  if (kPlain) {                                             // converted here; four pieces of eight values per thread on the way
    const int chunks = kc * 16, total = m * chunks;         // of a row, of all
    constexpr int kAhead = 4;
    for (int base = 0; base < total; base += kAhead * kCThreads) {
      const int i0 = base + tid;
      float v[kAhead][8];
      int col[kAhead], n[kAhead];
#pragma unroll
      for (int q = 0; q < kAhead; ++q) {
        const int i = i0 + q * kCThreads, r = i / chunks;
        col[q] = r;
        n[q] = (i - r * chunks) * 8;
        if (i < total) load_x8(p.x, p.x_dtype, ((size_t)(row0 + r) * p.bpr + k0) * kBlock + n[q], v[q]);
      }
      if (XT == 2 && p.ss && base == 0) {                   // rows in front of their norm, whose scale arrives beside them
        if (warp < m) {
          const float s = row_scale(p, row0 + warp, lane);
          if (lane == 0) s_scale[warp] = s;
        }
        __syncthreads();
      }
#pragma unroll
      for (int q = 0; q < kAhead; ++q) {
        if (i0 + q * kCThreads < total) {
          if (XT == 2 && p.ss) {
            float w[8];
            const float* src = p.w_next + k0 * kBlock + n[q];
            if ((uintptr_t)p.w_next % 16 == 0) {
              load_x8(src, NB_F32, 0, w);
            } else {
#pragma unroll
              for (int e = 0; e < 8; ++e) w[e] = __ldg(src + e);
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) v[q][e] = v[q][e] * s_scale[col[q]] * w[e];
          }
          uint32_t hi[4];
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int e = 0; e < 2; ++e) hi[2 * h + e] = f32x2_to_f16x2_sat(v[q][4 * h + e], v[q][4 * h + e + 2]);     // in the order 0, 2, 1, 3
          const int seg = n[q] >> 5 & 3, at = (n[q] >> 7) * 256 + seg * 64, c = XT * col[q];
          *reinterpret_cast<uint4*>(x_s + (size_t)c * kc_max * 256 + at + (((n[q] >> 3 & 3) ^ seg ^ (c & 1)) << 4)) =
              make_uint4(hi[0], hi[1], hi[2], hi[3]);
          if (XT == 2) {
            uint32_t lo[4];
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&hi[2 * h + e]));
                lo[2 * h + e] = f32x2_to_f16x2_sat(v[q][4 * h + e] - f.x, v[q][4 * h + e + 2] - f.y);
              }
            *reinterpret_cast<uint4*>(x_s + (size_t)(c + 1) * kc_max * 256 + at + (((n[q] >> 3 & 3) ^ seg ^ 1) << 4)) =
                make_uint4(lo[0], lo[1], lo[2], lo[3]);
          }
        }
      }
    }
  } else if (bulk) {
    const uint32_t bytes = (uint32_t)kc * 256u;
    if (warp == 0) {
      if (lane == 0) mbar_arrive_expect_tx(&s_xbar, 2u * m * bytes);
      __syncwarp();
      if (lane < 2 * m) bulk_g2s(x_s + (size_t)lane * kc_max * 256, xt + (size_t)lane * p.bpr * 256, bytes, &s_xbar);
      __syncwarp();
    }
  } else {
    const int chunks = kc * 16;                             // of a column
    for (int col = 0, i = tid; col < 2 * m; ++col) {
      for (; i < chunks; i += kCThreads) cp_async16(x_s + (size_t)col * kc_max * 256 + 16 * i, xt + (size_t)col * p.bpr * 256 + 16 * i);
      i -= chunks;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  if (tid == 0) {                                           // the next launch's weights into L2, behind the copies of this one
    const unsigned from = blockIdx.x * p.ahead_step;
    if (p.ahead && from < p.ahead_bytes)
      asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p.ahead + from), "r"(min(p.ahead_step, p.ahead_bytes - from)) : "memory");
  }
  // requested here, used behind the products: a row's partial sums of squares (one warp per row), residual values
  constexpr int kSq = 6;
  const bool sq_late = !kPlain && p.ss != nullptr, sq_mine = sq_late && warp < m;
  const float* sq = p.ss + (size_t)(row0 + warp) * p.ss_n;
  float sqv[kSq];
#pragma unroll
  for (int i = 0; i < kSq; ++i) sqv[i] = sq_mine && lane + 32 * i < p.ss_n ? __ldcg(sq + lane + 32 * i) : 0.f;
  const int rows_out = p.mode == NB_CHAIN_SWIGLU ? 8 : 16;
  const int items = own * m * rows_out;
  float res = 0.f, wn = 0.f;
  if (p.mode == NB_CHAIN_RESIDUAL && tid < items) {
    const int row = tid & 15, rest = tid >> 4, il = m == 1 ? rest : rest / m, mm = rest - il * m;
    const int n = (p.tile0 + ci + (rank + il * S) * p.clusters) * 16 + row;
    res = __ldcg(p.res + (size_t)(row0 + mm) * p.N + n);
    if (p.yt) wn = __ldg(p.w_next + n);
  }
  if (bulk) {
    chain_wait(&s_xbar, 0, p.status);
  }
  if (kRaw || !bulk) {                                      // (packed rows: one wait for all; an arrival per copying thread on a
    asm volatile("cp.async.wait_group 0;" ::: "memory");    // barrier per tile is a shared-memory atomic each)
    __syncthreads();
  }

  // ---- the products
  // (m_part takes at least one row of the last group of columns; its lanes without a column keep zeros)
  const uint8_t* xc[CG];
#pragma unroll
  for (int j = 0; j < CG; ++j) xc[j] = x_s + (size_t)min(8 * j + g, XT * m - 1) * kc_max * 256 + t * 64;
  const uint32_t act = 8 * (CG - 1) + g < XT * m;
  uint4 x_last[1] = {make_uint4(0u, 0u, 0u, 0u)};
  constexpr int kAcc = CG == 1 ? 2 : CG;
  bool cluster_up = !kCluster;
  const uint8_t *up = smem + (size_t)ua * kUnit, *cp = nullptr;
  int u = ua, i = i_first, kk = kk_first, slot_j = j_first;
#pragma unroll 1
  while (u < ub) {                                          // a tile's part of the run
    float c[kAcc][4];
#pragma unroll
    for (int j = 0; j < kAcc; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) c[j][e] = 0.f;
    const uint8_t* xp[CG];
#pragma unroll
    for (int j = 0; j < CG; ++j) xp[j] = xc[j] + kk * 256;
    const int tile_end = min(ub, u + kc - kk);
    if constexpr (kRaw) {
      const uint8_t* tile = smem + i * 16 * (raw.idx_stride + raw.cb_stride);
      up = tile + g * raw.idx_stride + (4 * kk + t) * (4 * BITS);
      cp = tile + 16 * raw.idx_stride + g * raw.cb_stride + kk * raw.cb_block;
    }
    if (!kRaw) chain_wait(&s_bar[i], 0, p.status);
#pragma unroll (CG == 1 ? 2 : 1)
    for (; u < tile_end; ++u) {
      chain_unit<BITS, CG, kRaw>(raw, up, cp, xp, lane, sm, act, x_last, c);
      up += kRaw ? 16 * BITS : kUnit;
      if constexpr (kRaw) cp += raw.cb_block;
#pragma unroll
      for (int j = 0; j < CG; ++j) xp[j] += 256;
    }
    if (!cluster_up) { cluster_wait(); cluster_up = true; }
    // lane (g, t): rows g and g + 8 of the tile, columns 8j + 2t and 8j + 2t + 1: both terms of activation row 4j + t, or two rows.
    // The warp that ends the tile leaves zeros in the places behind its own
    const uint32_t dst = smem_u32(parts + (size_t)(((i >> lg) * S + rank) * p.J) * slot);
    const int last_j = tile_end == (i + 1) * kc ? p.J - 1 : slot_j;
    if (CG == 1)
#pragma unroll
      for (int e = 0; e < 4; ++e) c[0][e] += c[kAcc - 1][e];
#pragma unroll
    for (int j = 0; j < CG; ++j) {
#pragma unroll
      for (int o = 0; o < (XT == 2 ? 1 : 2); ++o) {
        const int mm = XT == 2 ? 4 * j + t : 8 * j + 2 * t + o;
        if (mm < m) {
          float va = XT == 2 ? c[j][0] + c[j][1] : c[j][o];
          float vb = XT == 2 ? c[j][2] + c[j][3] : c[j][2 + o];
#pragma unroll 1
          for (int q = slot_j; q <= last_j; ++q) {
            const uint32_t at = dst + (uint32_t)(q * slot + mm * 16 + g) * 4u;
            if (kCluster) {
              st_cluster_f32(at, (uint32_t)(i & (S - 1)), va);
              st_cluster_f32(at + 32u, (uint32_t)(i & (S - 1)), vb);
            } else {
              asm volatile("st.shared.f32 [%0], %1;" ::"r"(at), "f"(va) : "memory");
              asm volatile("st.shared.f32 [%0], %1;" ::"r"(at + 32u), "f"(vb) : "memory");
            }
            va = vb = 0.f;
          }
        }
      }
    }
    kk = 0;
    ++i;
    slot_j = 0;
  }
  if (sq_mine) {                                            // in a fixed order: the same bits in every CTA
    float s = 0.f;
#pragma unroll
    for (int q = 0; q < kSq; ++q) s += sqv[q];
    for (int q = lane + 32 * kSq; q < p.ss_n; q += 32) s += __ldcg(sq + q);
    s = warp_sum(s);
    if (lane == 0) s_scale[warp] = 1.0f / sqrtf(s / (float)(p.bpr * kBlock) + p.eps);
  }
  if (kCluster) {
    if (!cluster_up) cluster_wait();
    cluster_arrive();
    cluster_wait();
  } else {
    __syncthreads();
  }

  // ---- the tiles this CTA finishes
  for (int e = tid; e < items; e += kCThreads) {
    const int row = p.mode == NB_CHAIN_SWIGLU ? e & 7 : e & 15, rest = p.mode == NB_CHAIN_SWIGLU ? e >> 3 : e >> 4;
    const int il = m == 1 ? rest : rest / m, mm = rest - il * m, tile = p.tile0 + ci + (rank + il * S) * p.clusters, b = row0 + mm;
    const float* src = parts + (size_t)il * S * p.J * slot + mm * 16 + row;
    float v = 0.f, v2 = 0.f;
#pragma unroll 4
    for (int q = 0; q < S * p.J; ++q) {
      v += src[(size_t)q * slot];
      if (p.mode == NB_CHAIN_SWIGLU) v2 += src[(size_t)q * slot + 8];
    }
    const float scale = sq_late ? s_scale[mm] : 1.f;
    if (p.mode == NB_CHAIN_STORE) {
      const int n = tile * 16 + row;
      if (n < p.N) store_y(p.y, p.y_dtype, (size_t)b * p.N + n, v * scale);
    } else if (p.mode == NB_CHAIN_SWIGLU) {                 // rows 0 .. 7 of a tile are gate channels, 8 .. 15 the matching up channels
      v *= scale;
      v2 *= scale;
      store_chain_terms(p.yt, p.N >> 8, b, tile * 8 + row, v / (1.f + __expf(-v)) * v2);
    } else {
      const int n = tile * 16 + row;
      if (e >= kCThreads) {
        res = __ldcg(p.res + (size_t)b * p.N + n);
        if (p.yt) wn = __ldg(p.w_next + n);
      }
      v = v * scale + res;
      p.res[(size_t)b * p.N + n] = v;
      if (p.yt) store_chain_terms(p.yt, p.N >> 7, b, n, v * wn);
      if (p.ss_out) {
        float s = v * v;                                    // the tile's 16 rows are 16 neighbouring lanes
        const uint32_t half = 0xffffu << (lane & 16);
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(half, s, o);
        if (row == 0) p.ss_out[(size_t)b * (p.N >> 4) + tile] = s;
      }
    }
  }
}

// x (B, C) = the tokens' rows of a bf16 table, their terms times the norm weight `w` (null: no terms), and the sums of squares per 16 columns.
__global__ void __launch_bounds__(256) chain_embed_kernel(const __nv_bfloat16* __restrict__ table, const long long* __restrict__ token,
                                                          const float* __restrict__ w, float* __restrict__ x, uint8_t* __restrict__ terms,
                                                          float* __restrict__ ss, int C, int V) {
  pdl_enter();
  const int b = blockIdx.y, n = blockIdx.x * 256 + threadIdx.x;
  if (n >= C) return;                                       // C is a multiple of 128: whole warps
  long long tk = token[b];
  tk = tk < 0 ? 0 : (tk >= V ? V - 1 : tk);
  const float v = __bfloat162float(table[(size_t)tk * C + n]);
  x[(size_t)b * C + n] = v;
  if (terms) store_chain_terms(terms, C >> 7, b, n, v * w[n]);
  float s = v * v;
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 15) == 0) ss[(size_t)b * (C >> 4) + (n >> 4)] = s;
}

constexpr size_t kChainSmemMax = 227 * 1024 - 2048;

struct ChainPlan {
  int S, clusters, parts, m_part, launches, per_launch, w_bytes, J, cg, terms;      // per_launch: row tiles
  int idx_stride, cb_stride;
  size_t smem;
  double cost;
};

// Split over clusters of S CTAs; false if even one row tile does not fit.  As many launches as it takes for a CTA's units, its
// share of the activations and the partial results to fit.
// cb_block: bytes of a block's codebook beside packed rows, 0 for the stream layout.
static bool chain_plan(int N, int bpr, int M, int terms, bool plain, int bits, int cb_block, int S, int max_clusters, ChainPlan& pl) {
  if (S > bpr) return false;
  const int n_tiles = (N + 15) / 16, unit = bits == 4 ? StreamUnit<4>::kBytes : StreamUnit<3>::kBytes;
  pl.S = S;
  pl.parts = (M + 15) / 16;
  pl.m_part = (M + pl.parts - 1) / pl.parts;
  pl.terms = terms;
  pl.cg = terms * pl.m_part <= 8 ? 1 : terms * pl.m_part <= 16 ? 2 : 4;
  const int room = std::max(1, max_clusters / pl.parts), kc_max = (bpr + S - 1) / S, kc_min = bpr / S;
  // rows an odd number of 16 (3 bits), 32 (2) or 64 bytes (4) apart, codebooks of 16: the rows that are read together meet different banks
  const int odd = bits == 3 ? 16 : bits == 2 ? 32 : 64;
  pl.idx_stride = ((kc_max * 16 * bits + odd - 1) / odd | 1) * odd;
  pl.cb_stride = ((kc_max * cb_block + 15) / 16 | 1) * 16;
  const int tile_bytes = cb_block ? 16 * (pl.idx_stride + pl.cb_stride) : kc_max * unit;
  for (pl.launches = 1; pl.launches <= n_tiles; ++pl.launches) {
    pl.per_launch = (n_tiles + pl.launches - 1) / pl.launches;
    pl.clusters = std::min(pl.per_launch, room);
    const int T = (pl.per_launch + pl.clusters - 1) / pl.clusters, last = n_tiles - (pl.launches - 1) * pl.per_launch;
    if (last < 1) continue;
    pl.w_bytes = T * tile_bytes;
    // a tile of kc units meets at most kc warps, and two more than it has whole runs
    const int run = std::max(1, std::max(1, last / pl.clusters) * kc_min / kCW);
    pl.J = std::min(kc_max, kc_max / run + 2);
    pl.smem = (size_t)pl.w_bytes + (size_t)terms * pl.m_part * kc_max * 256 + (size_t)((T + S - 1) / S) * S * pl.J * 64 * pl.m_part;
    if (T <= kChainTiles && pl.smem <= kChainSmemMax) {
      // clocks: units at the rate of their lookups and MMAs, staged columns (copied, or converted), launch and drain, a cluster's
      // barriers; within 15 % of the best of the four splits over eight shapes and 1 to 16 rows
      pl.cost = pl.launches * (T * kc_max * ((cb_block ? 80.0 : 60.0) + 9.0 * (pl.cg - 1)) + (double)terms * pl.m_part * kc_max * (plain ? 16.0 : 4.0) + 4000.0 + (S > 1 ? 2500.0 : 0.0));
      return true;
    }
    if (T == 1) return false;
  }
  return false;
}

template <int BITS, int CG, int XT, bool kCluster, bool kRaw, bool kPlain>
static int chain_launch_as(const ChainPlan& pl, const ChainParams& p, const ChainLayout<kRaw>& raw, bool ordered, cudaStream_t st) {
  static bool done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!done[dev & 63]) {
    if (cudaError_t e = cudaFuncSetAttribute(chain_kernel<BITS, CG, XT, kCluster, kRaw, kPlain>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kChainSmemMax))
      return record_cuda_error(e);
    done[dev & 63] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(pl.clusters * pl.parts * pl.S));
  cfg.blockDim = dim3(kCThreads);
  cfg.dynamicSmemBytes = pl.smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  cfg.attrs = attr;
  if (!ordered) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (kCluster) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = pl.S;
    attr[cfg.numAttrs].val.clusterDim.y = 1;
    attr[cfg.numAttrs++].val.clusterDim.z = 1;
  }
  return record_cuda_error(cudaLaunchKernelEx(&cfg, chain_kernel<BITS, CG, XT, kCluster, kRaw, kPlain>, p, raw));
}
template <int BITS, bool kRaw>
static int chain_launch(const ChainPlan& pl, const ChainParams& p, const ChainLayout<kRaw>& raw, bool ordered, cudaStream_t st) {
  const auto run = [&](auto cg, auto xt, auto plain) {
    constexpr int CG = decltype(cg)::value, XT = decltype(xt)::value;
    constexpr bool kPlain = decltype(plain)::value;
    return pl.S > 1 ? chain_launch_as<BITS, CG, XT, true, kRaw, kPlain>(pl, p, raw, ordered, st)
                    : chain_launch_as<BITS, CG, XT, false, kRaw, kPlain>(pl, p, raw, ordered, st);
  };
  const std::integral_constant<int, 1> one{};
  const std::integral_constant<int, 2> two{};
  const std::integral_constant<int, 4> four{};
  if (pl.terms == 1) return pl.cg == 1 ? run(one, one, std::true_type{}) : run(two, one, std::true_type{});
  if (p.x) return pl.cg == 1 ? run(one, two, std::true_type{}) : pl.cg == 2 ? run(two, two, std::true_type{}) : run(four, two, std::true_type{});
  if constexpr (!kRaw) {                                    // (terms against packed rows: steps of 9 to 16 sequences)
    if (pl.cg == 1) return run(one, two, std::false_type{});
    if (pl.cg == 2) return run(two, two, std::false_type{});
  }
  return run(four, two, std::false_type{});
}

// Clusters of S CTAs with a whole SM each that the device runs at once.
static int max_clusters(int S) {
  if (S == 1) return sm_count();
  static int found[64][9] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  int& n = found[dev & 63][S];
  if (n == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(S);
    cfg.blockDim = dim3(kCThreads);
    cfg.dynamicSmemBytes = kChainSmemMax;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = S;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int got = 0;
    if (cudaFuncSetAttribute(chain_kernel<3, 1, 2, true, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kChainSmemMax) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&got, chain_kernel<3, 1, 2, true, false, false>, &cfg) != cudaSuccess || got < 1) {
      cudaGetLastError();
      got = 1;
    }
    n = got;
  }
  return n;
}

}  // namespace nb

using namespace nb;

extern "C" size_t nb_chain_terms_bytes(int M, int K) { return M < 1 || K < kBlock || K % kBlock ? 0 : (size_t)M * K * 4; }

// Whether nb_chain_linear is the faster one for more rows than its columns were made for.  Its MMAs and parts grow with the rows, the
// tcgen05 kernel has its start, its k-steps and a sum over k splits whatever the rows are (fused | this, us, 3 bits, fp32 rows:
// 3072 x 1024 40 rows 11.1 | 7.2, 64: 12.0 | 8.6; 2560 x 2560 32: 11.6 | 9.4, 40: 10.8 | 11.2; 6144 x 2048 17: 11.8 | 10.9, 20: 11.8 | 11.5;
// bf16 6144 x 2048 32: 12.1 | 9.5; 7680 x 2560 20: 13.4 | 11.7, 24, which takes two launches: 13.4 | 17.4): up to 510 M products in one
// launch (453 - 503 M: 13824 x 512 32 rows 9.2 | 9.4, 1000 x 4096 56: 12.0 | 10.0, 4096 x 2048 28: 11.1 | 10.9).
extern "C" int nb_chain_takes(int M, int N, int K, int bits, int x_dtype) {
  if (M < 1 || N < 1 || K < kBlock || K % kBlock || (bits != 2 && bits != 3 && bits != 4) || M > 64) return 0;
  const int terms = x_dtype == NB_F32 ? 2 : 1;
  if ((double)M * terms * N * K > 510e6 || check_device() != NB_OK) return 0;
  ChainPlan pl{}, best{};
  best.cost = 1e30;
  for (int S : {1, 2, 4, 8})
    if (chain_plan(N, K / kBlock, M, terms, true, bits, 0, S, max_clusters(S), pl) && pl.cost < best.cost) best = pl;
  return best.cost < 1e30 && best.launches == 1;
}

// Whether plain rows against the packed matrix are for nb_chain_linear rather than nb_gemv.  Where few 16-bit rows meet many short
// rows of weights, every CTA of nb_gemv has whole rows, all CTAs run at once and its unpacking is the cheaper one (us, nb_gemv |
// this, 3 bits, 2 and 4 rows: 5632 x 1024 3.5 | 4.1, 3.9 | 4.2; 6912 x 2560 6.0 | 7.7, 6.9 | 8.0; 9472 x 2560 6.6 | 8.2, 7.3 | 8.4; on the
// other side of the line 4096 x 2560 5.7 | 5.7, 7.0 | 5.9; 6912 x 4096 11.6 | 9.3; 11008 x 2560 14.6 | 8.9; 6912 x 2560 with 5 rows 7.6 | 8.2, with
// 8 9.4 | 8.6; at 2 bits 8192 x 2560 8.3 | 7.4).
extern "C" int nb_chain_takes_packed(int M, int N, int K, int bits, int x_dtype) {
  if (M < 2 || M > 16 || N < 1 || K < kBlock || K % kBlock || (bits != 2 && bits != 3 && bits != 4)) return 0;
  return !(bits == 3 && x_dtype != NB_F32 && M <= 4 && N >= 5120 && K <= 2560 && (long long)N * K <= 25000000);
}

extern "C" int nb_chain_linear(const nb_chain_args* a, void* stream) {
  constexpr long long kMost = 1ll << 26;                    // products of sizes below stay in 32 bits
  if (!a || !a->w || (a->x ? a->sq && (!a->x_weight || a->x_dtype != NB_F32 || a->mode == NB_CHAIN_RESIDUAL) : !a->x_terms) || !a->status || a->M < 1 || a->N < 1) return NB_ERR_ARG;
  if (a->mode < NB_CHAIN_STORE || a->mode > NB_CHAIN_RESIDUAL) return NB_ERR_ARG;
  if (a->mode == NB_CHAIN_STORE ? !a->y : a->mode == NB_CHAIN_SWIGLU ? !a->y_terms : !a->residual) return NB_ERR_ARG;
  if (a->mode == NB_CHAIN_RESIDUAL && a->y_terms && (!a->next_weight || !a->sq_out)) return NB_ERR_ARG;
  if (a->sq && a->sq_n < 1) return NB_ERR_ARG;
  if (a->x && (a->x_dtype < NB_F32 || a->x_dtype > NB_BF16)) return NB_ERR_ARG;
  if (a->y_dtype < NB_F32 || a->y_dtype > NB_BF16) return NB_ERR_ARG;
  if (a->bits != 2 && a->bits != 3 && a->bits != 4) return NB_ERR_SHAPE;
  if (a->K < kBlock || a->K % kBlock) return NB_ERR_SHAPE;
  if (a->mode == NB_CHAIN_SWIGLU && a->N % (2 * kBlock)) return NB_ERR_SHAPE;
  if (a->mode == NB_CHAIN_RESIDUAL && a->N % kBlock) return NB_ERR_SHAPE;
  if (a->split < 0 || a->split > 8 || (a->split & (a->split - 1))) return NB_ERR_ARG;
  if ((long long)(a->N + 15) / 16 * (a->K / kBlock) > kMost || a->N > (1 << 24)) return NB_ERR_SHAPE;
  if (a->codebook && a->codebook_dtype != NB_F16 && a->codebook_dtype != NB_F32) return NB_ERR_ARG;
  if ((uintptr_t)a->w % 16 || (uintptr_t)a->codebook % 16 || (uintptr_t)a->x_terms % 16 || (uintptr_t)a->y_terms % 16 || (uintptr_t)a->ahead % 16 || a->ahead_bytes % 16 || (uintptr_t)a->x % 16)
    return NB_ERR_ALIGN;
  if (int rc = check_device()) return rc;
  const int bpr = a->K / kBlock, cb_block = a->codebook ? (a->codebook_dtype == NB_F16 ? 2 : 4) << a->bits : 0;
  ChainPlan pl{}, best{};
  best.cost = 1e30;
  for (int S : {1, 2, 4, 8}) {
    if (a->split && S != a->split) continue;
    if (chain_plan(a->N, bpr, a->M, a->x && a->x_dtype != NB_F32 ? 1 : 2, a->x != nullptr, a->bits, cb_block, S, max_clusters(S), pl) && pl.cost < best.cost) best = pl;
  }
  if (best.cost == 1e30) return NB_ERR_SHAPE;
  ChainParams p{};
  const ChainRaw raw{reinterpret_cast<const uint8_t*>(a->codebook), a->codebook_dtype, cb_block, best.idx_stride, best.cb_stride};
  p.w = a->w; p.xt = reinterpret_cast<const uint8_t*>(a->x_terms); p.ss = a->sq; p.y = a->y; p.yt = reinterpret_cast<uint8_t*>(a->y_terms);
  p.res = a->residual; p.w_next = a->x && a->sq ? a->x_weight : a->next_weight; p.ss_out = a->sq_out; p.status = a->status;
  p.x = a->x; p.x_dtype = a->x_dtype; p.y_dtype = a->y_dtype;
  p.N = a->N; p.bpr = bpr; p.M = a->M; p.mode = a->mode; p.ss_n = a->sq_n; p.eps = a->eps;
  p.m_part = best.m_part; p.parts = best.parts; p.lg_split = best.S == 8 ? 3 : best.S >> 1; p.w_bytes = best.w_bytes; p.J = best.J;
  auto rcp = [](int v) { return (unsigned)((0x100000000ull + v - 1) / v); };
  p.rcp_kc = rcp(std::max(1, bpr / best.S)); p.rcp_kc1 = rcp((bpr + best.S - 1) / best.S);
  const int n_tiles = (a->N + 15) / 16, most = best.clusters;
  for (int l = 0; l < best.launches; ++l) {
    p.tile0 = l * best.per_launch;
    p.n_tiles = std::min(best.per_launch, n_tiles - p.tile0);
    p.clusters = best.clusters = std::min(most, p.n_tiles);
    p.rcp_clusters = rcp(p.clusters);
    if (l == best.launches - 1 && a->ahead && a->ahead_bytes > 0) {
      const long long ctas = (long long)p.clusters * p.parts * best.S;
      p.ahead = a->ahead; p.ahead_bytes = (unsigned)std::min<long long>(a->ahead_bytes, 1ll << 30);
      p.ahead_step = (unsigned)((p.ahead_bytes + ctas * 1024 - 1) / (ctas * 1024) * 1024);
    }
    int rc = NB_OK;
    cudaStream_t st = (cudaStream_t)stream;
    const auto run = [&](auto packed, const auto& layout) {
      constexpr bool kRaw = decltype(packed)::value;
      return a->bits == 2 ? chain_launch<2, kRaw>(best, p, layout, a->ordered, st) : a->bits == 3 ? chain_launch<3, kRaw>(best, p, layout, a->ordered, st)
                                                                                                 : chain_launch<4, kRaw>(best, p, layout, a->ordered, st);
    };
    rc = a->codebook ? run(std::true_type{}, raw) : run(std::false_type{}, ChainCopy{});
    if (rc) return rc;
  }
  return NB_OK;
}

extern "C" int nb_chain_embed(const void* table_bf16, const int64_t* token, int B, int V, int C, const float* weight, float* x, void* terms,
                              float* sq, void* stream) {
  if (!table_bf16 || !token || (terms && !weight) || !x || !sq || B < 1 || V < 1 || C < 1) return NB_ERR_ARG;
  if (C % kBlock || B > 65535) return NB_ERR_SHAPE;
  if ((uintptr_t)terms % 16) return NB_ERR_ALIGN;
  if (int rc = check_device()) return rc;
  return launch_pdl(chain_embed_kernel, dim3((C + 255) / 256, B), dim3(256), 0, (cudaStream_t)stream,
                    reinterpret_cast<const __nv_bfloat16*>(table_bf16), reinterpret_cast<const long long*>(token), weight, x,
                    reinterpret_cast<uint8_t*>(terms), sq, C, V);
}
