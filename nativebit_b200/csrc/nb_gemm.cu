// Prefill GEMM for NativeBit packed linears on sm_100a: Y (M, N) = X (M, K) . W (N, K)^T for many
// activation rows, on the 5th-generation tensor cores (tcgen05.mma, accumulator in tensor memory).
//
// nb_gemm_prefill dequantises the packed weight once into an fp16 (N, K) scratch matrix (35 MB for
// 6912 x 2560: it stays in the 126 MB L2) with the gather kernel of nb_unpack.cu, then runs the
// kernel below on X and that matrix.  W enters as fp16 (the codebook entries themselves, so the
// weights are exact; the reference's any-M kernel rounds them to bf16,
// nativebit_jax/packed_kernel.py:151-159).  The tensor-core instruction wants both operands in one
// 16-bit format (a bf16 A with an fp16 B is an illegal instruction on sm_100a), so bf16 activations
// are first converted to fp16 (exact for magnitudes 6.1e-5..65504, saturating above, as in the
// GEMV).  Products are accumulated in fp32.
//
// Kernel: persistent, 192 threads per CTA, one CTA per SM; two CTAs of a cluster (CG = 2) share a 256 x BN output tile, or
// each works on a 128 x BN tile of its own (CG = 1: inputs of up to 128 rows, and shapes whose last wave it fills better).
// Two accumulator buffers in tensor memory; BN = a multiple of 32 up to 256:
//   warp 0   one lane issues TMA tile loads (cp.async.bulk.tensor.2d, 128-byte swizzle) of a 128 x 64 slab of X and of this
//            CTA's BN / CG rows of a BN x 64 slab of W per k-step into a ring of shared-memory stages, each completing on the
//            stage's "full" mbarrier (of the pair's first CTA);
//   warp 1   allocates the 512 columns of tensor memory; in the first CTA one lane waits for a full stage and issues four
//            tcgen05.mma (M = 128 * CG, N = BN, K = 16) per stage from shared-memory descriptors, then tcgen05.commit on the
//            stage's "empty" barriers of both CTAs (and on the accumulator barriers at the end);
//   warps 2-5  epilogue: each warp owns one 32-lane quadrant of tensor memory, reads the finished buffer with tcgen05.ld (32
//            columns at a time), turns its 32 x 128-byte piece of Y round in shared memory and stores whole 128-byte lines,
//            then hands the buffer back, while the MMA warp already fills the other one.
// Bound by the tensor cores (and, at long inputs, by the power limit).  The pair halves the W traffic into each SM and the
// MMA issues per FLOP; lines instead of 16-byte pieces of 32 rows let an fp32 epilogue keep up; the order of the tiles keeps
// X and W in L2.  bf16 in and out, before -> now: 8192 x 13824 x 2560 629 -> 371 us (1.56 PFLOP/s), 8192 x 2560 x 6912
// 299 -> 201 us, 2048 x 2560 x 6912 104 -> 64 us, 2048 x 6912 x 2560 55.6 -> 49.4 us.
// fp32 activations: X is (M, 2K) with a row's two fp16 terms side by side; the k-steps run over the second terms first, then
// over the first ones, against the same W: the small sums come first, so nothing of them is lost and the epilogue sees one
// finished sum.
// Every mbarrier wait is bounded: after kSpinLimit probes the waiter raises its CTA's abort flag, writes NB_ERR_TIMEOUT to the
// status word and all roles fall through to the common exit, where tensor memory is freed.
#include <cuda.h>
#include <cuda_runtime.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cfloat>
#include <cstdio>
#include <mutex>

#include "nb_common.cuh"
#include "nb_host.h"
#include "nb_launch.cuh"
#include "nb_umma.cuh"
#include "../../include/nativebit_b200_layered.h"

namespace nb {

struct GemmCfg {
  static constexpr int kMaxStages = 8;
  static constexpr int kMaxBN = 256;
  static constexpr int kABytes = kBM * kBK * 2;          // 16 KB
  static constexpr int kRing = 192 * 1024;               // operand stages
  static constexpr int kEpiRow = 36;                     // words of a staged row: 128 bytes and 16 that turn the banks
  static constexpr int kEpiWords = 32 * kEpiRow;         // per epilogue warp
  static constexpr int kSmem = kRing + 1024 /*alignment slack*/ + 256 /*barriers*/ + 4 * kEpiWords * 4;
  // number of stages that fit the ring: b_rows rows of W per stage
  __host__ __device__ static constexpr int stages(int b_rows) {
    return kRing / (kABytes + b_rows * kBK * 2) < kMaxStages ? kRing / (kABytes + b_rows * kBK * 2) : kMaxStages;
  }
  static constexpr int kTmemCols = 512;                  // two accumulator buffers of up to 256 columns
};

struct GemmArgs {
  void* y;
  const float* bias;
  int* status;
  float alpha, limit;
  int y_dtype, ldy, act, M, N, BN, m_tiles, n_tiles, f16;
  int a_bytes;    // of a stage's rows of X: 128 of them, or all there are, in eights (what lies behind them stays unread in Y)
  int w_steps;    // k-steps over W; the last one's columns past K arrive as zeros
  int k_steps;    // w_steps, or twice that over the two terms of fp32 activations
};

// ---- the instructions that differ between a CTA alone and a pair
template <int CG> struct Tc;
template <> struct Tc<1> {
  static __device__ __forceinline__ void alloc(uint32_t* slot, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s2u(slot)), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  static __device__ __forceinline__ void dealloc(uint32_t base, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(cols) : "memory");
  }
  static __device__ __forceinline__ void load(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y) { tma_load_2d(dst, map, bar, x, y); }
  static __device__ __forceinline__ void mma(uint32_t d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) { umma_f16(d, da, db, idesc, acc); }
  static __device__ __forceinline__ void commit(uint64_t* bar) { umma_commit(bar); }
  static __device__ __forceinline__ void arrive_first(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(s2u(bar)) : "memory");
  }
  static __device__ __forceinline__ uint32_t rank() { return 0; }
  static __device__ __forceinline__ void sync() {}
};
template <> struct Tc<2> {
  static __device__ __forceinline__ void alloc(uint32_t* slot, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s2u(slot)), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  static __device__ __forceinline__ void dealloc(uint32_t base, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(cols) : "memory");
  }
  // into this CTA's shared memory, completing on the barrier at the same place in the pair's first CTA (in shared::cluster
  // addresses bit 24 tells the two CTAs of a pair apart)
  static __device__ __forceinline__ void load(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(s2u(dst)), "l"(map), "r"(s2u(bar) & 0xFEFFFFFFu), "r"(x), "r"(y) : "memory");
  }
  static __device__ __forceinline__ void mma(uint32_t d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d), "l"(da), "l"(db), "r"(idesc), "r"(acc) : "memory");
  }
  static __device__ __forceinline__ void commit(uint64_t* bar) {     // arrives on the barrier of both CTAs
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(s2u(bar)), "h"((uint16_t)3) : "memory");
  }
  static __device__ __forceinline__ void arrive_first(uint64_t* bar) {   // on the barrier of the pair's first CTA
    asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %0, 0;\n\t"
                 "mbarrier.arrive.release.cluster.shared::cluster.b64 _, [a];\n\t}" ::"r"(s2u(bar)) : "memory");
  }
  static __device__ __forceinline__ uint32_t rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
  }
  static __device__ __forceinline__ void sync() {
    asm volatile("barrier.cluster.arrive;\n\tbarrier.cluster.wait;" ::: "memory");
  }
};

// Output tile t: groups of eight row tiles, inside a group all column tiles, row tiles fastest: CTAs that run together work on
// a block of about eight by eight tiles, so that X and W are read from memory about once per group.
constexpr int kGemmGroup = 8;
__device__ __forceinline__ void gemm_tile(const GemmArgs& p, int t, int& mt, int& nt) {
  const int per = kGemmGroup * p.n_tiles, grp = t / per, r = t - grp * per;
  const int rows = min(kGemmGroup, p.m_tiles - grp * kGemmGroup);
  nt = r / rows;
  mt = grp * kGemmGroup + r - nt * rows;
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// a / (1 + e^-x) without the branches of a full-range division, which run the 16 pairs of a chunk one after the other (2 x 10 us
// per 128 x 160 tile, more than the tile's products).  With e = e^-|x| the divisor 1 + e lies in [1, 2], well inside the range
// of __fdividef (2 ulp), for every x: a gate far below zero gives zero, one of -inf NaN, as the plain quotient does.
// One step of iterative refinement (the residual of the quotient over the same divisor, Wilkinson 1963) takes the two ulps
// off; a residual that is zero or no number (infinite quotients) leaves the quotient with its sign.
__device__ __forceinline__ float times_sigmoid(float a, float x) {
  const float e = __expf(-fabsf(x)), d = 1.0f + e, n = x < 0.0f ? a * e : a;
  const float q = __fdividef(n, d), c = __fdividef(fmaf(-d, q, n), d);
  return fabsf(c) > 0.0f ? q + c : q;
}

// silu(gate) * up, or the clamped form (alpha, limit)
__device__ __forceinline__ float glu_pair(int act, float alpha, float limit, float g, float u) {
  const bool clamped = act == NB_ACT_CLAMPED_GLU_PAIRS;
  g = clamped ? fminf(g, limit) : g;
  u = clamped ? fminf(fmaxf(u, -limit), limit) + 1.0f : u;
  return times_sigmoid(g, clamped ? alpha * g : g) * u;
}

template <int CG>
__global__ void __launch_bounds__(192, 1)
gemm_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const GemmArgs p) {
  using Cfg = GemmCfg;
  using T = Tc<CG>;
  const int b_rows = p.BN / CG;                       // rows of W this CTA loads per stage: a multiple of 16
  const int S = Cfg::stages(b_rows);
  const int b_bytes = b_rows * kBK * 2;               // a multiple of 1024
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* sA = smem;
  uint8_t* sB = smem + S * Cfg::kABytes;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + Cfg::kRing);
  uint64_t* empty = full + Cfg::kMaxStages;
  uint64_t* acc_full = empty + Cfg::kMaxStages;       // [2] MMA -> epilogue
  uint64_t* acc_empty = acc_full + 2;                 // [2] epilogue -> MMA
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint32_t* epi = reinterpret_cast<uint32_t*>(smem + Cfg::kRing + 256);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)T::rank();
  const int n_total = p.m_tiles * p.n_tiles;
  const int first = (int)blockIdx.x / CG, step = (int)gridDim.x / CG;
  int* const status = p.status;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) { bar_init(&full[s], 1); bar_init(&empty[s], 1); }
    for (int b = 0; b < 2; ++b) { bar_init(&acc_full[b], 1); bar_init(&acc_empty[b], 4 * CG); }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) T::alloc(tmem_slot, (uint32_t)Cfg::kTmemCols);   // a warp-wide operation
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  T::sync();                                          // the other CTA's barriers are ready
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (elect_one()) {  // ---- TMA producer
      int s = 0;           // ring position and its phase bit, carried across tiles
      uint32_t phase = 0;
      bool ok = true;
      asm volatile("griddepcontrol.wait;" ::: "memory");      // barriers and tensor memory were set up beside the launch before
      for (int t = first; t < n_total && ok; t += step) {
        int mt, nt;
        gemm_tile(p, t, mt, nt);
        const int m0 = mt * (kBM * CG) + rank * kBM, n0 = nt * p.BN + rank * b_rows;
        for (int kt = 0; kt < p.k_steps; ++kt) {
          ok = bar_wait(&empty[s], phase ^ 1, abort_flag, status);
          if (!ok) break;
          if (rank == 0) bar_expect_tx(&full[s], (uint32_t)(CG * (p.a_bytes + b_bytes)));
          // two terms: the second half of X's columns first, W from its first column again for the other half
          const int kx = p.k_steps == p.w_steps ? kt : kt < p.w_steps ? kt + p.w_steps : kt - p.w_steps;
          T::load(sA + s * Cfg::kABytes, &map_x, &full[s], kx * kBK, m0);
          T::load(sB + s * b_bytes, &map_w, &full[s], (kt < p.w_steps ? kt : kt - p.w_steps) * kBK, n0);
          if (++s == S) { s = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    if (rank == 0 && elect_one()) {  // ---- MMA issuer
      // instruction descriptor: fp32 accumulate (bit 4), A = X and B = W both bf16 (format 1) or both
      // fp16 (format 0) at bits 7 and 10, both K-major, N = BN, M = 128 * CG
      const uint32_t fmt = p.f16 ? 0u : 1u;
      const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(p.BN >> 3) << 17) | ((uint32_t)((kBM * CG) >> 4) << 24);
      const uint64_t desc_a0 = smem_desc_sw128(sA), desc_b0 = smem_desc_sw128(sB);
      int s = 0, local = 0;
      uint32_t phase = 0;
      for (int t = first; t < n_total; t += step, ++local) {
        const int buf = local & 1;
        // wait until the epilogues have drained this accumulator buffer (first use passes at once)
        bool ok = bar_wait(&acc_empty[buf], ((local >> 1) & 1) ^ 1, abort_flag, status);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t tmem_d = tmem_base + (uint32_t)(buf * Cfg::kMaxBN);
        for (int kt = 0; kt < p.k_steps && ok; ++kt) {
          ok = bar_wait(&full[s], phase, abort_flag, status);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          // the stage's descriptors: the start-address field counts 16-byte units, so a stage further on is an add
          const uint64_t da = desc_a0 + (uint64_t)(s * (Cfg::kABytes >> 4)), db = desc_b0 + (uint64_t)(s * (b_bytes >> 4));
          T::mma(tmem_d, da, db, idesc, kt > 0 ? 1u : 0u);
#pragma unroll
          for (int k4 = 1; k4 < kBK / 16; ++k4)  // 16 bf16 = 32 bytes = 2 descriptor address units per step
            T::mma(tmem_d, da + 2 * k4, db + 2 * k4, idesc, 1u);
          T::commit(&empty[s]);  // frees the stage once these MMAs have read it
          if (++s == S) { s = 0; phase ^= 1; }
        }
        T::commit(&acc_full[buf]);  // accumulator complete (or aborted: the epilogue checks the flag)
        if (!ok) break;
      }
    }
  } else {
    // ---- epilogue: warp w reads tensor-memory lanes 32*(w%4) .. +31 = rows m0 + 32*(w%4) + lane
    const int q = warp & 3;
    uint32_t* st = epi + (warp - 2) * Cfg::kEpiWords;
    const bool bf = p.y_dtype == NB_BF16, glu = p.act != NB_ACT_NONE;
    const int esize = bf ? 2 : 4, per_word = bf ? 2 : 1;
    const int n_out = glu ? p.N >> 1 : p.N;
    const bool vec = (reinterpret_cast<uintptr_t>(p.y) & 15) == 0 && ((size_t)p.ldy * esize) % 16 == 0;
    int local = 0;
    for (int t = first; t < n_total; t += step, ++local) {
      const int buf = local & 1;
      int mt, nt;
      gemm_tile(p, t, mt, nt);
      const int m0 = mt * (kBM * CG) + rank * kBM + q * 32, n0 = nt * p.BN;
      const bool ok = bar_wait<200>(&acc_full[buf], (local >> 1) & 1, abort_flag, status) && !*abort_flag;
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int chunks = (min(p.BN, p.N - n0) + 31) >> 5, rows = min(32, p.M - m0);
      int fill = 0;                                   // words of a row staged so far
      int col = glu ? n0 >> 1 : n0;                   // output column of the staged rows' first word
#pragma unroll 1
      for (int c = 0; c < chunks; ++c) {
        uint32_t r[32];
        const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * Cfg::kMaxBN + c * 32);
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
            "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
            "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
              "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
              "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
              "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
            : "r"(taddr));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (c + 1 == chunks) {                        // the buffer is read: one arrival per warp hands it back to the MMA warp
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) T::arrive_first(&acc_empty[buf]);
        }
        if (rows <= 0) continue;                      // only the rows past the input's last
        if (p.bias) {
          const int n = n0 + c * 32;
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (n + j < p.N) r[j] = __float_as_uint(__uint_as_float(r[j]) + __ldg(p.bias + n + j));
        }
        uint4* row = reinterpret_cast<uint4*>(st + lane * Cfg::kEpiRow + fill);
        if (glu) {                                    // columns 2i (gate) and 2i + 1 (up) -> output column i
          float o[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) o[j] = glu_pair(p.act, p.alpha, p.limit, __uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]));
          if (bf) {
#pragma unroll
            for (int j = 0; j < 2; ++j)
              row[j] = make_uint4(pack_bf16(o[8 * j], o[8 * j + 1]), pack_bf16(o[8 * j + 2], o[8 * j + 3]), pack_bf16(o[8 * j + 4], o[8 * j + 5]),
                                  pack_bf16(o[8 * j + 6], o[8 * j + 7]));
            fill += 8;
          } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
              row[j] = make_uint4(__float_as_uint(o[4 * j]), __float_as_uint(o[4 * j + 1]), __float_as_uint(o[4 * j + 2]), __float_as_uint(o[4 * j + 3]));
            fill += 16;
          }
        } else if (bf) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            auto two = [&](int i) { return pack_bf16(__uint_as_float(r[8 * j + i]), __uint_as_float(r[8 * j + i + 1])); };
            row[j] = make_uint4(two(0), two(2), two(4), two(6));
          }
          fill += 16;
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) row[j] = make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
          fill += 32;
        }
        if (fill < 32 && c + 1 < chunks) continue;
        // store the rows, `fill` words each: eight lanes per 128-byte line, all eight stores of a lane independent of each other (one
        // after the other behind their reads: 8192 rows x 200 columns x 520 deep 9.7 us, now 8.7; 16384 x 2560 x 64 57.9, now 38.7)
        __syncwarp();
        if (vec && fill == 32 && rows == 32 && col + 32 * per_word <= n_out) {
          const size_t hop = (size_t)4 * p.ldy * esize;
          const uint32_t* src = st + (lane >> 3) * Cfg::kEpiRow + 4 * (lane & 7);
          uint8_t* dst = reinterpret_cast<uint8_t*>(p.y) + ((size_t)(m0 + (lane >> 3)) * p.ldy + col + (lane & 7) * 4 * per_word) * esize;
#pragma unroll
          for (int j = 0; j < 8; ++j) *reinterpret_cast<uint4*>(dst + j * hop) = *reinterpret_cast<const uint4*>(src + j * 4 * Cfg::kEpiRow);
          __syncwarp();
          col += fill * per_word;
          fill = 0;
          continue;
        }
        const int per_row = fill >> 2;                // the edges: any number of rows, columns and words per row
        for (int i = lane; i < rows * per_row; i += 32) {
          const int rr = per_row == 8 ? i >> 3 : i / per_row, v = i - rr * per_row;
          const int m = m0 + rr, o = col + v * 4 * per_word;
          if (o >= n_out) continue;
          const uint4 d = *reinterpret_cast<const uint4*>(st + rr * Cfg::kEpiRow + 4 * v);
          uint8_t* dst = reinterpret_cast<uint8_t*>(p.y) + ((size_t)m * p.ldy + o) * esize;
          if (vec && o + 4 * per_word <= n_out) {
            *reinterpret_cast<uint4*>(dst) = d;
          } else {
            const uint32_t w[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              if (!bf) {
                if (o + j < n_out) reinterpret_cast<uint32_t*>(dst)[j] = w[j];
              } else {
                if (o + 2 * j < n_out) reinterpret_cast<uint16_t*>(dst)[2 * j] = (uint16_t)w[j];
                if (o + 2 * j + 1 < n_out) reinterpret_cast<uint16_t*>(dst)[2 * j + 1] = (uint16_t)(w[j] >> 16);
              }
            }
          }
        }
        __syncwarp();
        col += fill * per_word;
        fill = 0;
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  T::sync();                                          // neither CTA leaves while the other may still signal it
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    T::dealloc(tmem_base, (uint32_t)Cfg::kTmemCols);
  }
}

// CTAs per tile and tile width: the plan with the fewest estimated clocks.  A k-step takes the tensor cores' 2 * BN clocks, a
// quarter more in practice, and a part that does not depend on BN, and at least what its loads and issue take; a tile's
// epilogue 1200 and 12 per column, of which only what outlasts the next tile's k-steps and the last tile's show; a pair 2500
// more than a lone CTA for setting up and meeting.  Ties go to the pair and to the wider tile, which reads X fewer times.  The
// figures are fitted to all plans of 324 shapes (1 ... 16384 rows, 20 ... 13824 columns, 16 ... 6912 deep): 1 % above the best
// plan's time in the mean.  (1500 x 2560 x 960: a lone 224 12.5 us, a pair of 224 14.1; 1 x 6912 x 2560: 64 columns 12.3, 256
// 17.2; 8192 x 2560 x 2560: 160 columns in 7 waves 77, 256 in 5 waves 95; 128 x 2560 x 2560: 32 columns on 80 SMs 11.3, 128 on
// 20 SMs 12.9.)
struct GemmPlan { int cg, bn; };
static int step_clocks(int cg, int bn) { return cg == 2 ? std::max(bn * 5 / 2 + 100, 470) : std::max(bn * 5 / 2 + 150, 480); }
static GemmPlan plan_gemm(int M, int N, int k_steps, int sms) {
  GemmPlan best{1, 32};
  double best_cost = 1e30;
  for (int cg = M > kBM && sms > 1 ? 2 : 1; cg >= 1; --cg) {
    const long m_tiles = (M + kBM * cg - 1) / (kBM * cg);
    for (int bn = N >= 256 ? 256 : (N + 31) / 32 * 32; bn >= 32; bn -= 32) {
      const long tiles = m_tiles * ((N + bn - 1) / bn), slots = sms / cg, waves = (tiles + slots - 1) / slots;
      const double steps = (double)k_steps * step_clocks(cg, bn), epilogue = 1200.0 + 12.0 * bn;
      const double cost = waves * steps + epilogue + (waves - 1) * std::max(0.0, epilogue - steps) + (cg == 2 ? 2500 : 0);
      if (cost < best_cost * 0.999) { best_cost = cost; best = GemmPlan{cg, bn}; }
    }
  }
  return best;
}

// X (M rows, `ldx` apart; two: a row's two fp16 terms side by side) times W (N, K).
static int launch_gemm(const void* x, int ldx, const void* w, int ldw, int K, bool two, GemmArgs p, cudaStream_t st) {
  p.w_steps = (K + kBK - 1) / kBK;
  p.k_steps = two ? 2 * p.w_steps : p.w_steps;
  const GemmPlan plan = plan_gemm(p.M, p.N, p.k_steps, sm_count());
  p.BN = plan.bn;
  p.m_tiles = (p.M + kBM * plan.cg - 1) / (kBM * plan.cg);
  p.n_tiles = (p.N + p.BN - 1) / p.BN;
  // rows past X's last are not copied as zeros, which takes longer than copying them: one row x 6912 x 2560, 64 columns per CTA,
  // 20.0 us with a box of 128 rows, 12.3 with one of 8
  const int x_rows = std::min(kBM, (p.M + 7) / 8 * 8);
  p.a_bytes = x_rows * kBK * 2;
  CUtensorMap mx, mw;
  if (int rc = make_map(&mx, x, p.M, two ? 2 * K : K, x_rows, ldx)) return rc;
  if (int rc = make_map(&mw, w, p.N, K, p.BN / plan.cg, ldw)) return rc;
  static bool attr_done[64][3] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  const void* fn = plan.cg == 2 ? (const void*)gemm_kernel<2> : (const void*)gemm_kernel<1>;
  if (!attr_done[dev & 63][plan.cg]) {
    if (cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, GemmCfg::kSmem)) return record_cuda_error(e);
    attr_done[dev & 63][plan.cg] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(plan.cg * std::min(sm_count() / plan.cg, p.m_tiles * p.n_tiles));
  cfg.blockDim = dim3(192);
  cfg.dynamicSmemBytes = GemmCfg::kSmem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = plan.cg;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = plan.cg;                              // a CTA alone needs no cluster
  void* args[] = {&mx, &mw, &p};
  return record_cuda_error(cudaLaunchKernelExC(&cfg, fn, args));
}

}  // namespace nb

using namespace nb;

extern "C" size_t nb_prefill_workspace_bytes(int M, int N, int K) {
  if (M < 1 || N < 1 || K < 1) return 0;
  // status word (first 256 bytes) + fp16 weight + fp16 copy of the activations (two terms per element for fp32)
  return 256 + (((size_t)N * K * 2 + 255) & ~(size_t)255) + (size_t)2 * M * K * 2;
}

// x (M, K) times w (N, K), both bf16 or both fp16 (f16).  The tensor maps copy 2-byte elements either way.  two: x is (M, 2K),
// a row's two fp16 terms side by side.
static int gemm_16bit(const void* x, const void* w, int f16, int M, int N, int K, void* y, int y_dtype, int* status, void* stream,
                      bool two = false) {
  if (!x || !w || !y || M < 1 || N < 1 || K < 1) return NB_ERR_ARG;
  if (y_dtype != NB_BF16 && y_dtype != NB_F32) return NB_ERR_ARG;
  if (K % kBK != 0) return NB_ERR_SHAPE;
  if ((uintptr_t)x % 16 || (uintptr_t)w % 16 || (uintptr_t)y % 4) return NB_ERR_ALIGN;
  if (int rc = check_device()) return rc;
  GemmArgs p{};
  p.y = y; p.y_dtype = y_dtype; p.ldy = N; p.act = NB_ACT_NONE; p.M = M; p.N = N; p.f16 = f16; p.status = status;
  return launch_gemm(x, 0, w, 0, K, two, p, (cudaStream_t)stream);
}

extern "C" int nb_gemm_bf16(const void* x, const void* w, int M, int N, int K, void* y, int y_dtype, int* status, void* stream) {
  return gemm_16bit(x, w, 0, M, N, K, y, y_dtype, status, stream);
}

extern "C" int nb_linear_bf16(const void* x, int ldx, const void* w, int ldw, const float* bias, int act, float alpha, float limit, int M,
                              int N, int K, void* y, int y_dtype, int ldy, int* status, void* stream) {
  if (!x || !w || !y || M < 1 || N < 1 || K < 1 || ldx < K || ldw < K) return NB_ERR_ARG;
  if ((y_dtype != NB_BF16 && y_dtype != NB_F32) || act < NB_ACT_NONE || act > NB_ACT_CLAMPED_GLU_PAIRS) return NB_ERR_ARG;
  if (act != NB_ACT_NONE && N % 2) return NB_ERR_SHAPE;
  if (ldy < (act != NB_ACT_NONE ? N / 2 : N)) return NB_ERR_ARG;
  if ((uintptr_t)x % 16 || (uintptr_t)w % 16 || ldx % 8 || ldw % 8 || (uintptr_t)y % 4) return NB_ERR_ALIGN;
  if (int rc = check_device()) return rc;
  GemmArgs p{};
  p.y = y; p.y_dtype = y_dtype; p.ldy = ldy; p.bias = bias; p.act = act; p.alpha = alpha; p.limit = limit; p.M = M; p.N = N; p.status = status;
  return launch_gemm(x, ldx, w, ldw, K, false, p, (cudaStream_t)stream);
}

extern "C" int nb_gemm_prefill(const void* x, int x_dtype, int M, const uint8_t* packed, const void* codebook, int cb_dtype, int bits,
                               int block_size, int N, int K, void* y, int y_dtype, void* workspace, size_t workspace_bytes,
                               void* stream) {
  if (!x || !packed || !codebook || !y) return NB_ERR_ARG;
  if (x_dtype != NB_BF16 && x_dtype != NB_F16 && x_dtype != NB_F32 && x_dtype != NB_F16_TERMS) return NB_ERR_ARG;
  if (!workspace || workspace_bytes < nb_prefill_workspace_bytes(M, N, K)) return NB_ERR_WORKSPACE;
  if ((uintptr_t)workspace % 256) return NB_ERR_ALIGN;
  if (K % kBK != 0 || K % block_size != 0) return NB_ERR_SHAPE;
  if ((uintptr_t)x % 16) return NB_ERR_ALIGN;
  uint8_t* w = reinterpret_cast<uint8_t*>(workspace) + 256;
  uint8_t* xh = w + (((size_t)N * K * 2 + 255) & ~(size_t)255);
  if (x_dtype == NB_F16 || x_dtype == NB_F16_TERMS) {
    if (int rc = nb_dequant(packed, codebook, cb_dtype, bits, block_size, N, K, w, NB_F16, stream)) return rc;
    return gemm_16bit(x, w, 1, M, N, K, y, y_dtype, reinterpret_cast<int*>(workspace), stream, x_dtype == NB_F16_TERMS);
  }
  // the conversion runs beside the dequantisation: it reads and writes nothing of its (a call with 2048 rows
  // x 6912 x 2560 78.2 -> 75.2 us, together with the wider stores of nb_dequant)
  if (int rc = dequant_beside(packed, codebook, cb_dtype, bits, block_size, N, K, w, NB_F16, stream)) return rc;
  const size_t n8 = (size_t)M * K / 8;  // K % 64 == 0
  const dim3 grid((unsigned)((n8 + 255) / 256)), block(256);
  if (x_dtype == NB_F32) {  // two fp16 terms per element; rows 2i and 2i + 1 of the kernel's result are one row of 2K here
    if (int rc = launch_pdl(f32_to_f16_pair_kernel, grid, block, 0, (cudaStream_t)stream, reinterpret_cast<const float4*>(x),
                            reinterpret_cast<uint4*>(xh), M, K))
      return rc;
    return gemm_16bit(xh, w, 1, M, N, K, y, y_dtype, reinterpret_cast<int*>(workspace), stream, true);
  }
  if (int rc = launch_pdl(bf16_to_f16_kernel, grid, block, 0, (cudaStream_t)stream, reinterpret_cast<const uint4*>(x), reinterpret_cast<uint4*>(xh), n8))
    return rc;
  return gemm_16bit(xh, w, 1, M, N, K, y, y_dtype, reinterpret_cast<int*>(workspace), stream);
}
