// Fused prefill GEMM for NativeBit packed linears on sm_100a: Y (M, N) = X (M, K) . W (N, K)^T for many
// activation rows, with the dequantisation INSIDE the tensor-core kernel: producer warps turn packed
// indices + codebooks into fp16 tiles in shared memory and tcgen05.mma consumes them, so the weight never
// exists in global memory as a dense matrix.  The reference materialises the whole weight on every
// forward (unpack + gather + matmul, inference/triton_kernel.py:258-275); its tiled TPU kernel
// dequantises a tile and contracts it (nativebit_jax/packed_kernel.py:135-178), which is the semantics
// kept here with one difference: the weights enter as the fp16 codebook entries themselves (exact).
//
// Operands.  The WEIGHT tile is the M = 128 operand of the MMA (128 output features x 64 k), the
// ACTIVATION tile the N operand (BN = 16..256 tokens x 64 k), the accumulator D[feature][token] lives in
// tensor memory.  A weight tile is therefore dequantised once per BN tokens; at BN = 256 that is 8192
// lookups per 512 tensor-core clocks, a quarter of the SM's byte-permute throughput.
//
// Weights are read in the stream layout (nb_stream_pack: per 16 rows x 128 weights, every lane-group's
// indices as nibbles in position order + the rows' byte-plane lookup tables).  Persistent kernel, one CTA per SM, 736 threads:
//   warp 0       one lane issues the TMA loads (cp.async.bulk.tensor.2d, 128-byte swizzle, no multicast)
//                of the BN x 64 activation slab of every k-step into a ring of stages;
//   warp 1       allocates tensor memory; one lane waits on the stage's "full" barrier (four producer warps'
//                arrivals + the TMA bytes) and issues four tcgen05.mma (128 x BN x 16, fp16 x fp16 -> fp32)
//                per stage, then tcgen05.commit on the stage's "empty" barrier;
//   warps 2-5    epilogue: each warp owns one 32-lane quadrant of tensor memory (32 output features),
//                reads a finished accumulator with tcgen05.ld and stores Y (transposed: lanes run along
//                N, so a warp's store of one token covers 32 consecutive outputs);
//   warps 6-21   dequant producers, four groups of 4 warps that take turns at the k-steps (filling a stage is a chain of about
//                1200 clocks, most of it waits and barriers, so four are filled at a time): a warp owns two of the eight row
//                tiles of the 128 x 64 weight tile, a thread (row, half) of both reads four selector words and the row's
//                table from a raw stage, looks 32 weights up with byte permutes and, once the stage is free, writes them as
//                four 16-byte chunks into its 128-byte swizzle;
//   warp 22      one lane issues the TMA loads of the raw weights, the eight row tiles of a k-block (two k-steps) at once,
//                into a ring of its own.  (Producers that load through registers wait at every proxy fence until their
//                own prefetches have landed: a k-step then took half a memory latency, 0.40 - 0.45 us, whatever BN was and
//                however far ahead they loaded.)
// The kernel starts while the launch that converts the activations still runs (programmatic dependent launch): only warp 0
// waits for it, the producers fill the first stages meanwhile.
// From a graph over cold weights, before -> now (us): 17 fp32 rows x 7680 x 2560 16.9 -> 13.2, 129 rows 25.2 -> 20.7, 400 rows
// 45.1 -> 34.5; 17 rows x 13824 x 2560 22.7 -> 17.3; 400 rows x 2560 x 6912 52.6 -> 39.5.  A decode step of 32 sequences, per layer
// 108 -> 91.
// Two accumulators in tensor memory let the epilogue of one tile overlap the MMAs of the next.  Every
// mbarrier wait is bounded; on a timeout the waiter raises a shared abort flag, writes NB_ERR_TIMEOUT
// to the status word and all roles fall through to the exit, where tensor memory is freed.
#include <cuda.h>
#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cstdio>

#include "nb_common.cuh"
#include "nb_device.cuh"
#include "nb_host.h"
#include "nb_launch.cuh"
#include "nb_umma.cuh"

namespace nb {

constexpr int kFM = 128;                  // output features per tile (the MMA's M)
constexpr int kFK = 64;                   // k per stage
constexpr int kFProducerWarp0 = 6, kFProducerWarps = 4;   // warps per producer group
constexpr int kFGroups = 4;                                // groups take turns at the k-steps
constexpr int kFRawWarp = kFProducerWarp0 + kFGroups * kFProducerWarps;
constexpr int kFThreads = (kFRawWarp + 1) * 32;
constexpr int kFABytes = kFM * kFK * 2;   // 16 KB of weights per stage
constexpr int kFMaxStages = 8;
constexpr int kFRawBytes = 8 * 1536;       // raw weights: eight row tiles of a k-block at 4 bits
constexpr int kFMaxRaw = 4;
constexpr int kFOperands = 176 * 1024 + kFMaxRaw * kFRawBytes;      // operand stages and raw stages
constexpr int kFSmem = kFOperands + 1024 + 512;
static_assert(kFSmem <= 227 * 1024, "shared memory of a CTA");

// Operand stages are at least as many as producer groups at every BN: past 224 columns two raw stages give way to the fourth
// (a step then takes 512 clocks of the tensor cores, time enough for a raw stage to be filled again).  The raw stages are an
// even number, so that a group, which takes every second k-block, meets each of its stages every turn.
__host__ __device__ constexpr int fused_raw_stages(int bn) { return bn > 224 ? 2 : kFMaxRaw; }
__host__ __device__ constexpr int fused_ring(int bn) { return bn > 224 ? 192 * 1024 : 176 * 1024; }
__host__ __device__ constexpr int fused_stages(int bn) {
  return fused_ring(bn) / (kFABytes + bn * kFK * 2) < kFMaxStages ? fused_ring(bn) / (kFABytes + bn * kFK * 2) : kFMaxStages;
}
constexpr bool enough_stages() {
  for (int bn = 16; bn <= 256; bn += 16)
    if (fused_stages(bn) < kFGroups || fused_ring(bn) + fused_raw_stages(bn) * kFRawBytes > kFOperands) return false;
  return true;
}
static_assert(enough_stages(), "stages per producer group");

// k-steps of one of ks splits: whole k-blocks, as the raw weights arrive
__host__ __device__ constexpr int split_steps(int KT, int ks) { return (KT / 2 + ks - 1) / ks * 2; }

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
               ::"r"(s2u(dst)), "l"(map), "r"(s2u(bar)), "r"(x), "r"(y), "r"(z) : "memory");
}

template <int BITS>
__global__ void __launch_bounds__(kFThreads, 1)
gemm_fused_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, void* __restrict__ y, int y_dtype,
                  int M, int N, int K, int BN, int m_tiles, int w_tiles, int pair, int ks, float* __restrict__ partial, int* status) {
  using F = StreamUnit<BITS>;
  constexpr int kT = BITS == 4 ? 8 : 4;
  const int S = fused_stages(BN), R = fused_raw_stages(BN);
  const int b_bytes = BN * kFK * 2;           // multiple of 1024 because BN is a multiple of 16
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* sA = smem;                         // weights
  uint8_t* sB = smem + S * kFABytes;          // activations
  uint8_t* sW = smem + fused_ring(BN);        // raw weights
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kFOperands);   // a stage's weights (4 producer warps) AND activations (TMA bytes)
  uint64_t* empty = full + kFMaxStages;
  uint64_t* acc_full = empty + kFMaxStages;   // [2] MMA -> epilogue
  uint64_t* acc_empty = acc_full + 2;         // [2] epilogue -> MMA
  uint64_t* raw_full = acc_empty + 2;
  uint64_t* raw_empty = raw_full + kFMaxRaw;   // the two producer groups of a k-block have read it
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(raw_empty + kFMaxRaw);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int KT = K / kFK;
  const int KTs = split_steps(KT, ks);          // k-steps per k split (the last split may be shorter, never empty)
  const int n_total = m_tiles * w_tiles * ks;   // work item t: k split t % ks of output tile t / ks

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) { bar_init(&full[s], kFProducerWarps + 1); bar_init(&empty[s], 1); }
    for (int b = 0; b < 2; ++b) { bar_init(&acc_full[b], 1); bar_init(&acc_empty[b], 4); }
    for (int r = 0; r < R; ++r) { bar_init(&raw_full[r], 1); bar_init(&raw_empty[r], 2 * kFProducerWarps); }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {  // tensor-memory allocation is a warp-wide operation
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s2u(tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;

  // output tile o = t / ks: features 128 * (o / m_tiles), tokens BN * (o % m_tiles): CTAs running together share a
  // weight tile; with ks > 1 the k range of an output tile is cut into ks parts whose fp32 results go to
  // `partial` and are added in k order by a second kernel (short inputs would otherwise leave most SMs idle
  // behind a long serial chain of k-steps)
  if (ks > 1) asm volatile("griddepcontrol.launch_dependents;");      // the summing kernel: it waits for this one's end
  if (warp == 0) {
    if (elect_one()) {  // ---- TMA producer of the activation slabs
      asm volatile("griddepcontrol.wait;" ::: "memory");      // the fp16 operand is the launch before's result, the weights are not
      int s = 0;
      uint32_t phase = 0;
      for (int t = blockIdx.x; t < n_total; t += gridDim.x) {
        const int m0 = ((t / ks) % m_tiles) * BN;
        const int k_lo = (t % ks) * KTs, k_hi = min(KT, k_lo + KTs);
        bool ok = true;
        for (int kt = k_lo; kt < k_hi; ++kt) {
          ok = bar_wait(&empty[s], phase ^ 1, abort_flag, status);
          if (!ok) break;
          bar_expect_tx(&full[s], (uint32_t)b_bytes);
          tma_load_2d(sB + s * b_bytes, &map_x, &full[s], kt * kFK, m0);
          if (++s == S) { s = 0; phase ^= 1; }
        }
        if (!ok) break;
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {  // ---- MMA issuer
      // instruction descriptor: fp32 accumulate (bit 4), A and B fp16 (format 0 at bits 7 and 10), both K-major,
      // N = BN (tokens), M = 128 (features)
      const uint32_t idesc = (1u << 4) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(kFM >> 4) << 24);
      const uint64_t desc_a0 = smem_desc_sw128(sA), desc_b0 = smem_desc_sw128(sB);
      int s = 0, local = 0;
      uint32_t phase = 0;
      for (int t = blockIdx.x; t < n_total; t += gridDim.x, ++local) {
        const int buf = local & 1;
        bool ok = bar_wait(&acc_empty[buf], ((local >> 1) & 1) ^ 1, abort_flag, status);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t tmem_d = tmem_base + (uint32_t)(buf * 256);
        const int k_lo = (t % ks) * KTs, k_hi = min(KT, k_lo + KTs);
        for (int kt = k_lo; kt < k_hi && ok; ++kt) {
          ok = bar_wait(&full[s], phase, abort_flag, status);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          // the stage's descriptors: the start-address field counts 16-byte units, so a stage further on is an add
          const uint64_t da = desc_a0 + (uint64_t)(s * (kFABytes >> 4)), db = desc_b0 + (uint64_t)(s * (b_bytes >> 4));
          umma_f16(tmem_d, da, db, idesc, kt > k_lo ? 1u : 0u);
#pragma unroll
          for (int k4 = 1; k4 < kFK / 16; ++k4)  // 16 fp16 = 32 bytes = 2 descriptor address units per step
            umma_f16(tmem_d, da + 2 * k4, db + 2 * k4, idesc, 1u);
          umma_commit(&empty[s]);  // frees the stage once these MMAs have read it
          if (++s == S) { s = 0; phase ^= 1; }
        }
        umma_commit(&acc_full[buf]);
        if (!ok) break;
      }
    }
  } else if (warp < kFProducerWarp0) {
    // ---- epilogue: warp w reads tensor-memory lanes 32*(w%4) .. +31 = features n0 + 32*(w%4) + lane
    const int q = warp & 3;
    int local = 0;
    for (int t = blockIdx.x; t < n_total; t += gridDim.x, ++local) {
      const int buf = local & 1;
      const int o = t / ks;
      const int m0 = (o % m_tiles) * BN, n0 = (o / m_tiles) * kFM;
      // with k splits the tile's fp32 sums go to this split's slab of `partial` ((M >> pair) x N floats each)
      void* const y_t = ks > 1 ? (void*)(partial + (size_t)(t % ks) * (size_t)(M >> pair) * N) : y;
      const int y_dt = ks > 1 ? (int)NB_F32 : y_dtype;
      const bool ok = bar_wait<200>(&acc_full[buf], (local >> 1) & 1, abort_flag, status) && !*abort_flag;
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int n = n0 + q * 32 + lane;
#pragma unroll 1
      for (int c = 0; c < BN / 16; ++c) {
        uint32_t r[16];
        const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * 256 + c * 16);
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
            "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
              "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
            : "r"(taddr));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (n < N && pair) {
          // rows 2i and 2i+1 of the operand are the two fp16 terms of activation row i: their results are added
          const int mb = (m0 + c * 16) >> 1;
          const int m_out = M >> 1;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if (mb + j < m_out) {
              const float v = __uint_as_float(r[2 * j]) + __uint_as_float(r[2 * j + 1]);
              if (y_dt == NB_BF16) reinterpret_cast<__nv_bfloat16*>(y_t)[(size_t)(mb + j) * N + n] = __float2bfloat16_rn(v);
              else reinterpret_cast<float*>(y_t)[(size_t)(mb + j) * N + n] = v;
            }
          }
        } else if (n < N) {
          const int mb = m0 + c * 16;
          if (y_dt == NB_BF16) {
            __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(y_t) + (size_t)mb * N + n;
#pragma unroll
            for (int j = 0; j < 16; ++j)
              if (mb + j < M) dst[(size_t)j * N] = __float2bfloat16_rn(__uint_as_float(r[j]));
          } else {
            float* dst = reinterpret_cast<float*>(y_t) + (size_t)mb * N + n;
#pragma unroll
            for (int j = 0; j < 16; ++j)
              if (mb + j < M) dst[(size_t)j * N] = __uint_as_float(r[j]);
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(s2u(&acc_empty[buf])) : "memory");
    }
  } else if (warp == kFRawWarp) {
    if (elect_one()) {  // ---- TMA producer of the raw weights: row tiles past the matrix arrive as zeros
      int r = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < n_total && ok; t += gridDim.x) {
        const int rt0 = ((t / ks) / m_tiles) * (kFM / 16);
        const int k_lo = (t % ks) * KTs, k_hi = min(KT, k_lo + KTs);
        for (int kb = k_lo >> 1; kb < k_hi >> 1; ++kb) {
          ok = bar_wait(&raw_empty[r], phase ^ 1, abort_flag, status);
          if (!ok) break;
          bar_expect_tx(&raw_full[r], 8u * F::kBytes);
          tma_load_3d(sW + r * kFRawBytes, &map_w, &raw_full[r], 0, kb, rt0);
          if (++r == R) { r = 0; phase ^= 1; }
        }
      }
    }
  } else {
    // ---- dequant producers: thread (row, half) writes 32 weights = 64 bytes of row `row` of the stage.  A warp's lanes are
    // (row, half) with the halves side by side: eight lanes' chunks fall into eight different bank groups
    const int w = warp - kFProducerWarp0;
    const int grp = w / kFProducerWarps, rt0 = 2 * (w % kFProducerWarps);      // group `grp` fills the steps st with st % 4 == grp
    const int r16 = lane >> 1, q2 = lane & 1, g = r16 & 7, hrow = r16 >> 3;
    const uint8_t* raw0 = sW + rt0 * F::kBytes;
    // positions 64 * (grp & 1) .. + 63 of a k-block: this thread's lane group of the unit is 2 * (grp & 1) + q2
    const int sel_off = hrow * 512 + (g * 4 + 2 * (grp & 1) + q2) * 16, tab_off = 1024 + r16 * F::kTabBytes;
    // row r of a K-major tile with 128-byte swizzle: 16-byte chunk c sits at chunk c ^ (r & 7); a row tile is 2 KB
    uint8_t* const rbase = sA + rt0 * 2048 + hrow * 1024 + g * 128;
    uint32_t step0 = 0;                                  // k-steps of all earlier work items (even): stage = step % S, phase = (step / S) & 1
    bool ok = true;
    for (int t = blockIdx.x; t < n_total && ok; t += gridDim.x) {
      const int k_lo = (t % ks) * KTs, steps = min(KT, k_lo + KTs) - k_lo;
      const uint32_t end = step0 + (uint32_t)steps;
      uint32_t st = step0 + (((uint32_t)grp - step0) & (kFGroups - 1));           // the group's first step of this item
      int s = (int)(st % (uint32_t)S);
      uint32_t phase = (st / (uint32_t)S) & 1u;
      for (; st < end; st += kFGroups) {
        const uint32_t kb = st >> 1;                     // k-blocks since the start: the group's are every second one
        const int r = (int)(kb & (uint32_t)(R - 1));
        ok = bar_wait<20>(&raw_full[r], kb / (uint32_t)R & 1u, abort_flag, status);
        if (!ok) break;
        uint4 out[2][4];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint8_t* u = raw0 + r * kFRawBytes + h * F::kBytes;
          const uint4 sel = *reinterpret_cast<const uint4*>(u + sel_off);
          uint32_t T[kT];
#pragma unroll
          for (int j = 0; j < kT / 4; ++j) {
            const uint4 v = *reinterpret_cast<const uint4*>(u + tab_off + 16 * j);
            T[4 * j] = v.x; T[4 * j + 1] = v.y; T[4 * j + 2] = v.z; T[4 * j + 3] = v.w;
          }
          const uint32_t words[4] = {sel.x, sel.y, sel.z, sel.w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            lookup4<BITS>(words[j], T, out[h][j].x, out[h][j].y);              // positions 8j .. 8j+3
            lookup4<BITS>(words[j] >> 16, T, out[h][j].z, out[h][j].w);        // positions 8j+4 .. 8j+7
          }
        }
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(s2u(&raw_empty[r])) : "memory");
        // (a parity tells a phase from its neighbours only: with at least as many stages as groups, the wait for this group's step
        // before implies that the stage is at most one use behind)
        ok = bar_wait<20>(&empty[s], phase ^ 1u, abort_flag, status);
        if (!ok) break;
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int j = 0; j < 4; ++j) *reinterpret_cast<uint4*>(rbase + s * kFABytes + h * 2048 + (((4 * q2 + j) ^ g) << 4)) = out[h][j];
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // generic-proxy stores -> visible to the tensor core
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(s2u(&full[s])) : "memory");
        for (s += kFGroups; s >= S; s -= S) phase ^= 1u;
      }
      step0 += (uint32_t)steps;
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

// Tile plan of one call: token-tile width BN (a multiple of 16 up to 256) and number of k splits.  A k-step of a work
// item costs the longer of the tensor-core time, 2 * BN clocks, and the time the producers need to fill a stage, which
// does not depend on BN (measured: about kProducerClocks); a work item is one k split of one 128 x BN output tile, the
// items run in waves of one per SM.  The plan with the fewest estimated clocks wins: waves * k-steps per item * clocks
// per k-step, plus a charge for the second kernel that adds the splits' results (fixed part + its reads).  Splits keep at least four
// k-steps each and none is empty; inputs of up to 256 operand rows take one token tile.
constexpr int kProducerClocks = 340;
constexpr int kSplitCharge = 3000;
struct FusedPlan { int bn, ks; };
static FusedPlan plan_fused(int rows, int N, int K, int sms) {
  const int KT = K / kFK;
  const int w_tiles = (N + kFM - 1) / kFM;
  FusedPlan best{256, 1};
  double best_cost = 1e30;
  const int bn_hi = rows <= 256 ? std::min(256, (rows + 15) / 16 * 16) : 256;
  const int bn_lo = rows <= 256 ? bn_hi : 96;
  for (int bn = bn_hi; bn >= bn_lo; bn -= 16) {
    const long tiles = (long)w_tiles * ((rows + bn - 1) / bn);
    for (int ks = 1; ks <= 8; ++ks) {
      const int kts = split_steps(KT, ks);
      if (ks > 1 && (kts < 4 || (long)(ks - 1) * kts >= KT)) continue;
      const long waves = (tiles * ks + sms - 1) / sms;
      // the second kernel reads ks slabs of rows x N floats at roughly 3 KB per clock
      const double sum_cost = ks > 1 ? kSplitCharge + (double)ks * rows * N * 4.0 / 3000.0 : 0.0;
      const double cost = (double)waves * kts * std::max(2 * bn, kProducerClocks) + sum_cost;
      if (cost < best_cost * 0.98) { best_cost = cost; best = FusedPlan{bn, ks}; }
    }
  }
  return best;
}

// y (rows x N) = sum over the k splits' fp32 slabs, in split order; four outputs per thread.
__global__ void __launch_bounds__(256) splitk_sum_kernel(const float* __restrict__ partial, int ks, size_t slab, void* __restrict__ y,
                                                         int y_dtype, size_t n4) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (i >= n4) return;
  float4 acc = reinterpret_cast<const float4*>(partial)[i];
  for (int z = 1; z < ks; ++z) {
    const float4 v = reinterpret_cast<const float4*>(partial + (size_t)z * slab)[i];
    acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
  }
  if (y_dtype == NB_BF16) {
    __nv_bfloat162* dst = reinterpret_cast<__nv_bfloat162*>(y) + 2 * i;
    dst[0] = __floats2bfloat162_rn(acc.x, acc.y);
    dst[1] = __floats2bfloat162_rn(acc.z, acc.w);
  } else {
    reinterpret_cast<float4*>(y)[i] = acc;
  }
}

// The stream layout as (row tiles, k-blocks, units of 8-byte elements) with boxes of eight row tiles of one k-block.
static int make_map_units(CUtensorMap* map, const void* base, int unit_bytes, int bpr, int row_tiles) {
  const cuuint64_t dims[3] = {(cuuint64_t)unit_bytes / 8, (cuuint64_t)bpr, (cuuint64_t)row_tiles};
  const cuuint64_t strides[2] = {(cuuint64_t)unit_bytes, (cuuint64_t)bpr * unit_bytes};
  const cuuint32_t box[3] = {(cuuint32_t)unit_bytes / 8, 1, 8};
  return encode_map(map, CU_TENSOR_MAP_DATA_TYPE_INT64, 3, base, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE);
}

}  // namespace nb

using namespace nb;

// Workspace: [256 B status][fp16 operand rows x K][k-split slabs: ks x (M x N) floats]; sized for the worse of the
// one-term (bf16 / fp16) and two-term (fp32) forms of M activation rows.
static size_t fused_partial_bytes(int rows, int M, int N, int K) {
  const int ks = plan_fused(rows, N, K, sm_count()).ks;
  return ks > 1 ? (size_t)ks * M * N * sizeof(float) : 0;
}

extern "C" size_t nb_prefill_fused_workspace_bytes(int M, int N, int K) {
  if (M < 1 || N < 1 || K < kFK) return 0;
  const size_t x_bytes = ((size_t)2 * M * K * 2 + 255) / 256 * 256;
  return 256 + x_bytes + std::max(fused_partial_bytes(M, M, N, K), fused_partial_bytes(2 * M, M, N, K));
}

extern "C" int nb_gemm_prefill_fused(const void* x, int x_dtype, int M, const uint8_t* w_stream, int bits, int N, int K, void* y,
                                     int y_dtype, void* workspace, size_t workspace_bytes, void* stream) {
  if (!x || !w_stream || !y || M < 1 || N < 1 || K < 1) return NB_ERR_ARG;
  if (x_dtype != NB_BF16 && x_dtype != NB_F16 && x_dtype != NB_F32 && x_dtype != NB_F16_TERMS) return NB_ERR_ARG;
  if (y_dtype != NB_BF16 && y_dtype != NB_F32) return NB_ERR_ARG;
  if (bits != 2 && bits != 3 && bits != 4) return NB_ERR_SHAPE;
  if (K % kBlock != 0) return NB_ERR_SHAPE;
  if (!workspace || workspace_bytes < nb_prefill_fused_workspace_bytes(M, N, K)) return NB_ERR_WORKSPACE;
  if ((uintptr_t)workspace % 256 || (uintptr_t)x % 16 || (uintptr_t)w_stream % 16) return NB_ERR_ALIGN;
  if (int rc = check_device()) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  const void* xh = x;
  const int pair = x_dtype == NB_F32 || x_dtype == NB_F16_TERMS ? 1 : 0;
  const int rows = pair ? 2 * M : M;              // rows of the fp16 operand
  uint8_t* dst = reinterpret_cast<uint8_t*>(workspace) + 256;
  if (x_dtype == NB_BF16) {
    const size_t n8 = (size_t)M * K / 8;
    bf16_to_f16_kernel<<<(unsigned)((n8 + 255) / 256), 256, 0, st>>>(reinterpret_cast<const uint4*>(x), reinterpret_cast<uint4*>(dst), n8);
    if (int rc = check_launch()) return rc;
    xh = dst;
  } else if (x_dtype == NB_F32) {
    const size_t n8 = (size_t)M * K / 8;
    f32_to_f16_pair_kernel<<<(unsigned)((n8 + 255) / 256), 256, 0, st>>>(reinterpret_cast<const float4*>(x), reinterpret_cast<uint4*>(dst), M, K);
    if (int rc = check_launch()) return rc;
    xh = dst;
  }
  const int sms = sm_count();
  const FusedPlan plan = plan_fused(rows, N, K, sms);
  const int bn = plan.bn;
  CUtensorMap mx, mw;
  if (int rc = make_map(&mx, xh, rows, K, bn)) return rc;
  if (int rc = make_map_units(&mw, w_stream, bits == 4 ? StreamUnit<4>::kBytes : StreamUnit<3>::kBytes, K / kBlock, (N + 15) / 16)) return rc;
  const int m_tiles = (rows + bn - 1) / bn, w_tiles = (N + kFM - 1) / kFM;
  int ks = plan.ks;
  if (ks > 1 && (N % 4 != 0 || (uintptr_t)y % 16)) ks = 1;       // the summing kernel writes four outputs at a time
  float* partial = reinterpret_cast<float*>(dst + ((size_t)2 * M * K * 2 + 255) / 256 * 256);
  const int grid = std::min(sms, m_tiles * w_tiles * ks);
  int* status = reinterpret_cast<int*>(workspace);
  static bool attr_done[64][5] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  const void* fn = bits == 3 ? (const void*)gemm_fused_kernel<3> : bits == 2 ? (const void*)gemm_fused_kernel<2> : (const void*)gemm_fused_kernel<4>;
  if (!attr_done[dev & 63][bits]) {
    if (cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kFSmem)) return record_cuda_error(e);
    attr_done[dev & 63][bits] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kFThreads);
  cfg.dynamicSmemBytes = kFSmem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  // ahead of its turn only where the launch before wrote the activations, this call's own conversion or the kernel that wrote
  // the terms: whatever wrote the weights has then ended
  cfg.numAttrs = xh != x || x_dtype == NB_F16_TERMS ? 1 : 0;
  int y_tag = y_dtype, rows_arg = rows, n_arg = N, k_arg = K, bn_arg = bn, m_t = m_tiles, w_t = w_tiles, pair_arg = pair;
  void* args[] = {&mx, &mw, &y, &y_tag, &rows_arg, &n_arg, &k_arg, &bn_arg, &m_t, &w_t, &pair_arg, &ks, &partial, &status};
  if (cudaError_t e = cudaLaunchKernelExC(&cfg, fn, args)) return record_cuda_error(e);
  if (ks > 1) {
    const size_t n4 = (size_t)M * N / 4;
    return launch_pdl(splitk_sum_kernel, dim3((unsigned)((n4 + 255) / 256)), dim3(256), 0, st, partial, ks, (size_t)M * N, y, y_dtype, n4);
  }
  return NB_OK;
}
