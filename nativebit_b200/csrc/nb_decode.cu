// Small fused kernels of the decode step around the packed GEMVs (one new token per sequence):
// residual add + RMSNorm, RoPE + KV-cache write, single-query attention over the valid prefix of
// the cache, and SiLU(gate) * up.  All activations are fp32, as in the reference's cached path
// (inference/generate_torch.py:29-38 RMSNorm, :41-60 RoPE on interleaved pairs, :86-97 cache write
// and masked attention, :116-117 SwiGLU).  The position is read from device memory so that the
// step can be replayed from a CUDA graph.
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cooperative_groups.h>

#include <algorithm>
#include <cfloat>
#include <type_traits>

#include "nb_chain.cuh"
#include "nb_common.cuh"
#include "nb_device.cuh"
#include "nb_host.h"
#include "nb_launch.cuh"
#include "../../include/nativebit_b200_layered.h"

namespace nb {

namespace cg = cooperative_groups;

// x[b] += delta[b] (if delta); out[b] = x[b] / sqrt(mean(x[b]^2) + eps) * w.  One CTA per row; the
// row lives in registers (up to 16 elements per thread), so global memory is read exactly once.
__global__ void __launch_bounds__(256) add_rmsnorm_kernel(float* __restrict__ x, const float* __restrict__ delta,
                                                          const float* __restrict__ w, float eps, float* __restrict__ out, int C) {
  __shared__ float red[8];
  constexpr int kPer = 16;
  pdl_enter();
  float* xr = x + (size_t)blockIdx.x * C;
  const float* dr = delta ? delta + (size_t)blockIdx.x * C : nullptr;
  float v[kPer], wv[kPer];
  float ss = 0.f;
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    const int i = threadIdx.x + k * 256;
    v[k] = 0.f; wv[k] = 0.f;
    if (i < C) {
      v[k] = xr[i];
      wv[k] = w[i];
      if (dr) v[k] += dr[i];
    }
  }
#pragma unroll
  for (int k = 0; k < kPer; ++k) ss += v[k] * v[k];
  ss = warp_sum(ss);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) tot += red[i];
  const float inv = 1.0f / sqrtf(tot / (float)C + eps);
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    const int i = threadIdx.x + k * 256;
    if (i < C) {
      if (dr) xr[i] = v[k];
      out[(size_t)blockIdx.x * C + i] = v[k] * inv * wv[k];
    }
  }
}

// Four values at place `i` of row b as two fp16 terms each (saturating, then the rest): terms (B, 2, n4 * 4).
__device__ __forceinline__ void store_terms(void* terms, int b, int n4, int i, float4 v) {
  uint2 hi = make_uint2(f32x2_to_f16x2_sat(v.x, v.y), f32x2_to_f16x2_sat(v.z, v.w));
  const float2 h0 = __half22float2(*reinterpret_cast<const __half2*>(&hi.x)), h1 = __half22float2(*reinterpret_cast<const __half2*>(&hi.y));
  uint2* row = reinterpret_cast<uint2*>(terms) + (size_t)b * 2 * n4 + i;
  row[0] = hi;
  row[n4] = make_uint2(f32x2_to_f16x2_sat(v.x - h0.x, v.y - h0.y), f32x2_to_f16x2_sat(v.z - h1.x, v.w - h1.y));
}

// add_rmsnorm_kernel with its result as the GEMMs' operand: the fp32 row is neither written nor read again by a pass that
// splits it (2 x 13 us of a layer's 1.5 ms at 4096 rows of 2560; bound by its 16 bytes per value).
__global__ void __launch_bounds__(256) add_rmsnorm_terms_kernel(float4* __restrict__ x, const float4* __restrict__ delta,
                                                                const float4* __restrict__ w, float eps, void* __restrict__ terms, int n4) {
  __shared__ float red[8];
  constexpr int kPer = 4;
  const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
  float4 v[kPer], wv[kPer];
#pragma unroll
  for (int k = 0; k < kPer; ++k) wv[k] = (int)threadIdx.x + k * 256 < n4 ? __ldg(w + threadIdx.x + k * 256) : zero4;
  pdl_enter();
  float4* xr = x + (size_t)blockIdx.x * n4;
  const float4* dr = delta ? delta + (size_t)blockIdx.x * n4 : nullptr;
  float ss = 0.f;
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    const int i = threadIdx.x + k * 256;
    v[k] = zero4;
    if (i < n4) {
      v[k] = xr[i];
      if (dr) {
        const float4 d = dr[i];
        v[k].x += d.x; v[k].y += d.y; v[k].z += d.z; v[k].w += d.w;
      }
    }
  }
#pragma unroll
  for (int k = 0; k < kPer; ++k) ss += v[k].x * v[k].x + v[k].y * v[k].y + v[k].z * v[k].z + v[k].w * v[k].w;
  ss = warp_sum(ss);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) tot += red[i];
  const float inv = 1.0f / sqrtf(tot / (float)(4 * n4) + eps);
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    const int i = threadIdx.x + k * 256;
    if (i < n4) {
      if (dr) xr[i] = v[k];
      store_terms(terms, blockIdx.x, n4, i, make_float4(v[k].x * inv * wv[k].x, v[k].y * inv * wv[k].y, v[k].z * inv * wv[k].z, v[k].w * inv * wv[k].w));
    }
  }
}

// qkv (B, 3*H*hd) = [q | k | v]; rotates q and k pairs (2i, 2i+1) by the position's angle, writes
// k and v into the caches (B, H, ctx, hd) at `pos`, q into q_out (B, H, hd).  grid (H, B).
__global__ void rope_kv_kernel(const float* __restrict__ qkv, const float* __restrict__ cos2, const float* __restrict__ sin2,
                               const long long* __restrict__ pos_ptr, float* __restrict__ k_cache, float* __restrict__ v_cache,
                               float* __restrict__ q_out, int H, int hd, int ctx) {
  const int h = blockIdx.x, b = blockIdx.y;
  pdl_enter();                                             // releases after the wait: the attention kernel behind reads the cache early
  const long long pos = *pos_ptr;
  if (pos < 0 || pos >= ctx) return;
  const float* base = qkv + (size_t)b * 3 * H * hd;
  const float* q = base + h * hd;
  const float* k = base + H * hd + h * hd;
  const float* v = base + 2 * H * hd + h * hd;
  const size_t crow = (((size_t)b * H + h) * ctx + pos) * hd;
  for (int i = threadIdx.x; i < hd; i += blockDim.x) {
    const float c = cos2[pos * hd + i], s = sin2[pos * hd + i];
    const int j = i ^ 1;                       // partner of the pair
    const float sign = (i & 1) ? 1.f : -1.f;   // rot = (-x2, x1)
    q_out[((size_t)b * H + h) * hd + i] = q[i] * c + sign * q[j] * s;
    k_cache[crow + i] = k[i] * c + sign * k[j] * s;
    v_cache[crow + i] = v[i];
  }
}

// Single-query attention for one (head, batch): softmax over keys 0..pos, weighted sum of values; out[b, out_offset + h*hd + d].
// grid (H, B, S) in clusters of S CTAs along z: the CTAs of a cluster split the keys of one head into S contiguous ranges (the
// whole GPU works on the 32 heads of a batch-1 step instead of 32 SMs).  Inside a CTA a warp takes 8 keys per iteration and
// keeps running maximum, denominator and numerator for itself: for the scores four lanes share a key (16-byte loads, two
// shuffles), for the values a lane owns four head dimensions of all 8 keys.  Keys and values of the first iteration are
// requested before the dependency wait, so a context of up to 64*S keys costs one memory round trip.  One barrier later a thread
// per dimension merges the warps and pushes the CTA's result into rank 0's shared memory; behind the cluster's barrier rank 0
// merges those from its own.  What bounds it is that chain of latencies: with three more block-wide barriers around the
// softmax and rank 0 reading the others' results one remote load at a time, a step of the 2.2B decoder with 12 layers took 418 instead of 391 us.
// head_dim a multiple of 4, <= 128.
//
// When `qkv` is given (B, 3*H*hd = [q|k|v]) the kernel first does the work of rope_kv_kernel for its
// head: it rotates q and k by the position's angle, the CTA that owns key `pos` writes k and v into
// the caches, and all attend with the rotated q, so the step needs one launch instead of two.
constexpr int kAttnWarps = 8, kAttnMaxSplit = 8;
constexpr int kAttnKeysPerIter = kAttnWarps * 8;
static int attn_per_max(int ctx, int S) { return (((ctx + S - 1) / S) + 7) & ~7; }
static size_t attn_limit_floats(int ctx, int hd, int S) { return (size_t)attn_per_max(ctx, S) + (size_t)(2 + kAttnWarps) * hd + 4; }
static size_t attn_smem_floats(int hd) { return (size_t)(1 + kAttnWarps) * hd + (size_t)kAttnMaxSplit * (hd + 4); }

// kTerms: `out` is the terms buffer of the chain's next launch, out_stride columns wide, not rows of floats.
template <bool kTerms>
__global__ void __launch_bounds__(kAttnWarps * 32) decode_attention_kernel(
    const float* __restrict__ q, float* k_cache, float* v_cache, const long long* __restrict__ pos_ptr, float* __restrict__ out,
    int H, int hd, int ctx, int out_stride, int out_offset, const float* __restrict__ qkv, const float* __restrict__ cos2,
    const float* __restrict__ sin2) {
  extern __shared__ __align__(16) float sm[];  // q | per-warp numerators | rank 0: the CTAs' numerator, maximum, denominator
  __shared__ float s_m[kAttnWarps], s_l[kAttnWarps];
  cg::cluster_group cluster = cg::this_cluster();
  const int S = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int h = blockIdx.x, b = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  asm volatile("griddepcontrol.launch_dependents;");
  // The position was written at the end of the step before, and the cache rows below it in earlier steps: neither
  // depends on the launch before this one, so this CTA's first keys and values are requested BEFORE the dependency
  // wait and arrive while the qkv matvec drains.  Only the row this step writes (position pos) is fetched after it.
  long long pos = *pos_ptr;
  if (pos < 0) return;  // the same for every CTA of the cluster
  asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");     // this CTA runs: others may write to its shared memory
  if (pos >= ctx) pos = ctx - 1;
  const int n = (int)pos + 1, hd4 = hd >> 2;
  const int per = (((n + S - 1) / S) + 7) & ~7;
  const int k0 = rank * per;
  const int cnt = max(0, min(n, k0 + per) - k0);
  float* qs = sm;
  float* part = qs + hd;
  float* slots = part + kAttnWarps * hd;
  const int slot = hd + 4;
  const size_t head = ((size_t)b * H + h);
  float* kb = k_cache + head * ctx * hd;
  float* vb = v_cache + head * ctx * hd;
  const int kq = lane >> 2, t = lane & 3;
  const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
  float4 kv[8], vv[8];          // keys and values of an iteration
  auto load = [&](int it, int skip) {
    const int j0 = (it * kAttnWarps + warp) * 8;
    const bool ld = j0 + kq < cnt && k0 + j0 + kq != skip;
    const float4* krow = reinterpret_cast<const float4*>(kb + (size_t)(k0 + j0 + kq) * hd);
#pragma unroll
    for (int i = 0; i < 8; ++i) kv[i] = (ld && t + 4 * i < hd4) ? krow[t + 4 * i] : zero4;
#pragma unroll
    for (int u = 0; u < 8; ++u)
      vv[u] = (j0 + u < cnt && k0 + j0 + u != skip && lane < hd4) ? *reinterpret_cast<const float4*>(vb + (size_t)(k0 + j0 + u) * hd + 4 * lane)
                                                                   : zero4;
  };
  load(0, (int)pos);
  float c_pre = 0.f, s_pre = 0.f;  // this thread's entry of the rotary tables (head_dim <= 128 < threads per CTA)
  if (qkv && tid < hd) { c_pre = cos2[pos * hd + tid]; s_pre = sin2[pos * hd + tid]; }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (tid < hd) {
    if (qkv) {
      const float* qh = qkv + (size_t)b * 3 * H * hd + h * hd;
      const float *kh = qh + H * hd, *vh = kh + H * hd;
      const int j = tid ^ 1;
      const float sign = (tid & 1) ? 1.f : -1.f;   // rot = (-x2, x1) on interleaved pairs
      qs[tid] = (qh[tid] * c_pre + sign * qh[j] * s_pre) * rsqrtf((float)hd);
      if (pos >= k0 && pos < k0 + cnt) {
        kb[(size_t)pos * hd + tid] = kh[tid] * c_pre + sign * kh[j] * s_pre;
        vb[(size_t)pos * hd + tid] = vh[tid];
      }
    } else {
      qs[tid] = q[head * hd + tid] * rsqrtf((float)hd);
    }
  }
  __syncthreads();  // also orders the cache row written above before the reads below (same CTA)

  const int iters = (cnt + kAttnKeysPerIter - 1) / kAttnKeysPerIter;
  {  // the row written in this step (by this CTA above, or by the launch before): now it can be read
    const int jl = (int)pos - k0 - warp * 8;                 // its place among this warp's first keys
    if (jl >= 0 && jl < 8 && (int)pos - k0 < cnt) {
      if (kq == jl) {
        const float4* krow = reinterpret_cast<const float4*>(kb + (size_t)pos * hd);
#pragma unroll
        for (int i = 0; i < 8; ++i) kv[i] = (t + 4 * i < hd4) ? krow[t + 4 * i] : zero4;
      }
      const float4 vp = lane < hd4 ? *reinterpret_cast<const float4*>(vb + (size_t)pos * hd + 4 * lane) : zero4;
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (u == jl) vv[u] = vp;
    }
  }
  float mx = -FLT_MAX, sum = 0.f;
  float4 acc = zero4;
#pragma unroll 1
  for (int it = 0; it < iters; ++it) {
    if (it > 0) load(it, -1);
    const int j0 = (it * kAttnWarps + warp) * 8;
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (t + 4 * i < hd4) {
        const float4 qv = reinterpret_cast<const float4*>(qs)[t + 4 * i];
        s += qv.x * kv[i].x + qv.y * kv[i].y + qv.z * kv[i].z + qv.w * kv[i].w;
      }
    }
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    const bool valid = j0 + kq < cnt;
    if (!valid) s = -FLT_MAX;
    float m_new = fmaxf(mx, s);
    m_new = fmaxf(m_new, __shfl_xor_sync(0xffffffffu, m_new, 4));
    m_new = fmaxf(m_new, __shfl_xor_sync(0xffffffffu, m_new, 8));
    m_new = fmaxf(m_new, __shfl_xor_sync(0xffffffffu, m_new, 16));
    const float e = valid ? __expf(s - m_new) : 0.f;
    const float keep = __expf(mx - m_new);
    mx = m_new;
    float e_sum = e;
    e_sum += __shfl_xor_sync(0xffffffffu, e_sum, 4);
    e_sum += __shfl_xor_sync(0xffffffffu, e_sum, 8);
    e_sum += __shfl_xor_sync(0xffffffffu, e_sum, 16);
    sum = sum * keep + e_sum;
    acc.x *= keep; acc.y *= keep; acc.z *= keep; acc.w *= keep;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const float pj = __shfl_sync(0xffffffffu, e, 4 * u);
      if (j0 + u < cnt) {       // (a row past the range is not looked at, whatever its memory holds)
        acc.x += pj * vv[u].x; acc.y += pj * vv[u].y; acc.z += pj * vv[u].z; acc.w += pj * vv[u].w;
      }
    }
  }
  if (lane < hd4) reinterpret_cast<float4*>(part + warp * hd)[lane] = acc;
  if (lane == 0) { s_m[warp] = mx; s_l[warp] = sum; }
  __syncthreads();
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  if (tid < hd) {               // a warp without keys has maximum -FLT_MAX: its weight is exp(-inf) = 0, or it has nothing to weigh
    float m_all = s_m[0];
#pragma unroll
    for (int w = 1; w < kAttnWarps; ++w) m_all = fmaxf(m_all, s_m[w]);
    float num = 0.f, den = 0.f;
#pragma unroll
    for (int w = 0; w < kAttnWarps; ++w) {
      const float e = __expf(s_m[w] - m_all);
      num += e * part[w * hd + tid];
      den += e * s_l[w];
    }
    float* dst = cluster.map_shared_rank(slots, 0) + rank * slot;
    dst[tid] = num;
    if (tid == 0) { dst[hd] = m_all; dst[hd + 1] = den; }
  }
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  if (rank == 0 && tid < hd) {
    float m_all = -FLT_MAX;
#pragma unroll
    for (int r = 0; r < kAttnMaxSplit; ++r)
      if (r < S) m_all = fmaxf(m_all, slots[r * slot + hd]);
    float num = 0.f, den = 0.f;
#pragma unroll
    for (int r = 0; r < kAttnMaxSplit; ++r) {  // a rank without keys has max -FLT_MAX: its weight is exp(-inf) = 0
      if (r < S) {
        const float w = __expf(slots[r * slot + hd] - m_all);
        num += w * slots[r * slot + tid];
        den += w * slots[r * slot + hd + 1];
      }
    }
    if (kTerms) store_chain_terms(reinterpret_cast<uint8_t*>(out), out_stride >> 7, b, out_offset + h * hd + tid, num / den);
    else out[(size_t)b * out_stride + out_offset + h * hd + tid] = num / den;
  }
}

// The same with one CTA per (head, batch), for calls whose heads alone fill the GPU (taken where the kernel above would split
// a head over one or two CTAs; where it splits over four or eight, splitting wins).  Bound by the bytes of the cached
// keys and values.  A warp takes eight keys at a time, every fourth such chunk: its keys and values travel through the warp's
// own ring of asynchronous copies (two chunks ahead, no registers held), and scores, running maximum, denominator and numerator
// stay in the warp until one merge at the end, so no barrier separates the scores from the values.  The row this step writes
// never comes from the cache: warp 0 starts from it.  Against the cluster kernel over 149 ... 1024 heads of 64, 80 and 128 and
// 5 ... 8000 keys: 0.68 of its time in the middle of 230 sizes (256 heads of 64: 500 keys 21 -> 18 us), nowhere longer but for 256
// heads of 128 over 4000 and 8000 keys (167 -> 171, 319 -> 335 us: 6.3 TB/s, and 148 SMs hold 256 CTAs unevenly); the length
// is known on the device only, so those take it as well.
constexpr int kWideWarps = 4, kWideKeys = 8, kWideD = 3;
static size_t wide_smem_floats(int hd) { return (size_t)kWideWarps * kWideD * 2 * kWideKeys * hd + (size_t)(3 + kWideWarps) * hd; }

template <bool kTerms>
__global__ void __launch_bounds__(kWideWarps * 32) decode_attention_wide_kernel(
    const float* __restrict__ q, float* k_cache, float* v_cache, const long long* __restrict__ pos_ptr, float* __restrict__ out,
    int H, int hd, int ctx, int out_stride, int out_offset, const float* __restrict__ qkv, const float* __restrict__ cos2,
    const float* __restrict__ sin2) {
  extern __shared__ __align__(16) float sm[];  // per warp kWideD stages of keys | values, then q | key | value of this step | outputs
  __shared__ float s_m[kWideWarps], s_l[kWideWarps];
  const int h = blockIdx.x, b = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  asm volatile("griddepcontrol.launch_dependents;");
  // as above: position and older rows do not depend on the launch before this one
  long long pos = *pos_ptr;
  if (pos < 0) return;
  if (pos >= ctx) pos = ctx - 1;
  const int n = (int)pos, hd4 = hd >> 2, n_chunks = (n + kWideKeys - 1) / kWideKeys;
  const size_t head = (size_t)b * H + h;
  float* kb = k_cache + head * ctx * hd;
  float* vb = v_cache + head * ctx * hd;
  const int half = kWideKeys * hd, stage_floats = 2 * half;
  float* ring = sm + warp * kWideD * stage_floats;
  float* qs = sm + kWideWarps * kWideD * stage_floats;
  float *ks = qs + hd, *vs = ks + hd, *part = vs + hd;
  int rq = warp, rq_stage = 0;
  auto request = [&]() {      // the warp's next chunk, a contiguous span of each cache
    if (rq < n_chunks) {
      const int k0 = rq * kWideKeys, n4 = min(kWideKeys, n - k0) * hd4;
      float4* dst = reinterpret_cast<float4*>(ring + rq_stage * stage_floats);
      const float4* ksrc = reinterpret_cast<const float4*>(kb + (size_t)k0 * hd);
      const float4* vsrc = reinterpret_cast<const float4*>(vb + (size_t)k0 * hd);
      for (int i = lane; i < n4; i += 32) cp_async16(dst + i, ksrc + i);
      for (int i = lane; i < n4; i += 32) cp_async16(dst + kWideKeys * hd4 + i, vsrc + i);
      rq += kWideWarps;
    }
    if (++rq_stage == kWideD) rq_stage = 0;
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll 1
  for (int i = 0; i < kWideD - 1; ++i) request();
  float c_pre = 0.f, s_pre = 0.f;
  if (qkv && tid < hd) { c_pre = cos2[pos * hd + tid]; s_pre = sin2[pos * hd + tid]; }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (tid < hd) {             // head_dim <= 128 threads
    if (qkv) {
      const float* qh = qkv + (size_t)b * 3 * H * hd + h * hd;
      const float* kh = qh + H * hd;
      const int j = tid ^ 1;
      const float sign = (tid & 1) ? 1.f : -1.f;   // rot = (-x2, x1) on interleaved pairs
      const float k = kh[tid] * c_pre + sign * kh[j] * s_pre, v = kh[H * hd + tid];
      qs[tid] = (qh[tid] * c_pre + sign * qh[j] * s_pre) * rsqrtf((float)hd);
      ks[tid] = k;
      vs[tid] = v;
      kb[(size_t)pos * hd + tid] = k;
      vb[(size_t)pos * hd + tid] = v;
    } else {
      qs[tid] = q[head * hd + tid] * rsqrtf((float)hd);
      ks[tid] = kb[(size_t)pos * hd + tid];
      vs[tid] = vb[(size_t)pos * hd + tid];
    }
  }
  __syncthreads();

  const int kq = lane >> 2, t = lane & 3;
  const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
  float4 qv[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) qv[i] = t + 4 * i < hd4 ? reinterpret_cast<const float4*>(qs)[t + 4 * i] : zero4;
  float mx = -FLT_MAX, sum = 0.f;
  float4 acc = zero4;
  if (warp == 0) {
    float s = 0.f;
    if (lane < hd4) {
      const float4 a = reinterpret_cast<const float4*>(qs)[lane], c = reinterpret_cast<const float4*>(ks)[lane];
      s = a.x * c.x + a.y * c.y + a.z * c.z + a.w * c.w;
      acc = reinterpret_cast<const float4*>(vs)[lane];
    }
    mx = warp_sum(s);
    sum = 1.f;
  }
  int stage = 0;
#pragma unroll 1
  for (int c = warp; c < n_chunks; c += kWideWarps) {
    request();
    asm volatile("cp.async.wait_group %0;" ::"n"(kWideD - 1) : "memory");
    __syncwarp();
    const float* kst = ring + stage * stage_floats;
    const int cnt = min(kWideKeys, n - c * kWideKeys);
    float s = 0.f;
    if (kq < cnt) {
      const float4* krow = reinterpret_cast<const float4*>(kst + kq * hd);
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (t + 4 * i < hd4) {
          const float4 kv = krow[t + 4 * i];
          s += qv[i].x * kv.x + qv[i].y * kv.y + qv[i].z * kv.z + qv[i].w * kv.w;
        }
    }
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    if (kq >= cnt) s = -FLT_MAX;
    float m_new = fmaxf(mx, s);
    m_new = fmaxf(m_new, __shfl_xor_sync(0xffffffffu, m_new, 4));
    m_new = fmaxf(m_new, __shfl_xor_sync(0xffffffffu, m_new, 8));
    m_new = fmaxf(m_new, __shfl_xor_sync(0xffffffffu, m_new, 16));
    const float e = kq < cnt ? __expf(s - m_new) : 0.f;
    const float keep = __expf(mx - m_new);
    mx = m_new;
    float e_sum = e;
    e_sum += __shfl_xor_sync(0xffffffffu, e_sum, 4);
    e_sum += __shfl_xor_sync(0xffffffffu, e_sum, 8);
    e_sum += __shfl_xor_sync(0xffffffffu, e_sum, 16);
    sum = sum * keep + e_sum;
    acc.x *= keep; acc.y *= keep; acc.z *= keep; acc.w *= keep;
    const float4* vst = reinterpret_cast<const float4*>(kst + half);
#pragma unroll
    for (int u = 0; u < kWideKeys; ++u) {
      const float pj = __shfl_sync(0xffffffffu, e, 4 * u);
      if (u < cnt && lane < hd4) {
        const float4 vv = vst[u * hd4 + lane];
        acc.x += pj * vv.x; acc.y += pj * vv.y; acc.z += pj * vv.z; acc.w += pj * vv.w;
      }
    }
    if (++stage == kWideD) stage = 0;
    __syncwarp();             // every lane is done with this stage before it is requested again
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  if (lane < hd4) reinterpret_cast<float4*>(part + warp * hd)[lane] = acc;
  if (lane == 0) { s_m[warp] = mx; s_l[warp] = sum; }
  __syncthreads();
  if (tid < hd) {             // a warp without keys has maximum -FLT_MAX: its weight is exp(-inf) = 0
    float m_all = s_m[0];
#pragma unroll
    for (int w = 1; w < kWideWarps; ++w) m_all = fmaxf(m_all, s_m[w]);
    float num = 0.f, den = 0.f;
#pragma unroll
    for (int w = 0; w < kWideWarps; ++w) {
      const float e = __expf(s_m[w] - m_all);
      num += e * part[w * hd + tid];
      den += e * s_l[w];
    }
    if (kTerms) store_chain_terms(reinterpret_cast<uint8_t*>(out), out_stride >> 7, b, out_offset + h * hd + tid, num / den);
    else out[(size_t)b * out_stride + out_offset + h * hd + tid] = num / den;
  }
}

// Cluster size: enough CTAs for a few waves of the GPU, at most 8 per head.
static int attn_split(int B, int H) {
  const int want = 592 / std::max(1, B * H);
  return want >= 8 ? 8 : want >= 4 ? 4 : want >= 2 ? 2 : 1;
}

template <bool kTerms, typename... Args>
static int launch_attention(int B, int H, int hd, int ctx, cudaStream_t st, Args... args) {
  const int S = attn_split(B, H);
  if (attn_limit_floats(ctx, hd, S) * sizeof(float) > 48 * 1024) return NB_ERR_SHAPE;      // the contexts that are taken stay what they were
  if (S <= 2) {     // more heads than SMs: no split is needed to occupy the GPU
    static bool done[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (!done[dev & 63]) {
      if (cudaError_t e = cudaFuncSetAttribute(decode_attention_wide_kernel<kTerms>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)(wide_smem_floats(128) * sizeof(float))))
        return record_cuda_error(e);
      done[dev & 63] = true;
    }
    return launch_pdl(decode_attention_wide_kernel<kTerms>, dim3(H, B), dim3(kWideWarps * 32), wide_smem_floats(hd) * sizeof(float), st, args...);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(H, B, S);
  cfg.blockDim = dim3(kAttnWarps * 32);
  cfg.dynamicSmemBytes = attn_smem_floats(hd) * sizeof(float);
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 1;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = S;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return record_cuda_error(cudaLaunchKernelEx(&cfg, decode_attention_kernel<kTerms>, args...));
}

// The pairs (x, y) and (z, w) turned by their angles.
__device__ __forceinline__ float4 turn_pairs(float4 x, float2 c, float2 s) {
  return make_float4(x.x * c.x - x.y * s.x, x.y * c.x + x.x * s.x, x.z * c.y - x.w * s.y, x.w * c.y + x.z * s.y);
}

// Causal attention of a prompt (or a chunk of one that continues a cache of pos0 keys), two launches per layer: the first
// rotates the chunk's keys into the cache and copies its values there, the second is softmax(q k^T / sqrt(hd)) v over the
// cached keys 0 .. pos0 + t for query t (inference/generate_torch.py:41-60 RoPE, :86-97 cache write and masked attention).
// The second starts beside the first and turns its queries meanwhile.
// (Rotating the keys wherever they are read needs one launch, but every CTA then waits for its loads: 381 us against the
// 337 us of both launches, 8 sequences of 512 tokens, 32 heads of 80.)
__global__ void __launch_bounds__(256) prompt_keys_kernel(const float* __restrict__ qkv, const float* __restrict__ cos2,
                                                          const float* __restrict__ sin2, float* __restrict__ k_cache,
                                                          float* __restrict__ v_cache, int T, int H, int hd, int ctx, int pos0) {
  asm volatile("griddepcontrol.launch_dependents;");        // the attention behind it turns its queries meanwhile
  const int t = blockIdx.x, b = blockIdx.y, quarter = hd >> 2;
  const float* row = qkv + (size_t)(b * T + t) * 3 * H * hd + H * hd;
  for (int i = threadIdx.x; i < H * quarter; i += 256) {
    const int h = i / quarter, d = (i - h * quarter) * 4;
    const float4 k = *reinterpret_cast<const float4*>(row + 4 * i), v = *reinterpret_cast<const float4*>(row + H * hd + 4 * i);
    const size_t ri = (size_t)(pos0 + t) * hd + d, at = ((size_t)b * H + h) * (size_t)ctx * hd + ri;
    *reinterpret_cast<float4*>(k_cache + at) = turn_pairs(k, make_float2(cos2[ri], cos2[ri + 2]), make_float2(sin2[ri], sin2[ri + 2]));
    *reinterpret_cast<float4*>(v_cache + at) = v;
  }
}

// grid (H, B, ceil(T / BQ)): a CTA owns BQ = 8 R queries of one head (all heads' longest rows first); it walks the cached keys
// in chunks of PK staged in shared memory by asynchronous copies — a chunk's values arrive while its scores are formed, the
// next chunk's keys while the values are added — and keeps a running maximum, denominator and numerator per query.
//
// Everything is fp32 multiply-adds, so the floor is the fp32 pipe (74 TFLOP/s); what decides is how many operands a
// multiply-add costs.  Scores: a thread owns R queries x PK / 16 keys, and every 16-byte load feeds packed two-wide
// multiply-adds along the head dimension (12 loads per 64 of them at R = 8).  Values: the same thread owns its R queries x
// 2 * NP head dimensions (pairs 16 apart) for every second four keys — eight lanes of a half-warp take the even fours, eight
// the odd ones, and the halves meet once at the end — so the weights cross shared memory inside a half-warp only.
// head_dim a multiple of 4, <= 128; NP pairs per thread cover 16 * NP >= head_dim.  Two CTAs share an SM.  PK is 64, and 32 for
// tiles of 16 queries, which are taken where 32 keys are all there are.
constexpr int prompt_pairs(int hd) { return hd <= 32 ? 2 : hd <= 64 ? 4 : hd <= 80 ? 5 : 8; }
// Floats behind the values that the spare pairs of the last row read (and nobody uses): all 16 * NP dimensions of that row
// end before the weights, which other warps are writing.
constexpr int kPromptSpare = 40;
constexpr bool prompt_spare_covers() {
  for (int hd = 4; hd <= 128; hd += 4)
    if (16 * prompt_pairs(hd) > hd + 4 + kPromptSpare) return false;
  return true;
}
static_assert(prompt_spare_covers() && kPromptSpare % 4 == 0, "spare pairs of the last value row");
__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}

__device__ __forceinline__ void copy16_or_zero(float* dst, const float* src, bool there) {   // asynchronous, global -> shared
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(there ? 16 : 0) : "memory");
}

// What bounds it: two warps per scheduler that wait for their own loads; 58 % of the multiply-add pipe's slots are used at eight
// prompts of 512 tokens, 32 heads of 80 (333 us).  Two steps of the scores' loop in one put the second one's loads ahead of the first one's sums:
// one prompt of 512 tokens 58.7 -> 51.3 us, of 128 tokens 17.6 -> 15.7; with 64 queries of heads of 80 the registers for that are not
// there (333 -> 341), so that form takes one.  Three CTAs of 48 or 32 queries per SM: 361, 348.
template <int R, int PK, int NP>
__global__ void __launch_bounds__(128, 2) prefill_attention_kernel(
    const float* __restrict__ qkv, const float* __restrict__ cos2, const float* __restrict__ sin2, const float* __restrict__ k_cache,
    const float* __restrict__ v_cache, float* __restrict__ out, int T, int H, int hd, int ctx, int pos0, int out_stride, int out_offset,
    float scale) {
  constexpr int NT = 128, BQ = 8 * R, KI = PK / 16, kPStride = PK + 4;
  extern __shared__ __align__(16) float psm[];
  const int hdp = hd + 4;                       // row stride: 16-byte aligned, eight consecutive rows on different banks
  float* q_s = psm;                             // [BQ][hdp]
  float* k_s = q_s + BQ * hdp;                  // [PK][hdp]
  float* v_s = k_s + PK * hdp;                  // [PK][hdp]
  float* p_s = v_s + PK * hdp + kPromptSpare;   // [BQ][kPStride]
  const int tid = threadIdx.x, h = blockIdx.x, b = blockIdx.y, q0 = ((int)gridDim.z - 1 - (int)blockIdx.z) * BQ;
  const int row3 = 3 * H * hd, quarter = hd >> 2, rcp = 65536 / quarter + 1;      // i / quarter = i * rcp >> 16 for i < 2048
  const size_t cbase = ((size_t)b * H + h) * (size_t)ctx * hd;
  // this tile's queries, rotated (rows past the prompt's end repeat its last query and are not written)
#pragma unroll 2
  for (int i = tid; i < BQ * quarter; i += NT) {
    const int r = (i * rcp) >> 16, d = (i - r * quarter) * 4, t = min(q0 + r, T - 1);
    const size_t ri = (size_t)(pos0 + t) * hd + d;
    *reinterpret_cast<float4*>(q_s + r * hdp + d) = turn_pairs(*reinterpret_cast<const float4*>(qkv + (size_t)(b * T + t) * row3 + h * hd + d),
                                                               make_float2(cos2[ri], cos2[ri + 2]), make_float2(sin2[ri], sin2[ri + 2]));
  }

  asm volatile("griddepcontrol.wait;" ::: "memory");      // the chunk's keys and values are in the caches
  const int ty = tid >> 4, tx = tid & 15;       // scores: queries R ty .. + R - 1, keys tx + 16 i
  const int upper = (tid >> 3) & 1, tx2 = tid & 7;      // values: the same queries, one half of the keys, dimensions 2 tx2 + 16 i and the next
  const int kmax = pos0 + min(q0 + BQ - 1, T - 1);      // last key any query of this tile may see
  float m[R], l[R];
  unsigned long long acc[R][NP];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    m[r] = -INFINITY;
    l[r] = 0.f;
#pragma unroll
    for (int i = 0; i < NP; ++i) acc[r][i] = 0ull;
  }

  auto stage = [&](float* dst, const float* cache, int kc) {       // keys or values kc .. kc + PK - 1, zeros past kmax
    const float* src = cache + cbase + (size_t)kc * hd;
    const int there = (kmax - kc + 1) * quarter;
    for (int i = tid; i < PK * quarter; i += NT) {
      const int j = (i * rcp) >> 16;
      copy16_or_zero(dst + i * 4 + j * 4, src + (i < there ? i * 4 : 0), i < there);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  stage(k_s, k_cache, 0);
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  stage(v_s, v_cache, 0);

  for (int kc = 0; kc <= kmax; kc += PK) {
    float s[R][KI];
    {
      unsigned long long sum[R][KI];
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int i = 0; i < KI; ++i) sum[r][i] = 0ull;
      const float* qr = q_s + ty * R * hdp;
      const float* kr = k_s + tx * hdp;
      constexpr int kSteps = R == 8 && NP == 5 ? 1 : 2;
#pragma unroll kSteps
      for (int d = 0; d < hd; d += 4) {
        ulonglong2 y[KI];
#pragma unroll
        for (int i = 0; i < KI; ++i) y[i] = *reinterpret_cast<const ulonglong2*>(kr + 16 * i * hdp + d);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(qr + r * hdp + d);
#pragma unroll
          for (int i = 0; i < KI; ++i) { fma2(sum[r][i], x.x, y[i].x); fma2(sum[r][i], x.y, y[i].y); }
        }
      }
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int i = 0; i < KI; ++i) {
          const float2 e = unpack2(sum[r][i]);
          s[r][i] = (e.x + e.y) * scale;
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                            // this chunk's values are here, and nobody reads its keys any more
    if (kc + PK <= kmax) stage(k_s, k_cache, kc + PK);
    if (kc + PK - 1 > pos0 + q0) {              // some query of the tile does not see all keys of the chunk
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int my_pos = pos0 + min(q0 + R * ty + r, T - 1);
#pragma unroll
        for (int i = 0; i < KI; ++i)
          if (kc + tx + 16 * i > my_pos) s[r][i] = -INFINITY;
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      float cm = s[r][0];
#pragma unroll
      for (int i = 1; i < KI; ++i) cm = fmaxf(cm, s[r][i]);
#pragma unroll
      for (int o = 1; o < 16; o <<= 1) cm = fmaxf(cm, __shfl_xor_sync(0xffffffffu, cm, o));
      const float m_new = fmaxf(m[r], cm);      // finite from the first chunk on: key 0 is visible to every query
      const float corr = expf(m[r] - m_new);
      m[r] = m_new;
      float ps = 0.f;
#pragma unroll
      for (int i = 0; i < KI; ++i) {
        const float e = expf(s[r][i] - m_new);
        p_s[(R * ty + r) * kPStride + tx + 16 * i] = e;
        ps += e;
      }
      l[r] = l[r] * corr + ps;                  // this thread's keys; the sixteen parts meet at the end
      const unsigned long long c2 = pack2(corr, corr);
#pragma unroll
      for (int i = 0; i < NP; ++i) asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(acc[r][i]) : "l"(c2));
    }
    __syncwarp();                               // the sixteen threads of a query are lanes of one warp
    const float* pr = p_s + R * ty * kPStride;
    const float* vr = v_s + 2 * tx2;
    const int jn = min(PK, kmax - kc + 1);      // the weights past it are zero
#pragma unroll 1
    for (int j = upper * 4; j < jn; j += 8) {
      float4 w[R];
#pragma unroll
      for (int r = 0; r < R; ++r) w[r] = *reinterpret_cast<const float4*>(pr + r * kPStride + j);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        unsigned long long y[NP];
#pragma unroll
        for (int i = 0; i < NP; ++i) y[i] = *reinterpret_cast<const unsigned long long*>(vr + (j + e) * hdp + 16 * i);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const float x = e == 0 ? w[r].x : e == 1 ? w[r].y : e == 2 ? w[r].z : w[r].w;
          const unsigned long long x2 = pack2(x, x);
#pragma unroll
          for (int i = 0; i < NP; ++i) fma2(acc[r][i], x2, y[i]);
        }
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                            // the next chunk's keys are here, and nobody reads these values any more
    if (kc + PK <= kmax) stage(v_s, v_cache, kc + PK);
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) l[r] += __shfl_xor_sync(0xffffffffu, l[r], o);
    const float inv = 1.f / l[r];
    const int t = q0 + R * ty + r;
    float* o = out + (size_t)(b * T + t) * out_stride + out_offset + h * hd + 2 * tx2;
#pragma unroll
    for (int i = 0; i < NP; ++i) {              // the two halves of the keys
      float2 v = unpack2(acc[r][i]);
      v.x += __shfl_xor_sync(0xffffffffu, v.x, 8);
      v.y += __shfl_xor_sync(0xffffffffu, v.y, 8);
      if (t < T && upper == (r & 1) && 2 * tx2 + 16 * i < hd) *reinterpret_cast<float2*>(o + 16 * i) = make_float2(v.x * inv, v.y * inv);
    }
  }
}

template <int R, int NP, typename... Args>
static int launch_prefill_attention(int B, int T, int H, int hd, cudaStream_t st, Args... args) {
  constexpr int BQ = 8 * R, PK = R == 2 ? 32 : 64;
  const size_t smem = (size_t)((BQ + 2 * PK) * (hd + 4) + kPromptSpare + BQ * (PK + 4)) * sizeof(float);      // <= 92 KB
  static bool attr_done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_done[dev & 63]) {
    if (cudaError_t e = cudaFuncSetAttribute(prefill_attention_kernel<R, PK, NP>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024))
      return record_cuda_error(e);
    attr_done[dev & 63] = true;
  }
  return launch_pdl(prefill_attention_kernel<R, PK, NP>, dim3(H, B, (T + BQ - 1) / BQ), dim3(128), smem, st, args...);
}

// Tiles of 64 queries stage every key half as often as tiles of 32; short or few prompts take the latter, which puts
// twice as many SMs to work on them, and very short ones (one chunk of 32 keys in all) tiles of 16, whose padding and shared
// memory are half of that again.  32 sequences x 32 heads of 80, 64 / 32 / 16 queries: 5 tokens 36.9 / 25.1 / 14.9 us,
// 17 tokens 42.0 / 29.9 us; one sequence, 5 tokens 8.7 / 7.7 / 5.9 us.  Heads wider than 80 always take 32: with 64 only chunks of
// 32 keys fit beside them.  64 | 32 queries: 8 x 500 tokens, 16 heads of 128 296 | 283, 1 x 4000, 8 of 128 1023 | 888, 16 x 200, 16 of
// 128 171 | 139, 8 x 300, 8 of 88 68.7 | 55.1, 32 x 64, 8 of 128 25.2 | 25.2.
template <int NP, typename... Args>
static int prefill_attention_tile(int B, int T, int H, int hd, int pos0, cudaStream_t st, Args... args) {
  if (T <= 16 && pos0 + T <= 32) return launch_prefill_attention<2, NP>(B, T, H, hd, st, args...);
  if constexpr (NP <= 5)
    if (T > 32 && (long long)B * H * ((T + 63) / 64) >= 2 * sm_count()) return launch_prefill_attention<8, NP>(B, T, H, hd, st, args...);
  return launch_prefill_attention<4, NP>(B, T, H, hd, st, args...);
}

// The tied LM head of one sequence as a matvec over the bf16 embedding table, with the final residual add + RMSNorm
// in front and the soft-cap + arg-max behind it (inference/generate_torch.py:155-160 and :300-310): logits[v] =
// cap * tanh(dot(table[v], norm(x + delta) * w) / cap).  HBM-bound (164 MB per token at V = 32000, C = 2560): CTA b
// owns the table rows [V*b/G, V*(b+1)/G); a warp takes every tenth of them through its own ring of 16-byte
// asynchronous copies (four slots of one row at C = 2560: three rows are in flight while one is multiplied, 150 KB per SM
// on the way — plain loads were sunk to their uses by the compiler, four in flight per lane) and multiplies them
// with the activations staged once in shared memory as fp32 (bf16 x fp32 products are exact in fp32).  The
// norm's scale is one factor on the dot products.  Every CTA leaves its best (value, index) as a candidate;
// lm_head_finish_kernel picks the token (largest capped logit, lowest index among equals) and advances the
// position.  C = 256 * NC: a lane owns eight values of every 256, whose activations it keeps in registers (read from shared
// memory for every row they took twice the shared-memory cycles of the row itself).  32000 rows, three tables in turn, head and
// finish, with four slots and activations in shared memory -> now (us): C = 1024 22.4 -> 17.9, 2048 33.8 -> 27.1, 2560 38.4 -> 32.6
// (5.0 TB/s); in the step of a small model 32.5 -> 17.
constexpr int kHeadWarps = 10;
constexpr int kHeadThreads = kHeadWarps * 32;
constexpr int kHeadMaxCtas = 1024;
constexpr int kHeadMaxNC = 12;                               // C <= 3072
constexpr size_t kHeadSmemBudget = 216 * 1024;               // activations + the warps' rings
constexpr int kHeadMaxSlots = 10;                            // rows of one warp's ring

__device__ __forceinline__ void head_cp_async16(void* dst, const void* src) {   // 16 bytes global -> shared, past L1
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// All but the newest `n` requests have landed.
__device__ __forceinline__ void head_wait(int n) {
  switch (n) {
    case 1: asm volatile("cp.async.wait_group 1;" ::: "memory"); break;
    case 2: asm volatile("cp.async.wait_group 2;" ::: "memory"); break;
    case 3: asm volatile("cp.async.wait_group 3;" ::: "memory"); break;
    case 4: asm volatile("cp.async.wait_group 4;" ::: "memory"); break;
    case 5: asm volatile("cp.async.wait_group 5;" ::: "memory"); break;
    case 6: asm volatile("cp.async.wait_group 6;" ::: "memory"); break;
    case 7: asm volatile("cp.async.wait_group 7;" ::: "memory"); break;
    case 8: asm volatile("cp.async.wait_group 8;" ::: "memory"); break;
    default: asm volatile("cp.async.wait_group 9;" ::: "memory"); break;
  }
}

template <int NC>
__global__ void __launch_bounds__(kHeadThreads, 1) lm_head_kernel(const float* __restrict__ x, const float* __restrict__ delta,
                                                                  const float* __restrict__ w, float eps,
                                                                  const __nv_bfloat16* __restrict__ table, int V, int slots,
                                                                  float cap, float* __restrict__ logits_out,
                                                                  float* __restrict__ cand_val, int* __restrict__ cand_idx) {
  extern __shared__ __align__(16) uint8_t head_smem[];
  __shared__ float s_red[kHeadWarps];
  __shared__ int s_ci[kHeadWarps];
  __shared__ float s_scale;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int C = NC * 256, row_bytes = C * 2;
  float* hs = reinterpret_cast<float*>(head_smem);                                   // C floats
  uint8_t* ring = head_smem + (size_t)C * 4 + (size_t)warp * slots * row_bytes;     // [slots][row_bytes]
  const int G = gridDim.x, b = blockIdx.x;
  const int row0 = (int)((long long)V * b / G), row1 = (int)((long long)V * (b + 1) / G);
  // row i of this warp: row0 + warp + 10 i, copied into ring slot i % slots
  int rq = 0, rq_slot = 0;
  auto request = [&]() {
    const int r = row0 + warp + kHeadWarps * rq;
    if (r < row1) {
      const uint8_t* src = reinterpret_cast<const uint8_t*>(table) + (size_t)r * row_bytes;
      uint8_t* dst = ring + (size_t)rq_slot * row_bytes;
#pragma unroll
      for (int j = 0; j < NC; ++j) head_cp_async16(dst + (j * 32 + lane) * 16, src + (j * 32 + lane) * 16);
    }
    ++rq;
    if (++rq_slot == slots) rq_slot = 0;
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  asm volatile("griddepcontrol.launch_dependents;");
  for (int i = 0; i < slots - 1; ++i) request();             // the table does not depend on the launch before
  asm volatile("griddepcontrol.wait;" ::: "memory");
  float ss = 0.f;
  for (int i4 = tid; i4 < C / 4; i4 += kHeadThreads) {
    float4 v = __ldcg(reinterpret_cast<const float4*>(x) + i4);
    if (delta) {
      const float4 d = __ldcg(reinterpret_cast<const float4*>(delta) + i4);
      v.x += d.x; v.y += d.y; v.z += d.z; v.w += d.w;
    }
    ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
    if (w) {
      const float4 g = __ldg(reinterpret_cast<const float4*>(w) + i4);
      v.x *= g.x; v.y *= g.y; v.z *= g.z; v.w *= g.w;
    }
    reinterpret_cast<float4*>(hs)[i4] = v;
  }
  ss = warp_sum(ss);
  if (lane == 0) s_red[warp] = ss;
  __syncthreads();
  if (tid == 0) {
    float tot = 0.f;
    for (int i = 0; i < kHeadWarps; ++i) tot += s_red[i];
    s_scale = w ? 1.0f / sqrtf(tot / (float)C + eps) : 1.0f;
  }
  __syncthreads();
  const float scale = s_scale;
  float4 xr[2 * NC];                                         // this lane's eight values of every 256
#pragma unroll
  for (int j = 0; j < NC; ++j) {
    xr[2 * j] = *reinterpret_cast<const float4*>(hs + (j * 32 + lane) * 8);
    xr[2 * j + 1] = *reinterpret_cast<const float4*>(hs + (j * 32 + lane) * 8 + 4);
  }
  float best = -FLT_MAX;
  int best_i = 0x7fffffff;
  int use_slot = 0;
#pragma unroll 1
  for (int r = row0 + warp; r < row1; r += kHeadWarps) {
    request();                                               // (past the end: an empty group)
    head_wait(slots - 1);
    __syncwarp();
    const uint8_t* pr = ring + (size_t)use_slot * row_bytes;
    float acc = 0.f;
#pragma unroll
    for (int j = 0; j < NC; ++j) {
      const float4 x0 = xr[2 * j], x1 = xr[2 * j + 1];
      const uint4 t = *reinterpret_cast<const uint4*>(pr + (j * 32 + lane) * 16);
      // a word holds elements 2e (low half) and 2e + 1
      acc += __uint_as_float(t.x << 16) * x0.x + __uint_as_float(t.x & 0xffff0000u) * x0.y;
      acc += __uint_as_float(t.y << 16) * x0.z + __uint_as_float(t.y & 0xffff0000u) * x0.w;
      acc += __uint_as_float(t.z << 16) * x1.x + __uint_as_float(t.z & 0xffff0000u) * x1.y;
      acc += __uint_as_float(t.w << 16) * x1.z + __uint_as_float(t.w & 0xffff0000u) * x1.w;
    }
    if (++use_slot == slots) use_slot = 0;
    __syncwarp();                                            // every lane is done with this slot before it is requested again
    acc = warp_sum(acc);
    if (lane == 0) {
      const float y = cap * tanhf(acc * scale / cap);
      logits_out[r] = y;
      if (y > best || (y == best && r < best_i)) { best = y; best_i = r; }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();                                           // s_red is reused
  if (lane == 0) { s_red[warp] = best; s_ci[warp] = best_i; }
  __syncthreads();
  if (tid == 0) {
    for (int i = 1; i < kHeadWarps; ++i)
      if (s_red[i] > best || (s_red[i] == best && s_ci[i] < best_i)) { best = s_red[i]; best_i = s_ci[i]; }
    cand_val[b] = best;
    cand_idx[b] = best_i;
  }
}

__global__ void __launch_bounds__(256) lm_head_finish_kernel(const float* __restrict__ cand_val, const int* __restrict__ cand_idx, int G,
                                                             long long* __restrict__ token, long long* __restrict__ pos) {
  __shared__ float s_val[8];
  __shared__ int s_idx[8];
  pdl_enter();
  const int tid = threadIdx.x;
  float best = -FLT_MAX;
  int best_i = 0x7fffffff;
  for (int i = tid; i < G; i += 256) {
    const float v = cand_val[i];
    const int vi = cand_idx[i];
    if (v > best || (v == best && vi < best_i)) { best = v; best_i = vi; }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
    if (ov > best || (ov == best && oi < best_i)) { best = ov; best_i = oi; }
  }
  if ((tid & 31) == 0) { s_val[tid >> 5] = best; s_idx[tid >> 5] = best_i; }
  __syncthreads();
  if (tid == 0) {
    for (int i = 1; i < 8; ++i)
      if (s_val[i] > best || (s_val[i] == best && s_idx[i] < best_i)) { best = s_val[i]; best_i = s_idx[i]; }
    token[0] = best_i == 0x7fffffff ? 0 : best_i;
    if (pos) *pos += 1;
  }
}


// h[b, i] = silu(gu[b, i]) * gu[b, F + i]
__global__ void silu_mul_kernel(const float* __restrict__ gu, float* __restrict__ hmid, int F, int total) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  pdl_enter();
  if (i >= total) return;
  const int b = i / F, c = i - b * F;
  const float g = gu[(size_t)b * 2 * F + c], u = gu[(size_t)b * 2 * F + F + c];
  hmid[i] = g / (1.0f + __expf(-g)) * u;
}

// The same four values at a time, to fp32 or straight to the down projection's operand.  Bound by memory: 28 M values of 4096
// rows 120 us one at a time and 36 us more to split them, now one pass over 12 bytes per value.  CTAs of 256 threads take several
// rows where a row is shorter (4096 rows of 100: 2.6 us, one CTA per row 5.6 us).
template <bool kTerms>
__global__ void __launch_bounds__(256) silu_mul4_kernel(const float4* __restrict__ gu, void* __restrict__ out, int f4, int rows) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x, b = blockIdx.y * blockDim.y + threadIdx.y;
  pdl_enter();
  if (c >= f4 || b >= rows) return;
  const float4 g = __ldcs(gu + (size_t)b * 2 * f4 + c), u = __ldcs(gu + (size_t)b * 2 * f4 + f4 + c);
  const float4 h = make_float4(g.x / (1.0f + __expf(-g.x)) * u.x, g.y / (1.0f + __expf(-g.y)) * u.y, g.z / (1.0f + __expf(-g.z)) * u.z,
                               g.w / (1.0f + __expf(-g.w)) * u.w);
  if (kTerms) store_terms(out, b, f4, c, h);
  else reinterpret_cast<float4*>(out)[(size_t)b * f4 + c] = h;
}

// out[b, :] = float(table[token[b], :]) for a bf16 (V, C) embedding table; one CTA per sequence.
__global__ void embed_rows_kernel(const __nv_bfloat16* __restrict__ table, const long long* __restrict__ token, float* __restrict__ out,
                                  int C, int V) {
  pdl_enter();
  long long t = token[blockIdx.x];
  t = t < 0 ? 0 : (t >= V ? V - 1 : t);
  const __nv_bfloat16* row = table + (size_t)t * C;
  for (int i = threadIdx.x; i < C; i += blockDim.x) out[(size_t)blockIdx.x * C + i] = __bfloat162float(row[i]);
}

// The end of a decode step for one sequence per CTA: logits_out[b, v] = cap * tanh(float(logits[b, v]) / cap),
// token[b] = index of the largest capped logit (the lowest index among equals), and CTA 0 advances the
// position.  logits are bf16 (the LM-head product) or fp32.  Without logits_out: the arg-max of the logits as they are.
constexpr int kFinishThreads = 1024;
__global__ void __launch_bounds__(kFinishThreads) softcap_argmax_kernel(const void* __restrict__ logits, int is_bf16, int V, float cap,
                                                                        float* __restrict__ logits_out, long long* __restrict__ token,
                                                                        long long* __restrict__ pos) {
  __shared__ float s_val[kFinishThreads / 32];
  __shared__ int s_idx[kFinishThreads / 32];
  pdl_enter();
  const int b = blockIdx.x, tid = threadIdx.x;
  float best = -FLT_MAX;
  int best_i = 0x7fffffff;
  for (int i0 = tid; i0 < V; i0 += 8 * kFinishThreads) {  // eight loads in flight per thread
    float x[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int i = i0 + j * kFinishThreads;
      x[j] = 0.f;
      if (i < V)
        x[j] = is_bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(logits)[(size_t)b * V + i])
                       : reinterpret_cast<const float*>(logits)[(size_t)b * V + i];
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int i = i0 + j * kFinishThreads;
      if (i < V) {
        const float y = logits_out ? cap * tanhf(x[j] / cap) : x[j];
        if (logits_out) logits_out[(size_t)b * V + i] = y;
        if (y > best || (y == best && i < best_i)) { best = y; best_i = i; }   // NaN never wins, as in a max-reduction that skips it
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
    if (ov > best || (ov == best && oi < best_i)) { best = ov; best_i = oi; }
  }
  if ((tid & 31) == 0) { s_val[tid >> 5] = best; s_idx[tid >> 5] = best_i; }
  __syncthreads();
  if (tid < 32) {
    best = s_val[tid]; best_i = s_idx[tid];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
      if (ov > best || (ov == best && oi < best_i)) { best = ov; best_i = oi; }
    }
    if (tid == 0) {
      token[b] = best_i == 0x7fffffff ? 0 : best_i;
      if (b == 0 && pos) *pos += 1;
    }
  }
}

}  // namespace nb

using namespace nb;

extern "C" int nb_embed_rows(const void* table_bf16, const int64_t* token, int B, int V, int C, float* out, void* stream) {
  if (!table_bf16 || !token || !out || B < 1 || V < 1 || C < 1) return NB_ERR_ARG;
  if (int rc = check_device()) return rc;
  return launch_pdl(embed_rows_kernel, dim3(B), dim3(1024), 0, (cudaStream_t)stream, reinterpret_cast<const __nv_bfloat16*>(table_bf16),
                    reinterpret_cast<const long long*>(token), out, C, V);
}

extern "C" int nb_softcap_argmax(const void* logits, int logits_dtype, int B, int V, float cap, float* logits_out, int64_t* token,
                                 int64_t* pos, void* stream) {
  if (!logits || !logits_out || !token || B < 1 || V < 1 || !(cap > 0.f)) return NB_ERR_ARG;
  if (logits_dtype != NB_BF16 && logits_dtype != NB_F32) return NB_ERR_ARG;
  if (int rc = check_device()) return rc;
  return launch_pdl(softcap_argmax_kernel, dim3(B), dim3(kFinishThreads), 0, (cudaStream_t)stream, logits,
                    logits_dtype == NB_BF16 ? 1 : 0, V, cap, logits_out, reinterpret_cast<long long*>(token),
                    reinterpret_cast<long long*>(pos));
}

extern "C" int nb_argmax(const float* logits, int B, int V, int64_t* token, int64_t* pos, void* stream) {
  if (!logits || !token || B < 1 || V < 1) return NB_ERR_ARG;
  if (int rc = check_device()) return rc;
  return launch_pdl(softcap_argmax_kernel, dim3(B), dim3(kFinishThreads), 0, (cudaStream_t)stream, (const void*)logits, 0, V, 1.0f,
                    (float*)nullptr, reinterpret_cast<long long*>(token), reinterpret_cast<long long*>(pos));
}

extern "C" int nb_add_rmsnorm(float* x, const float* delta, const float* w, float eps, float* out, int B, int C, void* stream) {
  if (!x || !w || !out || B < 1 || C < 1) return NB_ERR_ARG;
  if (C > 16 * 256) return NB_ERR_SHAPE;
  if (int rc = check_device()) return rc;
  return launch_pdl(add_rmsnorm_kernel, dim3(B), dim3(256), 0, (cudaStream_t)stream, x, delta, w, eps, out, C);
}

extern "C" int nb_rope_kv_write(const float* qkv, int B, int H, int hd, const float* cos2, const float* sin2, const int64_t* pos,
                                float* k_cache, float* v_cache, int ctx, float* q_out, void* stream) {
  if (!qkv || !cos2 || !sin2 || !pos || !k_cache || !v_cache || !q_out || B < 1 || H < 1 || hd < 2 || (hd & 1) || ctx < 1)
    return NB_ERR_ARG;
  if (int rc = check_device()) return rc;
  return launch_pdl(rope_kv_kernel, dim3(H, B), dim3(128), 0, (cudaStream_t)stream, qkv, cos2, sin2,
                    reinterpret_cast<const long long*>(pos), k_cache, v_cache, q_out, H, hd, ctx);
}

extern "C" int nb_decode_attention_rope(const float* qkv, const float* cos2, const float* sin2, const int64_t* pos, float* k_cache,
                                        float* v_cache, int B, int H, int hd, int ctx, float* out, int out_stride, int out_offset,
                                        void* stream) {
  if (!qkv || !cos2 || !sin2 || !k_cache || !v_cache || !pos || !out || B < 1 || H < 1 || hd < 2 || (hd & 1) || ctx < 1)
    return NB_ERR_ARG;
  if (hd > 128 || hd % 4 != 0) return NB_ERR_SHAPE;
  if ((uintptr_t)k_cache % 16 || (uintptr_t)v_cache % 16) return NB_ERR_ALIGN;
  if (int rc = check_device()) return rc;
  return launch_attention<false>(B, H, hd, ctx, (cudaStream_t)stream, (const float*)nullptr, k_cache, v_cache,
                                 reinterpret_cast<const long long*>(pos), out, H, hd, ctx, out_stride, out_offset, qkv, cos2, sin2);
}

extern "C" int nb_decode_attention_terms(const float* qkv, const float* cos2, const float* sin2, const int64_t* pos, float* k_cache,
                                         float* v_cache, int B, int H, int hd, int ctx, void* terms, int out_cols, int out_offset,
                                         void* stream) {
  if (!qkv || !cos2 || !sin2 || !k_cache || !v_cache || !pos || !terms || B < 1 || H < 1 || hd < 2 || (hd & 1) || ctx < 1 || out_offset < 0)
    return NB_ERR_ARG;
  if (hd > 128 || hd % 4 != 0 || out_cols % kBlock || out_offset + H * hd > out_cols) return NB_ERR_SHAPE;
  if ((uintptr_t)k_cache % 16 || (uintptr_t)v_cache % 16 || (uintptr_t)terms % 16) return NB_ERR_ALIGN;
  if (int rc = check_device()) return rc;
  return launch_attention<true>(B, H, hd, ctx, (cudaStream_t)stream, (const float*)nullptr, k_cache, v_cache,
                                reinterpret_cast<const long long*>(pos), reinterpret_cast<float*>(terms), H, hd, ctx, out_cols, out_offset,
                                qkv, cos2, sin2);
}

extern "C" int nb_decode_attention(const float* q, const float* k_cache, const float* v_cache, const int64_t* pos, int B, int H,
                                   int hd, int ctx, float* out, int out_stride, int out_offset, void* stream) {
  if (!q || !k_cache || !v_cache || !pos || !out || B < 1 || H < 1 || hd < 1 || ctx < 1) return NB_ERR_ARG;
  if (hd > 128 || hd % 4 != 0) return NB_ERR_SHAPE;
  if ((uintptr_t)k_cache % 16 || (uintptr_t)v_cache % 16) return NB_ERR_ALIGN;
  if (int rc = check_device()) return rc;
  return launch_attention<false>(B, H, hd, ctx, (cudaStream_t)stream, q, const_cast<float*>(k_cache), const_cast<float*>(v_cache),
                                 reinterpret_cast<const long long*>(pos), out, H, hd, ctx, out_stride, out_offset, (const float*)nullptr,
                                 (const float*)nullptr, (const float*)nullptr);
}

extern "C" int nb_prefill_attention(const float* qkv, int B, int T, int H, int hd, const float* cos2, const float* sin2, int pos0,
                                    float* k_cache, float* v_cache, int ctx, float* out, int out_stride, int out_offset,
                                    void* stream) {
  if (!qkv || !cos2 || !sin2 || !k_cache || !v_cache || !out || B < 1 || T < 1 || H < 1 || hd < 4 || ctx < 1 || pos0 < 0 ||
      out_stride < 1 || out_offset < 0)
    return NB_ERR_ARG;
  if (hd > 128 || hd % 4 != 0 || pos0 + T > ctx || out_offset + H * hd > out_stride) return NB_ERR_SHAPE;
  if ((uintptr_t)qkv % 16 || (uintptr_t)k_cache % 16 || (uintptr_t)v_cache % 16 || (uintptr_t)out % 16 || out_stride % 4 ||
      out_offset % 4)
    return NB_ERR_ALIGN;
  if (H > 65535 || B > 65535) return NB_ERR_SHAPE;
  if (int rc = check_device()) return rc;
  const float scale = 1.0f / sqrtf((float)hd);
  prompt_keys_kernel<<<dim3(T, B), 256, 0, (cudaStream_t)stream>>>(qkv, cos2, sin2, k_cache, v_cache, T, H, hd, ctx, pos0);
  if (int rc = check_launch()) return rc;
  auto run = [&](auto pairs) {
    return prefill_attention_tile<decltype(pairs)::value>(B, T, H, hd, pos0, (cudaStream_t)stream, qkv, cos2, sin2, (const float*)k_cache,
                                                          (const float*)v_cache, out, T, H, hd, ctx, pos0, out_stride, out_offset, scale);
  };
  switch (prompt_pairs(hd)) {
    case 2: return run(std::integral_constant<int, 2>{});
    case 4: return run(std::integral_constant<int, 4>{});
    case 5: return run(std::integral_constant<int, 5>{});
    default: return run(std::integral_constant<int, 8>{});
  }
}

extern "C" size_t nb_lm_head_scratch_bytes(void) { return (size_t)kHeadMaxCtas * 8; }

template <int NC>
static int launch_head(const float* x, const float* delta, const float* w, float eps, const __nv_bfloat16* table, int V, float cap,
                       float* logits_out, float* cv, int* ci, int G, cudaStream_t st) {
  // ring slots per warp: as many rows in flight as the shared memory holds, which for narrow rows are many (C = 1024: ten slots
  // instead of four)
  constexpr size_t act = (size_t)NC * 256 * 4, row = (size_t)kHeadWarps * NC * 256 * 2;
  constexpr int slots = (kHeadSmemBudget - act) / row < kHeadMaxSlots ? (int)((kHeadSmemBudget - act) / row) : kHeadMaxSlots;
  static_assert(slots >= 2, "a row in flight while one is multiplied");
  static bool done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!done[dev & 63]) {
    if (cudaError_t e = cudaFuncSetAttribute(lm_head_kernel<NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kHeadSmemBudget)) return record_cuda_error(e);
    done[dev & 63] = true;
  }
  return launch_pdl(lm_head_kernel<NC>, dim3(G), dim3(kHeadThreads), act + slots * row, st, x, delta, w, eps, table, V, slots, cap, logits_out, cv, ci);
}

extern "C" int nb_lm_head(const float* x, const float* delta, const float* norm_weight, float eps, const void* table_bf16, int V, int C,
                          float cap, float* logits_out, int64_t* token, int64_t* pos, void* scratch, void* stream) {
  if (!x || !table_bf16 || !logits_out || !token || !scratch || V < 1 || C < 1 || !(cap > 0.f)) return NB_ERR_ARG;
  if (C % 256 != 0 || C / 256 > kHeadMaxNC) return NB_ERR_SHAPE;
  if ((uintptr_t)x % 16 || (uintptr_t)delta % 16 || (uintptr_t)norm_weight % 16 || (uintptr_t)table_bf16 % 16 || (uintptr_t)scratch % 16)
    return NB_ERR_ALIGN;
  if (int rc = check_device()) return rc;
  const int G = std::min(std::min(sm_count(), kHeadMaxCtas), V);
  float* cv = reinterpret_cast<float*>(scratch);
  int* ci = reinterpret_cast<int*>(cv + kHeadMaxCtas);
  cudaStream_t st = (cudaStream_t)stream;
  int rc = NB_OK;
  const auto launch = [&](auto nc) { rc = launch_head<decltype(nc)::value>(x, delta, norm_weight, eps, reinterpret_cast<const __nv_bfloat16*>(table_bf16), V, cap, logits_out, cv, ci, G, st); };
  switch (C / 256) {
    case 1: launch(std::integral_constant<int, 1>{}); break;
    case 2: launch(std::integral_constant<int, 2>{}); break;
    case 3: launch(std::integral_constant<int, 3>{}); break;
    case 4: launch(std::integral_constant<int, 4>{}); break;
    case 5: launch(std::integral_constant<int, 5>{}); break;
    case 6: launch(std::integral_constant<int, 6>{}); break;
    case 7: launch(std::integral_constant<int, 7>{}); break;
    case 8: launch(std::integral_constant<int, 8>{}); break;
    case 9: launch(std::integral_constant<int, 9>{}); break;
    case 10: launch(std::integral_constant<int, 10>{}); break;
    case 11: launch(std::integral_constant<int, 11>{}); break;
    default: launch(std::integral_constant<int, 12>{}); break;
  }
  if (rc) return rc;
  return launch_pdl(lm_head_finish_kernel, dim3(1), dim3(256), 0, st, (const float*)cv, (const int*)ci, G,
                    reinterpret_cast<long long*>(token), reinterpret_cast<long long*>(pos));
}

template <bool kTerms>
static int launch_silu4(const float* gu, int B, int F, void* out, cudaStream_t st) {
  const int f4 = F / 4, tx = std::min(256, (f4 + 31) / 32 * 32), ty = 256 / tx;
  return launch_pdl(silu_mul4_kernel<kTerms>, dim3((f4 + tx - 1) / tx, (B + ty - 1) / ty), dim3(tx, ty), 0, st, reinterpret_cast<const float4*>(gu),
                    out, f4, B);
}

extern "C" int nb_silu_mul(const float* gu, int B, int F, float* hmid, void* stream) {
  if (!gu || !hmid || B < 1 || F < 1) return NB_ERR_ARG;
  if (int rc = check_device()) return rc;
  // four values per thread where that still gives every SM a CTA: below it the four quotients of a thread take longer than four
  // threads (17 rows of 6912: 2.3 against 2.0 us)
  if (F % 4 == 0 && (uintptr_t)gu % 16 == 0 && (uintptr_t)hmid % 16 == 0 && B <= 65535 && (long long)B * (F / 4) >= 256ll * sm_count())
    return launch_silu4<false>(gu, B, F, hmid, (cudaStream_t)stream);
  const int total = B * F;
  return launch_pdl(silu_mul_kernel, dim3((total + 255) / 256), dim3(256), 0, (cudaStream_t)stream, gu, hmid, F, total);
}

extern "C" int nb_silu_mul_terms(const float* gu, int B, int F, void* terms, void* stream) {
  if (!gu || !terms || B < 1 || F < 1) return NB_ERR_ARG;
  if (F % 4 || B > 65535) return NB_ERR_SHAPE;
  if ((uintptr_t)gu % 16 || (uintptr_t)terms % 16) return NB_ERR_ALIGN;
  if (int rc = check_device()) return rc;
  return launch_silu4<true>(gu, B, F, terms, (cudaStream_t)stream);
}

extern "C" int nb_add_rmsnorm_terms(float* x, const float* delta, const float* w, float eps, void* terms, int B, int C, void* stream) {
  if (!x || !w || !terms || B < 1 || C < 1) return NB_ERR_ARG;
  if (C % 4 || C > 16 * 256) return NB_ERR_SHAPE;
  if ((uintptr_t)x % 16 || (uintptr_t)delta % 16 || (uintptr_t)w % 16 || (uintptr_t)terms % 16) return NB_ERR_ALIGN;
  if (int rc = check_device()) return rc;
  return launch_pdl(add_rmsnorm_terms_kernel, dim3(B), dim3(256), 0, (cudaStream_t)stream, reinterpret_cast<float4*>(x),
                    reinterpret_cast<const float4*>(delta), reinterpret_cast<const float4*>(w), eps, terms, C / 4);
}
