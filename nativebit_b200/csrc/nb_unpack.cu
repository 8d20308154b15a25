// Bit-unpack, bit-pack and whole-weight dequantisation kernels (integer / gather work, HBM bound).
//
// All three treat the packed buffer as one LSB-first bit stream: index i occupies bits
// [i*bits, (i+1)*bits).  That is what the reference's three packers produce
// (nativebit/pack.py:21-41, 75-82, 97-116).
#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <type_traits>
#include <cuda_bf16.h>

#include "nb_common.cuh"
#include "nb_device.cuh"
#include "nb_host.h"

namespace nb {

__device__ __forceinline__ uint32_t stream_index(const uint8_t* __restrict__ p, int64_t n_bytes, int64_t i, int bits) {
  const int64_t bit = i * bits;
  const int64_t byte = bit >> 3;
  uint32_t v = p[byte];
  if (((int)(bit & 7) + bits > 8) && byte + 1 < n_bytes) v |= (uint32_t)p[byte + 1] << 8;
  return (v >> (bit & 7)) & ((1u << bits) - 1u);
}

__host__ __device__ inline int64_t packed_bytes(int64_t count, int bits) {
  return bits == 3 ? 3 * ((count + 7) / 8) : (count * bits + 7) / 8;
}

// Quotient of a place by a block's size: a shift for powers of two (`shift` >= 0), else in 32 bits where they hold the place.
__device__ __forceinline__ int64_t block_of(int64_t i, int size, int shift) {
  return shift >= 0 ? i >> shift : i <= 0xFFFFFFFFll ? (int64_t)((uint32_t)i / (uint32_t)size) : i / size;
}
static int shift_of(int size) { return (size & (size - 1)) ? -1 : __builtin_ctz(size); }

// ---- unpack -------------------------------------------------------------------------------
// Fast path: one thread turns `BITS` aligned 32-bit words into 32 indices (two 16-byte stores).
template <int BITS>
__global__ void unpack32_kernel(const uint32_t* __restrict__ packed, int64_t n_chunks, uint4* __restrict__ out) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n_chunks) return;
  uint32_t w[BITS];
#pragma unroll
  for (int i = 0; i < BITS; ++i) w[i] = packed[c * BITS + i];
  uint32_t o[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    uint32_t v = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int bit = (4 * r + j) * BITS;
      const int wi = bit >> 5, sh = bit & 31;
      uint32_t f = w[wi] >> sh;
      if (sh + BITS > 32 && wi + 1 < BITS) f |= w[wi + 1] << (32 - sh);
      v |= (f & ((1u << BITS) - 1u)) << (8 * j);
    }
    o[r] = v;
  }
  out[2 * c] = make_uint4(o[0], o[1], o[2], o[3]);
  out[2 * c + 1] = make_uint4(o[4], o[5], o[6], o[7]);
}

__global__ void unpack_generic_kernel(const uint8_t* __restrict__ packed, int64_t n_bytes, int bits, int64_t first,
                                      int64_t count, uint8_t* __restrict__ out) {
  const int64_t i = first + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  out[i] = (uint8_t)stream_index(packed, n_bytes, i, bits);
}

// ---- pack ---------------------------------------------------------------------------------
// Output byte b: the (at most 5) indices that overlap it.
__device__ __forceinline__ uint8_t pack_byte(const uint8_t* __restrict__ idx, int64_t count, int bits, int64_t b) {
  const int64_t lo_bit = b * 8, hi_bit = lo_bit + 8;
  const uint32_t mask = (1u << bits) - 1u;
  uint32_t v = 0;
  for (int64_t i = lo_bit / bits; i * bits < hi_bit; ++i) {
    const uint32_t f = (i < count) ? (idx[i] & mask) : 0u;
    const int64_t sh = i * bits - lo_bit;
    v |= sh >= 0 ? (f << sh) : (f >> (-sh));
  }
  return (uint8_t)v;
}

// Fast path, the inverse of unpack32_kernel: one thread turns 32 indices (two 16-byte loads) into `BITS` words.  HBM-bound:
// 17.7 M indices to 3 bits in 6.7 us (24.3 MB); one thread per output byte took 40 us, on 64-bit index arithmetic.
template <int BITS>
__global__ void pack32_kernel(const uint4* __restrict__ idx, int64_t count, int64_t n_bytes, uint32_t* __restrict__ out) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, n_chunks = count >> 5;
  if (c >= n_chunks) {                                 // the bytes of the last, partial chunk (at most 16)
    const int64_t b = n_chunks * (4 * BITS) + (c - n_chunks);
    if (b < n_bytes) reinterpret_cast<uint8_t*>(out)[b] = pack_byte(reinterpret_cast<const uint8_t*>(idx), count, BITS, b);
    return;
  }
  const uint4 a = idx[2 * c], b = idx[2 * c + 1];
  const uint32_t in[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  uint32_t w[BITS];
#pragma unroll
  for (int i = 0; i < BITS; ++i) w[i] = 0;
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    const uint32_t f = (in[j >> 2] >> (8 * (j & 3))) & ((1u << BITS) - 1u);
    const int wi = (j * BITS) >> 5, sh = (j * BITS) & 31;
    w[wi] |= f << sh;
    if (sh + BITS > 32 && wi + 1 < BITS) w[wi + 1] |= f >> (32 - sh);
  }
#pragma unroll
  for (int i = 0; i < BITS; ++i) out[c * BITS + i] = w[i];
}

// Unaligned buffers and less than a chunk: one thread writes one output byte.
__global__ void pack_kernel(const uint8_t* __restrict__ idx, int64_t count, int bits, int64_t n_bytes, uint8_t* __restrict__ out) {
  const int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (b < n_bytes) out[b] = pack_byte(idx, count, bits, b);
}

// ---- dequant ------------------------------------------------------------------------------
// Fast path (fp16 codebook, block_size % 8 == 0, aligned): a thread dequantises the eight consecutive weights of ONE store of 16
// bytes, 32 for fp32 (four per thread there built every table twice: 6912 x 2560 at 3 bits 19.5 -> 14.5 us, 5.5 TB/s), so that a warp's stores are one contiguous run (a thread with 32 weights of its own left every store 64 or 128
// bytes from its neighbour's: 12.1 us for 6912 x 2560 to fp16 and 34.7 us to fp32, which take 6.7 and 12.2 us at the copy
// rate).  The 3- or 2-bit fields are spread to the nibbles of one selector word; the block's table, as byte planes, answers
// four lookups with two byte permutes.  A thread takes PER stores a block stride apart and requests all inputs first: four where
// that leaves every SM four CTAs (6912 x 2560 over six block sizes, three widths and three types 1237 us in sum, 1305 with one),
// else one, as small matrices wait for one thread's chain of loads and not for memory (1024 x 1024 211 -> 183 us in sum).
constexpr int kDqRuns = 4, kDqThreads = 256;

template <int BITS> __device__ __forceinline__ uint32_t load_selectors(const uint32_t* __restrict__ packed, int64_t c) {
  if (BITS == 4) return packed[c];
  if (BITS == 2) {
    uint32_t v = reinterpret_cast<const uint16_t*>(packed)[c];
    v = (v | (v << 8)) & 0x00FF00FFu;
    v = (v | (v << 4)) & 0x0F0F0F0Fu;
    return (v | (v << 2)) & 0x33333333u;
  }
  const int64_t bit = c * 24, wi = bit >> 5;
  const int sh = (int)(bit & 31);                      // 0, 8, 16 or 24
  const uint32_t lo = packed[wi], hi = sh > 8 ? packed[wi + 1] : 0u;
  uint32_t v = __funnelshift_r(lo, hi, sh) & 0xFFFFFFu;
  v = (v & 0xFFFu) | ((v & 0xFFF000u) << 4);           // twelve bits per half word
  v = (v & 0x003F003Fu) | ((v & 0x0FC00FC0u) << 2);    // six per byte
  return (v & 0x07070707u) | ((v & 0x38383838u) << 1); // three per nibble
}

// Eight lookups as one store of 16 bytes, 32 for fp32.
template <int BITS> __device__ __forceinline__ void store8(__half* dst, uint32_t sel, const uint32_t (&T)[BITS == 4 ? 8 : 4]) {
  uint32_t h[4];
  lookup4<BITS>(sel, T, h[0], h[1]);
  lookup4<BITS>(sel >> 16, T, h[2], h[3]);
  *reinterpret_cast<uint4*>(dst) = make_uint4(h[0], h[1], h[2], h[3]);
}
template <int BITS> __device__ __forceinline__ void store8(__nv_bfloat16* dst, uint32_t sel, const uint32_t (&T)[BITS == 4 ? 8 : 4]) {
  uint32_t h[4];
  lookup4<BITS>(sel, T, h[0], h[1]);
  lookup4<BITS>(sel >> 16, T, h[2], h[3]);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h[j]));
    const __nv_bfloat162 b = __floats2bfloat162_rn(f.x, f.y);
    h[j] = *reinterpret_cast<const uint32_t*>(&b);
  }
  *reinterpret_cast<uint4*>(dst) = make_uint4(h[0], h[1], h[2], h[3]);
}
template <int BITS> __device__ __forceinline__ void store8(float* dst, uint32_t sel, const uint32_t (&T)[BITS == 4 ? 8 : 4]) {
  uint32_t h[4];
  lookup4<BITS>(sel, T, h[0], h[1]);
  lookup4<BITS>(sel >> 16, T, h[2], h[3]);
  const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&h[0])), b = __half22float2(*reinterpret_cast<const __half2*>(&h[1]));
  const float2 c = __half22float2(*reinterpret_cast<const __half2*>(&h[2])), d = __half22float2(*reinterpret_cast<const __half2*>(&h[3]));
  if ((uintptr_t)dst % 32 == 0) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"l"(dst), "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y), "f"(d.x), "f"(d.y) : "memory");
  } else {
    reinterpret_cast<float4*>(dst)[0] = make_float4(a.x, a.y, b.x, b.y);
    reinterpret_cast<float4*>(dst)[1] = make_float4(c.x, c.y, d.x, d.y);
  }
}

// Sixteen lookups as one store of 32 bytes, where the address allows it.
template <int BITS, typename T16> __device__ __forceinline__ void store_pair(T16* dst, uint32_t sel0, uint32_t sel1, const uint32_t (&T)[BITS == 4 ? 8 : 4]) {
  if ((uintptr_t)dst % 32 != 0) {
    store8<BITS>(dst, sel0, T);
    store8<BITS>(dst + 8, sel1, T);
    return;
  }
  uint32_t h[8];
  lookup4<BITS>(sel0, T, h[0], h[1]);
  lookup4<BITS>(sel0 >> 16, T, h[2], h[3]);
  lookup4<BITS>(sel1, T, h[4], h[5]);
  lookup4<BITS>(sel1 >> 16, T, h[6], h[7]);
  if (std::is_same<T16, __nv_bfloat16>::value) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h[j]));
      const __nv_bfloat162 b = __floats2bfloat162_rn(f.x, f.y);
      h[j] = *reinterpret_cast<const uint32_t*>(&b);
    }
  }
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"l"(dst), "r"(h[0]), "r"(h[1]), "r"(h[2]), "r"(h[3]), "r"(h[4]), "r"(h[5]), "r"(h[6]), "r"(h[7]) : "memory");
}

// W: chunks of eight weights per store (2: 16-bit types in blocks of whole 16 weights, at 3 and 4 bits: 13824 x 2560 to fp16 20.2 -> 16.8
// and 18.7 -> 15.2 us; at 2 bits, whose lookups and loads are few, 12.4 -> 14.4).
template <int BITS, int PER, int W, typename OutT>
__global__ void __launch_bounds__(kDqThreads) dequant16b_kernel(const uint32_t* __restrict__ packed, const __half* __restrict__ codebook,
                                                               int64_t n_stores, int64_t n_bytes, int64_t total, int block_size, int shift,
                                                               OutT* __restrict__ out, bool beside) {
  if (beside) asm volatile("griddepcontrol.launch_dependents;");
  constexpr int kT = BITS == 4 ? 8 : 4;
  const int64_t i0 = (int64_t)blockIdx.x * (kDqThreads * PER) + threadIdx.x;
  uint32_t sel[PER][W], e[PER][kT];
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    const int64_t i = i0 + u * kDqThreads;
#pragma unroll
    for (int q = 0; q < W; ++q) sel[u][q] = 0;
#pragma unroll
    for (int j = 0; j < kT; ++j) e[u][j] = 0;
    if (i < n_stores) {
#pragma unroll
      for (int q = 0; q < W; ++q) sel[u][q] = load_selectors<BITS>(packed, W * i + q);
      const int64_t block = block_of(i, block_size / (8 * W), shift);
      const uint8_t* row = reinterpret_cast<const uint8_t*>(codebook) + block * (2 << BITS);
      if (BITS == 2) {
        const uint2 v = *reinterpret_cast<const uint2*>(row);
        e[u][0] = v.x; e[u][1] = v.y;
      } else {
#pragma unroll
        for (int j = 0; j < kT / 4; ++j) {
          const uint4 v = reinterpret_cast<const uint4*>(row)[j];
          e[u][4 * j] = v.x; e[u][4 * j + 1] = v.y; e[u][4 * j + 2] = v.z; e[u][4 * j + 3] = v.w;
        }
      }
    }
  }
  int64_t i = i0;
#pragma unroll
  for (int u = 0; u < PER; ++u, i += kDqThreads) {
    if (i >= n_stores) break;
    uint32_t T[kT];
    if (BITS == 2) {
      T[0] = prmt(e[u][0], e[u][1], 0x6420); T[2] = prmt(e[u][0], e[u][1], 0x7531);
      T[1] = T[2]; T[3] = T[0];
    } else {
#pragma unroll
      for (int j = 0; j < kT; j += 4) {
        T[j + 0] = prmt(e[u][j], e[u][j + 1], 0x6420); T[j + 1] = prmt(e[u][j + 2], e[u][j + 3], 0x6420);
        T[j + 2] = prmt(e[u][j], e[u][j + 1], 0x7531); T[j + 3] = prmt(e[u][j + 2], e[u][j + 3], 0x7531);
      }
    }
    if constexpr (W == 2) store_pair<BITS>(out + i * 16, sel[u][0], sel[u][1], T);
    else store8<BITS>(out + i * 8, sel[u][0], T);
  }
  // fewer than 32 weights behind the last whole packed word, one for each of the threads without a store
  const int64_t one = n_stores * (8 * W) + (i - n_stores);
  if (i >= n_stores && i < i0 + PER * kDqThreads && one < total) {
    const uint32_t at = stream_index(reinterpret_cast<const uint8_t*>(packed), n_bytes, one, BITS);
    out[one] = (OutT)(float)codebook[block_of(one, block_size, -1) * (1 << BITS) + at];
  }
}

template <typename CbT, typename OutT>
__global__ void dequant_generic_kernel(const uint8_t* __restrict__ packed, int64_t n_bytes, const CbT* __restrict__ codebook,
                                       int bits, int block_size, int64_t total, OutT* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  const uint32_t e = stream_index(packed, n_bytes, i, bits);
  const float v = (float)codebook[(i / block_size) * (1 << bits) + e];
  out[i] = (OutT)v;
}

// ---- quantise: nearest codebook entry per weight (the exporter's argmin) ------------------------
// idx[i] = argmin_e |w[i] - codebook[i / block_size][e]|, first minimum on ties; weights past `total`
// (padding of the last block) count as 0, as in the reference's zero-padded argmin.
template <typename CbT>
__global__ void quantize_kernel(const float* __restrict__ w, int64_t total, int64_t padded, const CbT* __restrict__ codebook,
                                int n_entries, int block_size, uint8_t* __restrict__ idx) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= padded) return;
  const float v = i < total ? w[i] : 0.f;
  const CbT* cb = codebook + (i / block_size) * n_entries;
  float best = fabsf(v - (float)cb[0]);
  int arg = 0;
  for (int e = 1; e < n_entries; ++e) {
    const float d = fabsf(v - (float)cb[e]);
    if (d < best) { best = d; arg = e; }
  }
  idx[i] = (uint8_t)arg;
}

// The same for four consecutive weights per thread (one block's: block_size % 4 == 0); with PACK the indices leave as the packed
// stream, 32 of them gathered by the shuffles of eight lanes.  64-bit index arithmetic and single-byte stores held the general
// kernel at 92 us for 6912 x 2560 weights; what bounds this one is the argmin itself, three operations of the half-rate pipe
// per entry and weight (floor 20 us).  (Four such runs per thread take 1 % longer there and 4.4 instead of 2.6 us for 100 x 100.)
constexpr int kQThreads = 256;
// from this many weights on the search is faster (us, every entry tried | search: 3 bits, 1 M weights 3.3 | 3.5, 2 M 5.1 | 4.5,
// 17.7 M 32.3 | 20.3; 4 bits, 262 k 2.5 | 2.3, 524 k 3.3 | 2.7, 17.7 M 55.5 | 26.9; 2 bits 17.7 M 20.5 | 19.7, below slower)
constexpr int64_t kQSearch3 = 1 << 21, kQSearch4 = 1 << 19;

template <typename CbT, int NE> __device__ __forceinline__ void load_entries(const CbT* cb, float (&c)[NE]);
template <> __device__ __forceinline__ void load_entries<float, 4>(const float* cb, float (&c)[4]) {
  const float4 v = *reinterpret_cast<const float4*>(cb);
  c[0] = v.x; c[1] = v.y; c[2] = v.z; c[3] = v.w;
}
template <> __device__ __forceinline__ void load_entries<float, 8>(const float* cb, float (&c)[8]) {
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const float4 v = reinterpret_cast<const float4*>(cb)[i];
    c[4 * i] = v.x; c[4 * i + 1] = v.y; c[4 * i + 2] = v.z; c[4 * i + 3] = v.w;
  }
}
template <> __device__ __forceinline__ void load_entries<float, 16>(const float* cb, float (&c)[16]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float4 v = reinterpret_cast<const float4*>(cb)[i];
    c[4 * i] = v.x; c[4 * i + 1] = v.y; c[4 * i + 2] = v.z; c[4 * i + 3] = v.w;
  }
}

template <int BITS, bool PACK>
__global__ void __launch_bounds__(kQThreads) quantize4_kernel(const float* __restrict__ w, int64_t total, int64_t padded,
                                                              const float* __restrict__ codebook, int block4, int shift,
                                                              uint32_t* __restrict__ out) {
  constexpr int NE = 1 << BITS;
  const int64_t i = (int64_t)blockIdx.x * kQThreads + threadIdx.x;      // in units of four weights
  const int lane = threadIdx.x & 31;
  const bool in = 4 * i < padded;
  float v[4];
  if (4 * i + 4 <= total) {
    const float4 x = reinterpret_cast<const float4*>(w)[i];
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = 4 * i + j < total ? w[4 * i + j] : 0.f;
  }
  uint32_t arg[4] = {0u, 0u, 0u, 0u};
  if (in) {
    float c[NE];
    load_entries<float, NE>(codebook + block_of(i, block4, shift) * NE, c);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float best = fabsf(v[j] - c[0]);
#pragma unroll
      for (int e = 1; e < NE; ++e) {
        const float d = fabsf(v[j] - c[e]);
        if (d < best) { best = d; arg[j] = e; }
      }
    }
  }
  if (!PACK) {
    if (in) out[i] = arg[0] | (arg[1] << 8) | (arg[2] << 16) | (arg[3] << 24);
  } else {
    // two lanes hold 8 indices = 8 * BITS bits; at 3 bits even lane 2 q < 6 of eight writes word q: bits 32 q .. 32 q + 31 of
    // the four pairs of 24, which lie in its own pair and the next
    const uint32_t f = arg[0] | (arg[1] << BITS) | (arg[2] << (2 * BITS)) | (arg[3] << (3 * BITS));
    const uint32_t pair = f | (__shfl_down_sync(0xffffffffu, f, 1) << (4 * BITS));      // of the even lanes
    const uint32_t next = __shfl_down_sync(0xffffffffu, pair, 2);
    const int q = (lane & 7) >> 1;
    if (!in || (lane & 1)) return;
    uint32_t* dst = out + (i >> 3) * BITS;
    if (BITS == 4) dst[q] = pair;
    else if (BITS == 2) { if (!(q & 1)) dst[q >> 1] = pair | (next << 16); }
    else if (q < 3) dst[q] = __funnelshift_r(pair | (next << 24), next >> 8, 8 * q);
  }
}

// The same with the indices packed, eight weights per thread, for large matrices.  Trying every entry is 48 instructions per weight
// at 3 bits, and issuing them bounds the kernel above.  The exporter's codebooks are in ascending order, and there a binary
// search in shared memory, three instructions a step, finds the entries on either side of a weight, one of which is the nearest.
//   The answer has to be that of the trial of all entries in fp32, first minimum on ties: distances are rounded, so an entry
// further away may round to the same distance as its neighbour and come first.  With entries in order, more than 2^-20 of their
// range apart, and a weight below the last entry by any distance or above it by less than three ranges, the distances to tell
// apart are at most 4 ranges, an ulp of which is at most 2^-21 ranges: entries on one side of the weight are then at different
// distances.  A tie between the two sides goes to the lower one, as there.  Every other block or weight (codebooks
// out of order, with equal, infinite or NaN entries; weights far above, infinite or NaN) is tried entry by entry.
__device__ __forceinline__ float lds_f32(uint32_t at) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
  return v;
}

constexpr int kQRows = kQThreads * 8 / 32 + 1;               // codebooks that a CTA's 2048 weights may meet (blocks of 32 and more)

template <int BITS>
__global__ void __launch_bounds__(kQThreads) quantize8_pack_kernel(const float* __restrict__ w, int64_t total, int64_t padded,
                                                                   const float* __restrict__ codebook, int block8, int shift,
                                                                   uint32_t* __restrict__ out) {
  constexpr int NE = 1 << BITS;
  __shared__ __align__(16) float rows[kQRows][NE + 4];      // the entries, the last one once more
  __shared__ float limits[kQRows];                           // weights below may be searched for
  const int64_t i0 = (int64_t)blockIdx.x * kQThreads, i = i0 + threadIdx.x, units = padded >> 3;      // in units of eight weights
  const bool in = i < units;
  float v[8];
  if (8 * i + 8 <= total) {
    const float4 a = reinterpret_cast<const float4*>(w)[2 * i], b = reinterpret_cast<const float4*>(w)[2 * i + 1];
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = 8 * i + j < total ? w[8 * i + j] : 0.f;
  }
  const int64_t row0 = block_of(i0, block8, shift), last = block_of(min(i0 + kQThreads, units) - 1, block8, shift);
  if ((int)threadIdx.x <= (int)(last - row0)) {
    float c[NE];
    load_entries<float, NE>(codebook + (row0 + threadIdx.x) * NE, c);
    float gap = c[1] - c[0];
    bool plain = c[0] < c[1];
#pragma unroll
    for (int e = 2; e < NE; ++e) {
      gap = fminf(gap, c[e] - c[e - 1]);
      plain = plain && c[e - 1] < c[e];                      // (false for NaN, which fminf drops)
    }
    const float range = c[NE - 1] - c[0];
    limits[threadIdx.x] = plain && gap > range * 0x1p-20f && range < 8e37f ? c[NE - 1] + 3.f * range : -INFINITY;
#pragma unroll
    for (int e = 0; e < NE; e += 4) *reinterpret_cast<float4*>(&rows[threadIdx.x][e]) = make_float4(c[e], c[e + 1], c[e + 2], c[e + 3]);
    rows[threadIdx.x][NE] = c[NE - 1];
  }
  __syncthreads();
  uint32_t f = 0;
  if (in) {
    const int r = (int)(block_of(i, block8, shift) - row0);
    const float *row = rows[r], limit = limits[r];
    bool plain = true;
#pragma unroll
    for (int j = 0; j < 8; ++j) plain = plain && v[j] < limit;
    if (plain) {
      // byte offsets of the entries found, summed at their places and freed of the row's own offset at the end
      const uint32_t base = smem_u32(row);
      constexpr int kGroup = BITS == 4 ? 4 : 8;              // weights whose sums fit 32 bits
#pragma unroll
      for (int h = 0; h < 8 / kGroup; ++h) {
        uint32_t sum = 0, ones = 0;
#pragma unroll
        for (int q = 0; q < kGroup; ++q) {
          const float x = v[h * kGroup + q];
          uint32_t p = base;
#pragma unroll
          for (int half = NE / 2; half > 0; half >>= 1)
            if (x >= lds_f32(p + 4 * half)) p += 4 * half;
          if (fabsf(x - lds_f32(p + 4)) < fabsf(x - lds_f32(p))) p += 4;
          sum += p << (BITS * q);
          ones += 1u << (BITS * q);
        }
        f |= ((sum - base * ones) >> 2) << (16 * h);
      }
    } else {
#pragma unroll 1
      for (int j = 0; j < 8; ++j) {
        float x = v[0];
#pragma unroll
        for (int q = 1; q < 8; ++q) x = q == j ? v[q] : x;
        float best = fabsf(x - row[0]);
        uint32_t arg = 0;
#pragma unroll
        for (int e = 1; e < NE; ++e) {
          const float d = fabsf(x - row[e]);
          if (d < best) { best = d; arg = e; }
        }
        f |= arg << (BITS * j);
      }
    }
  }
  if (BITS == 4) {
    if (in) out[i] = f;
  } else {                                                               // four lanes hold 96 bits
    const uint32_t next = __shfl_down_sync(0xffffffffu, f, 1);
    const int q = threadIdx.x & 3;
    if (in && q < 3) out[(i >> 2) * 3 + q] = (f >> (8 * q)) | (next << (24 - 8 * q));
  }
}

// Whether the four-wide kernels take these arguments: fp32 entries (the exporter's), 2 to 4 bits, four weights per load
// and four indices per store (a packed word holds 32 indices of whole blocks).
static bool quantize4_fits(const float* w, const void* codebook, int cb_dtype, int n_entries, int block_size, const void* out, bool pack) {
  return cb_dtype == NB_F32 && (n_entries == 4 || n_entries == 8 || n_entries == 16) && block_size % (pack ? 32 : 4) == 0 && (uintptr_t)w % 16 == 0 &&
         (uintptr_t)codebook % 16 == 0 && (uintptr_t)out % 4 == 0;
}

template <bool PACK>
static int launch_quantize4(const float* w, int64_t total, int64_t padded, const float* codebook, int n_entries, int block_size, void* out,
                            cudaStream_t st) {
  if (PACK && ((n_entries == 8 && padded >= kQSearch3) || (n_entries == 16 && padded >= kQSearch4))) {
    const int block8 = block_size / 8, shift8 = shift_of(block8);
    const unsigned g = (unsigned)((padded / 8 + kQThreads - 1) / kQThreads);
    uint32_t* o8 = (uint32_t*)out;
    if (n_entries == 8) quantize8_pack_kernel<3><<<g, kQThreads, 0, st>>>(w, total, padded, codebook, block8, shift8, o8);
    else quantize8_pack_kernel<4><<<g, kQThreads, 0, st>>>(w, total, padded, codebook, block8, shift8, o8);
    return check_launch();
  }
  const int block4 = block_size / 4, shift = shift_of(block4);
  const unsigned grid = (unsigned)((padded / 4 + kQThreads - 1) / kQThreads);
  uint32_t* o = (uint32_t*)out;
  if (n_entries == 4) quantize4_kernel<2, PACK><<<grid, kQThreads, 0, st>>>(w, total, padded, codebook, block4, shift, o);
  else if (n_entries == 8) quantize4_kernel<3, PACK><<<grid, kQThreads, 0, st>>>(w, total, padded, codebook, block4, shift, o);
  else quantize4_kernel<4, PACK><<<grid, kQThreads, 0, st>>>(w, total, padded, codebook, block4, shift, o);
  return check_launch();
}

// beside: the launch behind may start before this one ends.  Only for a caller that knows that launch (dequant_beside): one that
// reads the dequantised matrix ahead of its dependency wait, as the LM head reads its table, must not.
template <typename OutT>
static int dequant_dispatch(const uint8_t* packed, const void* codebook, int cb_dtype, int bits, int block_size,
                            int64_t total, OutT* out, bool beside, cudaStream_t st) {
  const int64_t n_blocks = (total + block_size - 1) / block_size;
  const int64_t n_bytes = packed_bytes(n_blocks * block_size, bits);
  const bool aligned = ((uintptr_t)packed % 4 == 0) && ((uintptr_t)out % 16 == 0) && ((uintptr_t)codebook % 16 == 0);
  if (cb_dtype == NB_F16 && block_size % 8 == 0 && aligned) {
    const auto start = [&](auto width) {
      constexpr int W = decltype(width)::value;
      const int64_t stores = total / 32 * (4 / W);          // whole packed words
      const int shift = shift_of(block_size / (8 * W));
      const bool several = stores >= (int64_t)kDqRuns * kDqThreads * 4 * sm_count();
      const int64_t per = kDqThreads * (several ? kDqRuns : 1);
      auto run = [&](auto kernel) {
        kernel<<<(unsigned)((stores + 31 + per - 1) / per), kDqThreads, 0, st>>>((const uint32_t*)packed, (const __half*)codebook, stores, n_bytes, total,
                                                                            block_size, shift, out, beside);
        return check_launch();
      };
      if (bits == 3) return several ? run(dequant16b_kernel<3, kDqRuns, W, OutT>) : run(dequant16b_kernel<3, 1, W, OutT>);
      if (bits == 2) return several ? run(dequant16b_kernel<2, kDqRuns, W, OutT>) : run(dequant16b_kernel<2, 1, W, OutT>);
      return several ? run(dequant16b_kernel<4, kDqRuns, W, OutT>) : run(dequant16b_kernel<4, 1, W, OutT>);
    };
    if (total >= 32) {
      if constexpr (sizeof(OutT) == 2) {
        if (bits != 2 && block_size % 16 == 0) return start(std::integral_constant<int, 2>{});
      }
      return start(std::integral_constant<int, 1>{});
    }
  }
  const unsigned grid = (unsigned)((total + 255) / 256);
  if (cb_dtype == NB_F16)
    dequant_generic_kernel<__half, OutT><<<grid, 256, 0, st>>>(packed, n_bytes, (const __half*)codebook, bits, block_size, total, out);
  else
    dequant_generic_kernel<float, OutT><<<grid, 256, 0, st>>>(packed, n_bytes, (const float*)codebook, bits, block_size, total, out);
  return check_launch();
}

static int dequant_checked(const uint8_t* packed, const void* codebook, int cb_dtype, int bits, int block_size, int64_t n_rows,
                           int64_t n_cols, void* w_out, int w_dtype, bool beside, void* stream) {
  if (!packed || !codebook || !w_out || n_rows <= 0 || n_cols <= 0 || block_size <= 0) return NB_ERR_ARG;
  if (bits != 2 && bits != 3 && bits != 4) return NB_ERR_ARG;
  if (cb_dtype != NB_F16 && cb_dtype != NB_F32) return NB_ERR_ARG;
  if (int rc = check_device()) return rc;
  const int64_t total = n_rows * n_cols;
  cudaStream_t st = (cudaStream_t)stream;
  switch (w_dtype) {
    case NB_F32: return dequant_dispatch<float>(packed, codebook, cb_dtype, bits, block_size, total, (float*)w_out, beside, st);
    case NB_F16: return dequant_dispatch<__half>(packed, codebook, cb_dtype, bits, block_size, total, (__half*)w_out, beside, st);
    case NB_BF16: return dequant_dispatch<__nv_bfloat16>(packed, codebook, cb_dtype, bits, block_size, total, (__nv_bfloat16*)w_out, beside, st);
    default: return NB_ERR_ARG;
  }
}

int dequant_beside(const uint8_t* packed, const void* codebook, int cb_dtype, int bits, int block_size, int64_t n_rows, int64_t n_cols,
                   void* w_out, int w_dtype, void* stream) {
  return dequant_checked(packed, codebook, cb_dtype, bits, block_size, n_rows, n_cols, w_out, w_dtype, true, stream);
}

}  // namespace nb

using namespace nb;

extern "C" int nb_unpack(const uint8_t* packed, int bits, int64_t count, uint8_t* idx_out, void* stream) {
  if (!packed || !idx_out || count < 0 || (bits != 2 && bits != 3 && bits != 4)) return NB_ERR_ARG;
  if (count == 0) return NB_OK;
  if (int rc = check_device()) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t n_bytes = packed_bytes(count, bits);
  int64_t done = 0;
  if ((uintptr_t)packed % 4 == 0 && (uintptr_t)idx_out % 16 == 0) {
    const int64_t chunks = count / 32;
    if (chunks > 0) {
      const unsigned grid = (unsigned)((chunks + 255) / 256);
      if (bits == 2) unpack32_kernel<2><<<grid, 256, 0, st>>>((const uint32_t*)packed, chunks, (uint4*)idx_out);
      if (bits == 3) unpack32_kernel<3><<<grid, 256, 0, st>>>((const uint32_t*)packed, chunks, (uint4*)idx_out);
      if (bits == 4) unpack32_kernel<4><<<grid, 256, 0, st>>>((const uint32_t*)packed, chunks, (uint4*)idx_out);
      done = chunks * 32;
    }
  }
  if (done < count) {
    const unsigned grid = (unsigned)((count - done + 255) / 256);
    unpack_generic_kernel<<<grid, 256, 0, st>>>(packed, n_bytes, bits, done, count, idx_out);
  }
  return check_launch();
}

extern "C" int nb_pack(const uint8_t* idx, int bits, int64_t count, uint8_t* packed_out, void* stream) {
  if (!idx || !packed_out || count < 0 || (bits != 2 && bits != 3 && bits != 4)) return NB_ERR_ARG;
  if (count == 0) return NB_OK;
  if (int rc = check_device()) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t n_bytes = packed_bytes(count, bits);
  if ((uintptr_t)idx % 16 == 0 && (uintptr_t)packed_out % 4 == 0 && count >= 32) {
    const unsigned grid = (unsigned)((count / 32 + 16 + 127) / 128);
    if (bits == 2) pack32_kernel<2><<<grid, 128, 0, st>>>((const uint4*)idx, count, n_bytes, (uint32_t*)packed_out);
    if (bits == 3) pack32_kernel<3><<<grid, 128, 0, st>>>((const uint4*)idx, count, n_bytes, (uint32_t*)packed_out);
    if (bits == 4) pack32_kernel<4><<<grid, 128, 0, st>>>((const uint4*)idx, count, n_bytes, (uint32_t*)packed_out);
  } else {
    pack_kernel<<<(unsigned)((n_bytes + 255) / 256), 256, 0, st>>>(idx, count, bits, n_bytes, packed_out);
  }
  return check_launch();
}

extern "C" int nb_dequant(const uint8_t* packed, const void* codebook, int cb_dtype, int bits, int block_size,
                          int64_t n_rows, int64_t n_cols, void* w_out, int w_dtype, void* stream) {
  return dequant_checked(packed, codebook, cb_dtype, bits, block_size, n_rows, n_cols, w_out, w_dtype, false, stream);
}

extern "C" int nb_quantize(const float* w, int64_t total, const void* codebook, int cb_dtype, int n_entries, int block_size,
                           uint8_t* idx_out, void* stream) {
  if (!w || !codebook || !idx_out || total <= 0 || block_size <= 0 || n_entries < 2 || n_entries > 256) return NB_ERR_ARG;
  if (cb_dtype != NB_F16 && cb_dtype != NB_F32) return NB_ERR_ARG;
  if (int rc = check_device()) return rc;
  const int64_t padded = (total + block_size - 1) / block_size * block_size;
  if (quantize4_fits(w, codebook, cb_dtype, n_entries, block_size, idx_out, false))
    return launch_quantize4<false>(w, total, padded, (const float*)codebook, n_entries, block_size, idx_out, (cudaStream_t)stream);
  const unsigned grid = (unsigned)((padded + 255) / 256);
  if (cb_dtype == NB_F16)
    quantize_kernel<__half><<<grid, 256, 0, (cudaStream_t)stream>>>(w, total, padded, (const __half*)codebook, n_entries, block_size, idx_out);
  else
    quantize_kernel<float><<<grid, 256, 0, (cudaStream_t)stream>>>(w, total, padded, (const float*)codebook, n_entries, block_size, idx_out);
  return check_launch();
}

extern "C" int nb_quantize_pack(const float* w, int64_t total, const void* codebook, int cb_dtype, int bits, int block_size,
                                uint8_t* packed_out, void* stream) {
  if (!w || !codebook || !packed_out || total <= 0 || block_size <= 0 || (bits != 2 && bits != 3 && bits != 4)) return NB_ERR_ARG;
  if (!quantize4_fits(w, codebook, cb_dtype, 1 << bits, block_size, packed_out, true)) return NB_ERR_SHAPE;
  if (int rc = check_device()) return rc;
  const int64_t padded = (total + block_size - 1) / block_size * block_size;
  return launch_quantize4<true>(w, total, padded, (const float*)codebook, 1 << bits, block_size, packed_out, (cudaStream_t)stream);
}
