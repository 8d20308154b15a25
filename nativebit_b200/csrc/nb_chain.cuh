// The layout in which the decode step's launches hand activations to the packed matvec behind them (nb_chain.cu).
#pragma once
#include <cuda_fp16.h>

#include "nb_device.cuh"

namespace nb {

// One activation row's 128-column block of one term: four segments of 32 values (a lane's share of a unit), the four 16-byte
// chunks of segment t at chunk ^ t ^ term, so that the eight lanes that read together (four segments of both terms of a row)
// meet eight different bank groups.  Four values are kept in the order 0, 2, 1, 3, that of lookup4_pairs' weights.
__device__ __forceinline__ uint8_t* chain_term(uint8_t* terms, int bpr, int row, int s, int n) {
  return terms + ((size_t)(2 * row + s) * bpr + (n >> 7)) * 256 + ((n >> 5) & 3) * 64 + ((((n >> 3) & 3) ^ ((n >> 5) & 3) ^ s) << 4) +
         ((n & 4) | (n & 1) << 1 | (n >> 1 & 1)) * 2;
}
// Saturating like every split into terms here, and NaN stays NaN in both: it has to come out of the products behind.
__device__ __forceinline__ void store_chain_terms(uint8_t* terms, int bpr, int row, int n, float v) {
  const __half hi = to_half_sat(v);
  *reinterpret_cast<__half*>(chain_term(terms, bpr, row, 0, n)) = hi;
  *reinterpret_cast<__half*>(chain_term(terms, bpr, row, 1, n)) = to_half_sat(v - __half2float(hi));
}

}  // namespace nb
