// row_chunks.h — a row's entries a chunk at a time, by position.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define WC_HOST_DEVICE __host__ __device__
#else
#define WC_HOST_DEVICE
#endif

namespace wc {

// Calls chunk(e) for e = first, first + step, ... below `end`, until one
// returns true.  Positions are counted in 64 bits: an entry's fits 32, but the
// step past a row that ends within one of 2^32 does not, and would begin again
// at the first row.
#ifdef __CUDACC__
#pragma nv_exec_check_disable
#endif
template <class Chunk>
WC_HOST_DEVICE inline void each_chunk(uint32_t first, uint32_t end, uint32_t step, Chunk&& chunk) {
  for (uint64_t e = first; e < end; e += step)
    if (chunk(e)) return;
}

// Whether entry q of a row [lo, hi) is in it (lo + q may not fit 32 bits).
WC_HOST_DEVICE inline bool in_row(uint32_t lo, uint32_t hi, uint32_t q) { return q < hi - lo; }

}  // namespace wc
