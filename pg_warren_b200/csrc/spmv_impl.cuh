// spmv_impl.cuh — kernels and dispatch of the product y = A ⊗ x (SpMV) and
// Y = A ⊗ X (SpMM), instantiated once per element type in spmv_<dtype>.cu.
#pragma once

#include <type_traits>

#include "lanes.cuh"
#include "pull.cuh"
#include "pull_multi.cuh"
#include "product.h"
#include "spmm_rows.cuh"

namespace wc {

template <class E, int S, class W>
__global__ void __launch_bounds__(kPullThreads, 3)
    spmv_pull_kernel(CsrView<W> A, const E* __restrict__ x, WriteEpi<E, S> epi, DeviceError* err) {
  extern __shared__ __align__(16) unsigned char smem[];
  PullRing<E, W>* ring = reinterpret_cast<PullRing<E, W>*>(smem) + (threadIdx.x >> 5);
  pull_units<E, S, W>(A, x, epi, err, ring);
}

template <class E, int S, class W>
__global__ void __launch_bounds__(kLaneThreads, 1)
    spmv_lane_kernel(LaneView<W> A, const E* __restrict__ x, WriteEpi<E, S> epi, DeviceError* err) {
  extern __shared__ __align__(16) unsigned char smem[];
  E* hot = reinterpret_cast<E*>(smem);
  lane_fill_hot<E, W>(A, x, hot);
  lane_units<E, S, W>(A, x, hot, epi, err);
}

// SpMM, width > 1: spmm_rows.cuh or pull_multi.cuh (spmm_rows_pay says which)
// over a block of P columns at a time, and the write
// (compute/product/kernel.rs:200-240) per (row, column).
template <class E, int S, int V> struct SpmmEpi {
  WriteArgs w;
  E* y;
  uint32_t width, c0;
  DeviceError* err;
  __device__ void cells(uint32_t row, uint32_t c, bool present, const E (&t)[V]) {
    E* out = y + (size_t)row * width + c0 + c;
    const E identity = Identity<E>::of(semiring_add(S));
    if (V * sizeof(E) == 16 && !w.mask && w.accumulate < 0) {
      SpmmVec<E, V> r;
#pragma unroll
      for (int v = 0; v < V; v++) r.v[v] = present ? t[v] : identity;
      *reinterpret_cast<SpmmVec<E, V>*>(out) = r;
      return;
    }
    const bool selected = mask_selects(w, row);
#pragma unroll 1
    for (int v = 0; v < V; v++) {
      if (!selected) {
        if (w.replace) out[v] = identity;
      } else if (w.accumulate < 0) {
        out[v] = present ? t[v] : identity;
      } else if (present) {
        E r;
        int32_t s = apply_rt<E>(w.accumulate, out[v], t[v], &r);
        if (s) raise(err, s, row);
        else out[v] = r;
      }
    }
  }
};

template <class E, int S, class W, int P, int V>
__global__ void __launch_bounds__(32 * kSpmmWarps, 3)
    spmm_rows_kernel(CsrView<W> A, const E* __restrict__ x, E* y, uint32_t width, uint32_t c0,
                     WriteArgs w, DeviceError* err, Partial<E, semiring_add(S)>* carry) {
  __shared__ SpmmWarp<E> sm[kSpmmWarps];
  SpmmEpi<E, S, V> epi{w, y, width, c0, err};
  spmm_rows<E, S, W, P, V>(A, x + c0, epi, err, carry, width, min(P, width - c0),
                           sm[threadIdx.x >> 5]);
}

// A lane takes 16 bytes of a row where every row of x and y starts on a
// 16-byte boundary (and so every block of 32 columns, and every lane's part),
// else one element; and one element of the types whose accumulator is wide.
template <class E, int S> constexpr int spmm_vector() {
  return sizeof(Acc<E, semiring_add(S)>) > 8 || sizeof(E) < 4 ? 1 : 16 / (int)sizeof(E);
}

// The same for pull_multi, a column a call.
template <class E, int S> struct SpmmCellEpi {
  WriteArgs w;
  E* y;
  uint32_t width, c0;
  DeviceError* err;
  __device__ void cell(uint32_t row, uint32_t c, bool present, E t) {
    const uint32_t col = c0 + c;
    if (col >= width) return;
    E* out = y + (size_t)row * width + col;
    const E identity = Identity<E>::of(semiring_add(S));
    if (!mask_selects(w, row)) {
      if (w.replace) *out = identity;
      return;
    }
    if (w.accumulate < 0) {
      *out = present ? t : identity;
    } else if (present) {
      E r;
      int32_t s = apply_rt<E>(w.accumulate, *out, t, &r);
      if (s) raise(err, s, row);
      else *out = r;
    }
  }
};

template <class E, int S, class W, int P>
__global__ void __launch_bounds__(256)
    spmm_multi_kernel(CsrView<W> A, const E* __restrict__ x, E* y, uint32_t width, uint32_t c0,
                      WriteArgs w, DeviceError* err, Partial<E, semiring_add(S)>* carry) {
  SpmmCellEpi<E, S> epi{w, y, width, c0, err};
  pull_multi<E, S, W, P>(A, x + c0, epi, err, carry, width, min(P, width - c0));
}

// Whether a block of `cols` columns is spmm_rows' (else pull_multi's): `vector`,
// a lane takes 16 bytes.  It casts an entry's weight once, not once a column,
// and gathers fewer, larger pieces of X's rows; it stages each unit first,
// which a few columns of elements that need no cast do not earn back.  Device
// time, pull_multi and spmm_rows, µs, over a G(n, m) of 16,628 nodes in rows of
// 8; over an R-MAT of 262,144 in rows of 16.
//   f32, weights cast:     4 columns 16.4, 12.6; 246, 150.  32: 57.1, 20.5; 498, 179
//   f64, weights, plus:    4 columns 11.4, 14.4; 152, 168.  8: 22.6, 18.7; 269, 194.
//                          32: 37.0, 34.1; 365, 237
//   f64, no weights:       4 columns 10.4, 14.4; 86, 165.  32: 32.0, 33.5; 226, 234
//   i64 min_plus, weights: 4 columns 14.5, 15.5; 194, 220.  32: 49.2, 37.0; 438, 324
// pull_multi's over spmm_rows' time, likewise: f64 min_plus 8 columns 0.8; 0.9, 32:
// 0.95; 1.2 (G(n, m) of 1.2 M entries 1.4); f32 without weights 16: 1.5; 0.9, 32:
// 1.8; 1.0; i64 plus_times, whose sums are of 128 bits, 0.6 to 0.95 at every width;
// bool 4: 1.0; 0.8, 32: 1.2; 1.0.
template <class E, int S, class W>
bool spmm_rows_pay(const PullLaunch& L, uint32_t cols, bool vector) {
  constexpr bool f64 = std::is_same_v<E, double>, i64 = std::is_same_v<E, int64_t>;
  if constexpr (std::is_same_v<W, double> && !f64) return true;  // a cast an entry
  if constexpr (sizeof(E) == 1) return cols > 16 && (L.skewed || L.entries < 3u << 18);
  if (!vector) return false;
  if constexpr (f64) {
    if (semiring_add(S) == WC_OP_PLUS) return cols > 4 && (!L.skewed || L.entries >= 3u << 18);
    return cols > 8 && L.entries >= (L.skewed ? 1u << 21 : 1u << 20);
  }
  if (L.skewed) return cols > 16 && L.entries >= 1u << 20;
  return cols > (i64 ? 4u : 8u);
}

template <class E, int S, class W, int P>
void launch_spmm(const CsrView<W>& A, const PullLaunch& L, const E* x, E* y, uint32_t c0,
                 uint32_t blocks) {
  constexpr int V = spmm_vector<E, S>();
  // The types spmm_rows is built for: those that spmm_rows_pay may name.
  constexpr bool f64 = std::is_same_v<E, double>, none = WSize<W>::v == 0;
  constexpr bool cast = std::is_same_v<W, double> && !f64;
  constexpr bool rows = cast ? Entry<E, S, W>::reads_weight
                             : sizeof(E) == 1 ? P > 16 : V > 1 && P > 4 && !(f64 && none);
  auto* carry = static_cast<Partial<E, semiring_add(S)>*>(L.carry_multi);
  const uint32_t cols = L.width - c0 < 32 ? L.width - c0 : 32;
  const uintptr_t at = reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y);
  const bool vector = V > 1 && P >= V && at % 16 == 0 && (size_t)L.width * sizeof(E) % 16 == 0;
  if constexpr (rows) {
    if (spmm_rows_pay<E, S, W>(L, cols, vector)) {
      if constexpr (V > 1 && P >= V) {
        if (vector) {
          note_launch(), spmm_rows_kernel<E, S, W, P, V><<<blocks, 32 * kSpmmWarps, 0, L.stream>>>(
              A, x, y, L.width, c0, L.write, L.err, carry);
          return;
        }
      }
      if constexpr (cast || sizeof(E) == 1) {
        note_launch(), spmm_rows_kernel<E, S, W, P, 1><<<blocks, 32 * kSpmmWarps, 0, L.stream>>>(
            A, x, y, L.width, c0, L.write, L.err, carry);
        return;
      }
    }
  }
  if constexpr (!(rows && cast))
    note_launch(), spmm_multi_kernel<E, S, W, P><<<blocks, 256, 0, L.stream>>>(
        A, x, y, L.width, c0, L.write, L.err, carry);
}

template <class E, int S, class W>
wc_status launch_one(const PullLaunch& L, const void* x, void* y) {
  CsrView<W> A{L.off, L.tgt, static_cast<const W*>(L.weights), L.units, L.unit_count,
               L.counters, L.carry};
  if (L.width == 1 && L.lanes) {
    WriteEpi<E, S> epi{L.write, static_cast<E*>(y), L.err};
    static const cudaError_t attr = cudaFuncSetAttribute(
        spmv_lane_kernel<E, S, W>, cudaFuncAttributeMaxDynamicSharedMemorySize,
        (int)(kHotSlots * sizeof(E)));
    if (attr != cudaSuccess) return cuda_status(attr, L.detail, "product kernel attributes");
    const LaneView<W> V = lane_view<W>(L);
    note_launch(), spmv_lane_kernel<E, S, W><<<lane_grid(L), kLaneThreads,
                                               V.hot_count * sizeof(E), L.stream>>>(
        V, static_cast<const E*>(x), epi, L.err);
  } else if (L.width == 1) {
    WriteEpi<E, S> epi{L.write, static_cast<E*>(y), L.err};
    constexpr size_t smem = pull_smem_bytes<E, W>();
    static const cudaError_t attr = cudaFuncSetAttribute(
        spmv_pull_kernel<E, S, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (attr != cudaSuccess) return cuda_status(attr, L.detail, "product kernel attributes");
    uint32_t blocks = (L.unit_count + kPullWarps - 1) / kPullWarps;
    blocks = blocks < 1 ? 1 : (blocks > L.max_blocks ? L.max_blocks : blocks);
    note_launch(), spmv_pull_kernel<E, S, W><<<blocks, kPullThreads, smem, L.stream>>>(
        A, static_cast<const E*>(x), epi, L.err);
  } else {
    uint32_t blocks = (L.unit_count + kSpmmWarps - 1) / kSpmmWarps;
    blocks = blocks < 1 ? 1 : (blocks > L.max_blocks ? L.max_blocks : blocks);
    // Blocks of P columns: P the smallest power of two covering the width,
    // at most 32.
    const E* xe = static_cast<const E*>(x);
    E* ye = static_cast<E*>(y);
    for (uint32_t c0 = 0; c0 < L.width; c0 += 32) {
      const uint32_t cols = L.width - c0;
      if (cols > 16) launch_spmm<E, S, W, 32>(A, L, xe, ye, c0, blocks);
      else if (cols > 8) launch_spmm<E, S, W, 16>(A, L, xe, ye, c0, blocks);
      else if (cols > 4) launch_spmm<E, S, W, 8>(A, L, xe, ye, c0, blocks);
      else if (cols > 2) launch_spmm<E, S, W, 4>(A, L, xe, ye, c0, blocks);
      else launch_spmm<E, S, W, 2>(A, L, xe, ye, c0, blocks);
    }
  }
  return cuda_status(cudaGetLastError(), L.detail, "product kernel launch");
}

template <class E, class W>
wc_status launch_semiring(const PullLaunch& L, const void* x, void* y) {
  switch (L.semiring) {
    case WC_PLUS_TIMES: return launch_one<E, WC_PLUS_TIMES, W>(L, x, y);
    case WC_MIN_PLUS: return launch_one<E, WC_MIN_PLUS, W>(L, x, y);
    case WC_MAX_PLUS: return launch_one<E, WC_MAX_PLUS, W>(L, x, y);
    case WC_MAX_TIMES: return launch_one<E, WC_MAX_TIMES, W>(L, x, y);
    case WC_MIN_TIMES: return launch_one<E, WC_MIN_TIMES, W>(L, x, y);
    case WC_LOR_LAND: return launch_one<E, WC_LOR_LAND, W>(L, x, y);
    case WC_ANY_PAIR: return launch_one<E, WC_ANY_PAIR, W>(L, x, y);
    case WC_PLUS_PAIR: return launch_one<E, WC_PLUS_PAIR, W>(L, x, y);
    case WC_PLUS_FIRST: return launch_one<E, WC_PLUS_FIRST, W>(L, x, y);
    case WC_PLUS_SECOND: return launch_one<E, WC_PLUS_SECOND, W>(L, x, y);
    case WC_MIN_FIRST: return launch_one<E, WC_MIN_FIRST, W>(L, x, y);
    case WC_MIN_SECOND: return launch_one<E, WC_MIN_SECOND, W>(L, x, y);
    case WC_MAX_SECOND: return launch_one<E, WC_MAX_SECOND, W>(L, x, y);
  }
  return WC_UNKNOWN_SEMIRING;
}

template <class E>
wc_status launch_typed(const PullLaunch& L, const void* x, void* y) {
  switch (L.weight_kind) {
    case WEIGHTS_F64: return launch_semiring<E, double>(L, x, y);
    case WEIGHTS_I32:  // prepare_pull: the i64 products alone read the i32 copy
      if constexpr (std::is_same_v<E, int64_t>) return launch_semiring<E, int32_t>(L, x, y);
      return WC_DTYPE_MISMATCH;
    default: return launch_semiring<E, void>(L, x, y);
  }
}

}  // namespace wc
