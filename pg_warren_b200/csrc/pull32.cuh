// pull32.cuh — the pull of a 32-column f64 SpMM over a CSR's row-split
// schedule (the batched personalised PageRank, the PageRank adjoint).
//
// A row of the gathered operand is 256 bytes and one lane owns one column.
// A unit's targets and weights go to the warp's shared memory; its entries
// are then gathered sixteen at a time into registers, whatever rows they belong
// to, and folded in ascending order per row, as pull_multi folds them, so
// each row's sum is the same to the bit.  A row that ends leaves its sum in
// shared memory, and the tile's rows are emitted together afterwards, four
// rows' operands in flight.  A long row's pieces are combined in piece order
// by the warp that brings the last of them.
//
// What bounds it: the latency of the row gathers, 256 bytes an entry out of
// L2, so the bytes in flight: sixteen rows a warp, twenty warps an SM at 96
// registers.  Eight rows in flight take 1.25 times as long on R-MAT 20's
// personalised ranks; a ring filled by cp.async (24 rows in flight) 1.1 times,
// its copies reading half as many L2 sectors again; 16 warps 1.05 times.  An
// entry takes a target's broadcast, an address, the gather and the fold, and
// a row-end test where its sixteen are not inside one row: 16 warp
// instructions with the rows' updates, against 32 for the pull that staged
// every row in shared memory.  Personalised PageRank of 64 sets on R-MAT 20
// 45.1 -> 36.0 ms; the adjoint of 32 losses on R-MAT 18 45.3 -> 28.8 ms.
//
// The solver's epilogue `Epi` provides:
//   Row                      per-row values, loaded by the tile's lane r for
//                            its row r (coalesced) and shuffled at the emit;
//   Row row(i) const         those of row i;
//   Row shfl(Row, src) const lane src's;
//   Old old(i) const         this lane's column of what emit reads of row i;
//   void emit(i, present, y, Old, Row)   row i's sum for this lane's column;
//   bool active              whether this lane's column runs at all.
#pragma once

#include "pull.cuh"

namespace wc {

constexpr uint32_t kPull32Warps = 4;  // warps a block
constexpr uint32_t kPull32Rows = 16;  // rows whose sums wait to be emitted
constexpr uint32_t kPull32Unroll = 16;  // entries gathered at once

// A warp's shared memory: the unit's targets and weights, the rows' sums.
template <class W> struct alignas(16) Pull32Warp {
  double y[kPull32Rows][32];
  WSpan<W> w;
  uint32_t j[kTileEntries];
};
template <class W> constexpr size_t pull32_smem() { return kPull32Warps * sizeof(Pull32Warp<W>); }

// The warp's units of A's schedule (warp, warp + warps, ...): X is the
// gathered operand (n × 32).
template <class W, class Epi>
__device__ inline void pull32_units(const CsrView<W>& A, const double* __restrict__ X, Epi& epi,
                                    DeviceError* err, Partial<double, WC_OP_PLUS>* carry,
                                    Pull32Warp<W>& sm) {
  constexpr int ADD = WC_OP_PLUS;
  constexpr uint32_t U = kPull32Unroll;
  typedef Partial<double, ADD> Part;
  typedef typename Epi::Row Row;
  typedef typename Epi::Old Old;
  const unsigned lane = threadIdx.x & 31;
  const bool active = epi.active;
  const double* Xl = X + lane;
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  // The product of entry k of the unit with its gathered value.
  auto term = [&](uint32_t k, double x) {
    if constexpr (WSize<W>::v == 0) return x;
    else return (double)sm.w.v[k] * x;
  };
  auto gather = [&](uint32_t k) { return active ? __ldg(Xl + (size_t)sm.j[k] * 32) : 0.0; };

  Unit unit{};
  if (warp < A.unit_count) unit = A.units[warp];
  for (uint32_t u = warp; u < A.unit_count; u += warps) {
    Unit next{};
    if (u + warps < A.unit_count) next = A.units[u + warps];
    const bool tile = (unit.c >> 31) == 0;
    const uint32_t a = unit.a;
    const uint32_t R = tile ? unit.b - unit.a : 1;
    const uint32_t base = unit_first(unit), count = unit_count(unit);
    __syncwarp();  // every lane is done with the last unit's shared memory
#pragma unroll
    for (uint32_t q = 0; q < kTileEntries / 32; q++) {
      const uint32_t k = 32 * q + lane;
      if (k < count) {
        sm.j[k] = __ldcs(A.tgt + base + k);
        if constexpr (WSize<W>::v != 0) sm.w.v[k] = __ldcs(A.w + base + k);
      }
    }
    uint32_t hi_l = count;
    Row row_l{};
    if (tile && lane < R) {
      hi_l = __ldg(A.off + a + lane + 1) - base;
      row_l = epi.row(a + lane);
    }
    // The next unit's entries into L2 while this one folds.
    if (u + warps < A.unit_count && 32 * lane < unit_count(next)) {
      const uint32_t e = unit_first(next) + 32 * lane;
      asm volatile("prefetch.global.L2 [%0];" ::"l"(A.tgt + e));
      if constexpr (WSize<W>::v != 0) {
        asm volatile("prefetch.global.L2 [%0];" ::"l"(A.w + e));
        if constexpr (WSize<W>::v == 8)
          if (32 * lane + 16 < unit_count(next))
            asm volatile("prefetch.global.L2 [%0];" ::"l"(A.w + e + 16));
      }
    }
    __syncwarp();
    // A sum starts at -0.0, to which the first product adds as itself.
    double acc = -0.0;
    uint32_t k = 0;
    for (uint32_t r0 = 0; r0 < R; r0 += kPull32Rows) {
      const uint32_t r1 = min(R, r0 + kPull32Rows);
      const uint32_t end = __shfl_sync(0xffffffffu, hi_l, r1 - 1);
      uint32_t r = r0;
      uint32_t hi = __shfl_sync(0xffffffffu, hi_l, r);
      // Row r's sum is complete at entry k.
      auto close = [&](uint32_t at) {
        while (at == hi && r < r1) {
          sm.y[r - r0][lane] = acc;
          acc = -0.0;
          r++;
          hi = __shfl_sync(0xffffffffu, hi_l, r & 31);
        }
      };
      for (; k + U <= end; k += U) {
        double x[U];
#pragma unroll
        for (uint32_t q = 0; q < U; q++) x[q] = gather(k + q);
        if (!tile || k + U <= hi) {
#pragma unroll
          for (uint32_t q = 0; q < U; q++) acc = acc + term(k + q, x[q]);
        } else {
#pragma unroll
          for (uint32_t q = 0; q < U; q++) {
            if (k + q == hi) close(k + q);
            acc = acc + term(k + q, x[q]);
          }
        }
      }
      if (k < end) {
        double x[U];
#pragma unroll
        for (uint32_t q = 0; q < U - 1; q++) x[q] = k + q < end ? gather(k + q) : 0.0;
#pragma unroll
        for (uint32_t q = 0; q < U - 1; q++)
          if (k + q < end) {
            if (tile && k + q == hi) close(k + q);
            acc = acc + term(k + q, x[q]);
          }
        k = end;
      }
      if (!tile) break;
      close(k);
      // The rows' sums are in: emit them, four rows' operands in flight.
      uint32_t lo = r0 ? __shfl_sync(0xffffffffu, hi_l, r0 - 1) : 0u;
      for (uint32_t e = r0; e < r1; e += 4) {
        Old old[4];
#pragma unroll
        for (uint32_t q = 0; q < 4; q++)
          if (e + q < r1) old[q] = epi.old(a + e + q);
#pragma unroll
        for (uint32_t q = 0; q < 4; q++)
          if (e + q < r1) {
            const uint32_t row_end = __shfl_sync(0xffffffffu, hi_l, e + q);
            epi.emit(a + e + q, row_end > lo, sm.y[e + q - r0][lane], old[q],
                     epi.shfl(row_l, e + q));
            lo = row_end;
          }
      }
    }
    if (!tile) {
      // A piece of a long row: its partial in the carry slot; the warp that
      // brings the row's last piece combines the pieces in order and emits.
      const uint32_t row = a, slot = unit.c & 0x7fffffffu;
      const uint32_t row_lo = __ldg(A.off + row);
      const uint32_t deg = __ldg(A.off + row + 1) - row_lo;
      const uint32_t pieces = (deg + kPieceEntries - 1) / kPieceEntries;
      const uint32_t first = slot - (base - row_lo) / kPieceEntries;
      carry[(size_t)slot * 32 + lane] = Part{Acc<double, ADD>::of(acc), true};
      __threadfence();
      __syncwarp();
      uint32_t arrived = 0;
      if (lane == 0) arrived = atomicAdd(A.counters + first, 1u);
      arrived = __shfl_sync(0xffffffffu, arrived, 0);
      if (arrived == pieces - 1) {
        __threadfence();
        const Part total = combine_pieces<double, ADD, 32>(carry, first, pieces, lane, 0);
        double y;
        total.acc.value(&y);
        epi.emit(row, true, y, epi.old(row), epi.row(row));
        __syncwarp();
        if (lane == 0) A.counters[first] = 0;
      }
    }
    unit = next;
  }
}

}  // namespace wc
