// spmm_rows.cuh — the pull Y = A ⊗ X over a block of up to 32 columns of a
// row-major X (wc_spmm), walked by the row-split schedule.
//
// A warp takes a unit.  Its targets and weights (cast to the element once an
// entry, not once a column) go to the warp's shared memory; then LPR = P / V
// lanes own a row's P columns, V consecutive ones a lane (one 16-byte gather
// where X allows it), and the warp's G = 32 / LPR lane groups each take a run
// of the tile's rows of about equal entries.  A group gathers up to eight of a
// row's entries at once and folds them in ascending order, the reference's
// order (compute/product/kernel.rs:184-198) to the bit.  A long row's piece is
// split between the groups as contiguous runs, combined left to right, and a
// row's pieces in piece order by the last to finish.
//
// What bounds it: the latency of the gathers of X's rows, row after row of a
// group.  pull_multi, which runs the blocks that this does not pay for
// (spmm_rows_pay), has a group's offsets, targets and gathers one after another,
// a lane a column: 16 weighted f32 columns over an R-MAT graph of 300,007 nodes
// and 4.6 M entries take it 405 µs, 196 here.
#pragma once

#include "pull.cuh"

namespace wc {

constexpr int kSpmmWarps = 8;  // warps a block

template <class E> struct SpmmWarp {
  uint32_t j[kTileEntries];
  uint32_t end[kTileRows];  // the tile's rows' ends, from its first entry
  E w[kTileEntries];
};

// V consecutive elements, moved as one access.
template <class E, int V> struct alignas(sizeof(E) * V) SpmmVec { E v[V]; };

template <class E, int V> __device__ inline SpmmVec<E, V> spmm_load(const E* p) {
  SpmmVec<E, V> r;
  if constexpr (sizeof r == 16) {
    const uint4 w = __ldg(reinterpret_cast<const uint4*>(p));
    memcpy(&r, &w, 16);
  } else {
#pragma unroll
    for (int v = 0; v < V; v++) r.v[v] = load_x(p, v);
  }
  return r;
}

// An entry's weight as the element (E{1} where every weight is 1).
template <class E, int S, class W>
__device__ inline int32_t spmm_weight(const W* w, uint64_t e, E* out) {
  if constexpr (WSize<W>::v == 0 || !Entry<E, S, W>::reads_weight) {
    return Elem<E>::from_weight(1.0, out);
  } else if constexpr (WSize<W>::v == 8) {
    return Elem<E>::from_weight(__ldcs(w + e), out);
  } else {
    *out = (E)__ldcs(w + e);
    return 0;
  }
}

// `epi.cells(row, c, present, out)` is called once per (row, lane's first
// column c); X's rows are `ld` elements apart, `columns` of them in this
// block (a multiple of V).
template <class E, int S, class W, int P, int V, class Epi>
__device__ inline void spmm_rows(const CsrView<W>& A, const E* __restrict__ X, Epi& epi,
                                 DeviceError* err, Partial<E, semiring_add(S)>* carry, uint32_t ld,
                                 uint32_t columns, SpmmWarp<E>& sm) {
  constexpr int ADD = semiring_add(S), MUL = semiring_mul(S);
  constexpr uint32_t LPR = P / V, G = 32 / LPR, U = 8;
  typedef Acc<E, ADD> Sum;
  typedef Partial<E, ADD> Part;
  typedef SpmmVec<E, V> Vec;
  const unsigned lane = threadIdx.x & 31;
  const uint32_t g = lane / LPR, c = (lane % LPR) * V;
  const bool active = c < columns;
  const E* Xc = X + c;
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  Unit next{};
  if (warp < A.unit_count) next = A.units[warp];
  for (uint32_t u = warp; u < A.unit_count; u += warps) {
    const Unit unit = next;
    if (u + warps < A.unit_count) next = A.units[u + warps];
    const bool tile = (unit.c >> 31) == 0;
    const uint32_t R = tile ? unit.b - unit.a : 1;
    const uint32_t base = unit_first(unit), count = unit_count(unit);
    __syncwarp();  // every lane is done with the last unit's shared memory
#pragma unroll
    for (uint32_t q = 0; q < kTileEntries / 32; q++) {
      const uint32_t k = 32 * q + lane;
      if (k < count) {
        sm.j[k] = __ldcs(A.tgt + base + k);
        E w{};
        const int32_t s = spmm_weight<E, S, W>(A.w, (uint64_t)base + k, &w);
        if (s) raise(err, s, unit.a);
        sm.w[k] = w;
      }
    }
    uint32_t end_l = count;
    if (tile && lane < R) end_l = __ldg(A.off + unit.a + lane + 1) - base;
    sm.end[lane] = end_l;
    // Row r belongs to the group its first entry falls to, of G about equal
    // runs of entries; the groups' rows are consecutive runs.
    uint32_t r = 0, r_end = 1, k, k_end;
    if (tile) {
      const uint32_t up = __shfl_up_sync(0xffffffffu, end_l, 1);
      const uint32_t first = lane ? up : 0u;
      const uint32_t mine = count ? min(G - 1, first * G / count) : 0u;
      r = r_end = 0;
#pragma unroll
      for (uint32_t q = 0; q < G; q++) {
        const uint32_t before = __popc(__ballot_sync(0xffffffffu, lane < R && mine < q));
        const uint32_t through = __popc(__ballot_sync(0xffffffffu, lane < R && mine <= q));
        if (g == q) {
          r = before;
          r_end = through;
        }
      }
      const uint32_t lo = __shfl_sync(0xffffffffu, end_l, (r + 31) & 31);
      const uint32_t hi = __shfl_sync(0xffffffffu, end_l, (r_end + 31) & 31);
      k = r ? lo : 0u;
      k_end = r_end > r ? hi : k;
    } else {
      constexpr uint32_t run = kPieceEntries / G;
      k = min(count, g * run);
      k_end = min(count, k + run);
    }
    __syncwarp();
    Sum acc[V];
#pragma unroll
    for (int v = 0; v < V; v++) acc[v] = Sum::of(E{});
    bool present = false;
    int32_t bad = 0;
    // Row after row of the group; a piece is one run of one row.
    while (tile ? r < r_end : k < k_end) {
      const uint32_t hi = tile ? sm.end[r] : k_end;
      for (; k < hi; k += U) {
        const uint32_t n = min(U, hi - k);
        Vec x[U];
#pragma unroll
        for (uint32_t q = 0; q < U; q++)
          if (q < n && active) x[q] = spmm_load<E, V>(Xc + (size_t)sm.j[k + q] * ld);
#pragma unroll
        for (uint32_t q = 0; q < U; q++)
          if (q < n && active) {
            const E w = sm.w[k + q];
#pragma unroll
            for (int v = 0; v < V; v++) {
              E p;
              const int32_t s = Multiply<E, ADD, MUL>::go(w, x[q].v[v], &p);
              if (s) bad = s;
              acc[v] = present || q ? Sum::combine(acc[v], Sum::of(p)) : Sum::of(p);
            }
          }
        present = true;
      }
      k = hi;
      if (!tile) break;
      E out[V];
#pragma unroll
      for (int v = 0; v < V; v++) {
        out[v] = E{};
        if (present) {
          const int32_t s = acc[v].value(&out[v]);
          if (s) bad = s;
        }
      }
      if (active) epi.cells(unit.a + r, c, present, out);
      present = false;
      r++;
    }
    if (!tile) {
      // A piece of a long row: the groups' runs left to right, then the carry.
      Part mine[V];
#pragma unroll
      for (int v = 0; v < V; v++) mine[v] = Part{present ? acc[v] : Sum::of(E{}), present};
      auto join_groups = [&]() {
        for (uint32_t o = LPR; o < 32; o <<= 1)
#pragma unroll
          for (int v = 0; v < V; v++) {
            const Part other = shfl_partial(mine[v], o);
            if ((g & (2 * (o / LPR) - 1)) == 0) mine[v] = join(mine[v], other);
          }
      };
      join_groups();
      const uint32_t row = unit.a, slot = unit.c & 0x7fffffffu;
      const uint32_t row_lo = __ldg(A.off + row);
      const uint32_t deg = __ldg(A.off + row + 1) - row_lo;
      const uint32_t pieces = (deg + kPieceEntries - 1) / kPieceEntries;
      const uint32_t first = slot - (base - row_lo) / kPieceEntries;
      if (g == 0 && active)
#pragma unroll
        for (int v = 0; v < V; v++) carry[(size_t)slot * P + c + v] = mine[v];
      __syncwarp();
      uint32_t arrived = 0;
      if (lane == 0) arrived = arrive_acq_rel(A.counters + first);
      arrived = __shfl_sync(0xffffffffu, arrived, 0);
      if (arrived == pieces - 1) {
        __threadfence();
        // The groups take contiguous runs of the pieces.
        const uint32_t per = (pieces + G - 1) / G;
        const uint32_t p0 = min(pieces, g * per), p1 = min(pieces, p0 + per);
#pragma unroll
        for (int v = 0; v < V; v++) mine[v] = Part{Sum::of(E{}), false};
        for (uint32_t p = p0; active && p < p1; p++)
#pragma unroll
          for (int v = 0; v < V; v++)
            mine[v] = join(mine[v], load_cg(carry + (size_t)(first + p) * P + c + v));
        __syncwarp();
        join_groups();
        if (g == 0 && active) {
          E out[V];
#pragma unroll
          for (int v = 0; v < V; v++) {
            const int32_t s = mine[v].acc.value(&out[v]);
            if (s) bad = s;
          }
          epi.cells(row, c, true, out);
        }
        if (lane == 0) A.counters[first] = 0;
      }
    }
    if (bad) raise(err, bad, unit.a);
  }
}

}  // namespace wc
