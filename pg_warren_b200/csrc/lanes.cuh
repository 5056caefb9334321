// lanes.cuh — the pull y_i = ⊕_{entries (i, j)} ⊗(w_ij, x_j) of one vector
// over a lane-major copy (LaneCsr, built by lanes.cu): a warp per unit, each
// lane folding one row of a slice in its stored order, or the pieces of a
// long row folded and combined as pull.cuh folds and combines them, so every
// row's result is pull_units' to the bit.
//
// What bounds it: the gathers of x.  Every entry reads a value at a random
// place; L1 serves about one such line a cycle and each miss costs a 32-byte
// L2 sector.  The row-major kernel spent 4.7 warp instructions an entry
// moving products from the lanes that gathered them to the lane that folds
// the row; here a step of 32 entries is a target load, a gather and the
// fold.  The values of the most gathered nodes are copied to shared memory
// by each block first (A.hot): those gathers cost a bank access instead.
// One block of 24 warps an SM, so the table exists once, at 80 registers a
// thread: four gathers a lane in flight and the next four targets loading.
// 32 warps (64 registers) spill and take 1.2 times as long over R-MAT 22's
// weighted product; eight gathers in flight spill at either size (1.5 times).
// The code is kept to one copy of each loop: a small graph's launch is over
// in the time its instructions take to arrive.
//
// R-MAT 22 (65 M entries): the weighted f64 plus_times product 768 -> 381 µs,
// a PageRank solve of 10 iterations 5.89 -> 3.53 ms; min_plus over i64 on a
// G(n, m) of 16 M entries 116 -> 98 µs.  Over few entries the row-split schedule
// is the faster: lanes_pay (product.cu), solve_lanes_pay (pagerank.cu).
#pragma once

#include "lanes.h"
#include "pull.cuh"

namespace wc {

constexpr int kLaneThreads = 768;

template <class W> struct LaneView {
  const LaneUnit* units;
  uint32_t unit_count;
  const uint32_t* rows;     // NULL: the vectors are in the sorted order itself,
  uint32_t first_short;     //   the short rows from this number on
  const uint32_t* numbers;  //   and a long row's number by its id
  const uint16_t* lengths;
  uint32_t filled, shorts;  // of `rows`: those with entries, then to here the empty ones
  const uint32_t* tgt;
  const W* w;
  const uint32_t* off;  // the row-major offsets (the long rows' lengths)
  const uint32_t* hot;
  uint32_t hot_count;
  uint32_t* counters;
  void* carry;
};

template <class W> LaneView<W> lane_view(const PullLaunch& L) {
  const LaneCsr& c = *L.lanes;
  return LaneView<W>{c.units.as<LaneUnit>(), c.count, c.rows.as<uint32_t>(), 0u, nullptr,
                     c.lengths.as<uint16_t>(), c.filled, c.shorts, c.targets.as<uint32_t>(),
                     static_cast<const W*>(L.lane_weights), L.off, c.hot.as<uint32_t>(),
                     c.hot_count, L.counters, L.carry};
}

// One block an SM, none without a unit or a block's worth of empty rows.
inline uint32_t lane_grid(const PullLaunch& L) {
  const uint32_t sms = L.max_blocks / 8;
  const uint32_t useful =
      L.lanes->count + (L.lanes->shorts - L.lanes->filled + kLaneThreads - 1) / kLaneThreads;
  return useful < sms ? (useful ? useful : 1u) : sms;
}

template <class W> struct LaneWeight { typedef W type; };
template <> struct LaneWeight<void> { typedef char type; };

// The block's table of hot values.  Every thread of the block calls it.
template <class E, class W>
__device__ inline void lane_fill_hot(const LaneView<W>& A, const E* __restrict__ x, E* hot) {
  for (uint32_t h = threadIdx.x; h < A.hot_count; h += blockDim.x)
    hot[h] = load_x(x, __ldg(A.hot + h));
  __syncthreads();
}

// Adds `n` arrivals to a long row's counter (arrive_acq_rel's, of several
// pieces at once): the earlier arrivals.
__device__ inline uint32_t arrive_many(uint32_t* counter, uint32_t n) {
  uint32_t old;
  asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], %2;"
               : "=r"(old) : "l"(counter), "r"(n) : "memory");
  return old;
}

// Lane src's value (XOR: lane ^ src's), word by word.
template <class T, bool XOR = false> __device__ inline T shfl_value(const T& v, unsigned src) {
  constexpr int N = (sizeof(T) + 3) / 4;
  uint32_t words[N] = {};
  memcpy(words, &v, sizeof v);
#pragma unroll
  for (int i = 0; i < N; i++)
    words[i] = XOR ? __shfl_xor_sync(0xffffffffu, words[i], src)
                   : __shfl_sync(0xffffffffu, words[i], src);
  T r;
  memcpy(&r, words, sizeof r);
  return r;
}

// The lanes' values combined left to right, pairs first (lane 0 has the
// total): those of lanes 0 .. held - 1.
template <class Sum> __device__ inline Sum fold_lanes(Sum v, unsigned lane, uint32_t held) {
#pragma unroll
  for (unsigned o = 1; o < 32; o <<= 1) {
    const Sum other = shfl_value<Sum, true>(v, o);
    if ((lane & (2 * o - 1)) == 0 && lane + o < held) v = Sum::combine(v, other);
  }
  return v;
}

__device__ inline void prefetch_l2(const void* p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// Walks the units, a warp each.  Block b takes units b, b + blocks, ... (so
// each SM gets its share of the long ones, which come first) and deals them
// to its warps back and forth, which evens their sums out; the deal is fixed,
// so what an epilogue sums does not vary from run to run.  `epi` is
// pull_units': `pre(row)` as a unit starts, `row(...)` once a row, by one
// lane, with a slot for what the row adds to a sum where the row was finished
// by whichever warp came last (a long row of several units: its first carry
// slot, read by then), else NULL.
template <class E, int S, class W, class Epi>
__device__ inline void lane_units(const LaneView<W>& A, const E* __restrict__ x, const E* hot,
                                  Epi& epi, DeviceError* err) {
  constexpr int ADD = semiring_add(S);
  constexpr uint32_t U = 4;  // steps in flight
  constexpr uint32_t G = kWideLanes;
  static_assert(8 % U == 0 && kPieceEntries == 256, "a piece is whole batches of steps");
  typedef typename LaneWeight<W>::type WT;
  typedef EntryOf<E, S, W> Ent;
  typedef Acc<E, ADD> Sum;
  typedef Partial<E, ADD> Part;
  const unsigned lane = threadIdx.x & 31;
  const uint32_t hot_bit = A.hot_count ? kHotTarget : 0u;
  Part* carry = static_cast<Part*>(A.carry);
  auto gather = [&](uint32_t t) {
    E v;
    if (t & hot_bit) v = hot[t ^ kHotTarget];
    else v = load_x(x, t);
    return v;
  };
  // The rows without entries follow the units as slices of no steps.
  const uint32_t all = A.unit_count + (A.shorts - A.filled + 31) / 32;
  // The warp's k-th unit, past the end when there is none.
  // (The units are far fewer than 2^32 / the warps: no product here wraps.)
  const uint32_t warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  auto nth = [&](uint32_t k) -> uint32_t {
    const uint32_t at = k * warps + ((k & 1) ? warps - 1 - warp : warp);
    return at * gridDim.x + blockIdx.x;
  };
  auto load_unit = [&](uint32_t at) {
    uint4 d = make_uint4(0u, 0u, 0u, 0u);
    if (at < A.unit_count) {
      d = __ldg(reinterpret_cast<const uint4*>(A.units) + at);
    } else if (at < all) {
      d.x = A.filled + 32 * (at - A.unit_count);
      d.w = min(32u, A.shorts - d.x) << 8;
    }
    return LaneUnit{d.x, d.y, d.z, d.w};
  };
  // A slice: the lane's row and its entries; a long row: its first entry and
  // its end.
  auto load_row = [&](const LaneUnit& d, uint32_t& r, uint32_t& l) {
    r = l = 0u;
    if (d.d >> 31) {
      r = __ldg(A.off + d.a);
      l = __ldg(A.off + d.a + 1);
      return;
    }
    const uint32_t q = lane >> (d.d & 31u);
    if (q < ((d.d >> 8) & 255u)) {
      r = A.rows ? __ldg(A.rows + d.a + q) : A.first_short + d.a + q;
      if (d.b) l = __ldg(A.lengths + d.a + q);
    }
  };
  // Requests a unit's targets (and weights) into L2: a line a lane.  They
  // stream from DRAM, whose latency the steps in flight do not cover.
  auto prefetch = [&](const LaneUnit& d) {
    const uint32_t lines = d.d >> 31 ? 8 * (d.b & 255u) : d.b;
    for (uint32_t l = lane; l < lines; l += 32) {
      const size_t at = (size_t)d.c * 32 + 32 * l;
      prefetch_l2(A.tgt + at);
      if constexpr (WSize<W>::v >= 4) prefetch_l2(A.w + at);
      if constexpr (WSize<W>::v == 8) prefetch_l2(A.w + at + 16);
    }
  };
  // This unit's descriptor and row, and the next one's descriptor, loading
  // while the last one folds.
  uint32_t u = nth(0), u1 = nth(1);
  LaneUnit unit = load_unit(u), ahead = load_unit(u1);
  uint32_t row = 0, len = 0;
  load_row(unit, row, len);
  for (uint32_t next = 2; u < all; next++) {
    const uint32_t u2 = nth(next);
    const LaneUnit after = load_unit(u2);
    uint32_t row1, len1;
    load_row(ahead, row1, len1);
    prefetch(ahead);
    const bool piece = unit.d >> 31;
    const bool wide = !piece && (unit.d & 31u);
    const uint32_t* tg = A.tgt + (size_t)unit.c * 32 + lane;
    const W* wt = A.w;
    if constexpr (WSize<W>::v != 0) wt += (size_t)unit.c * 32 + lane;
    // The lane's steps.  A slice: one entry a step of the lane's row (of
    // every kWideLanes-th of it where the row has that many lanes).  Pieces
    // [f, f + np) of a long row: eight steps each, entries 8l .. 8l + 7 in
    // lane l, every lane's eight present but in the row's last piece.
    const uint32_t f = (unit.b >> 8) & (piece ? ~0u : 0u), np = unit.b & 255u;
    const uint32_t deg = len - row;  // a long row's
    uint32_t steps, full, mine;
    uint32_t erow = row;
    bool emits;
    if (piece) {
      const uint32_t whole = min(np, deg / kPieceEntries - f);
      steps = 8 * np;
      full = 8 * whole;
      const uint32_t left = deg - (f + whole) * kPieceEntries;  // of a piece that is not whole
      mine = full + (8 * lane < left ? min(8u, left - 8 * lane) : 0u);
      erow = A.rows ? unit.a : __ldg(A.numbers + unit.a);
      emits = lane == 0;
    } else {
      steps = unit.b;
      const uint32_t sub = wide ? lane % G : 0u;
      full = wide ? 0u : (unit.d >> 16) / U * U;
      mine = wide ? (len + G - 1 - sub) / G : len;
      emits = sub == 0 && (lane >> (unit.d & 31u)) < ((unit.d >> 8) & 255u);
    }
    typename Epi::Pre pre{};
    if (emits) pre = epi.pre(erow);
    Sum sum = Sum::of(E{});
    Part keep{Sum::of(E{}), false};  // lane p: piece p's partial
    int32_t bad = 0;
    uint32_t t[U];
    WT wv[U];
    // Steps [k0, k0 + U) of every lane (ALL) or of those that have them.
    auto load = [&](uint32_t k0, bool every) {
#pragma unroll
      for (uint32_t q = 0; q < U; q++) {
        const bool has = every || k0 + q < mine;
        t[q] = has ? __ldcs(tg + 32 * (k0 + q)) : 0u;
        if constexpr (WSize<W>::v != 0) wv[q] = has ? __ldcs(wt + 32 * (k0 + q)) : WT{};
        else wv[q] = WT{};
      }
    };
    auto add = [&](uint32_t k, E p) {
      sum = k == 0 ? Sum::of(p) : Sum::combine(sum, Sum::of(p));
    };
    // A piece's eight steps are in: its tree over the lanes, and on to the next.
    auto close_piece = [&](uint32_t p, uint32_t held) {
      sum = shfl_value(fold_lanes(sum, lane, held), 0u);
      if (lane == p) keep = Part{sum, true};
    };
    if (full) load(0, true);
    uint32_t k0 = 0;
    for (; k0 < full; k0 += U) {
      E xv[U];
      WT wc[U];
#pragma unroll
      for (uint32_t q = 0; q < U; q++) {
        wc[q] = wv[q];
        xv[q] = gather(t[q]);
      }
      if (k0 + U < full) load(k0 + U, true);
      const uint32_t in = piece ? k0 & 7u : k0;
#pragma unroll
      for (uint32_t q = 0; q < U; q++) {
        E p;
        const int32_t s = Ent::product(wc[q], xv[q], &p);
        if (s) bad = s;
        add(in + q, p);
      }
      if (piece && in + U == 8) close_piece(k0 >> 3, 32u);
    }
    for (; k0 < steps; k0 += U) {
      load(k0, false);
      E xv[U];
#pragma unroll
      for (uint32_t q = 0; q < U; q++)
        if (k0 + q < mine) xv[q] = gather(t[q]);
      const uint32_t in = piece ? k0 & 7u : k0;
#pragma unroll
      for (uint32_t q = 0; q < U; q++) {
        E p{};
        if (k0 + q < mine) {
          const int32_t s = Ent::product(wv[q], xv[q], &p);
          if (s) bad = s;
          if (!wide) add(in + q, p);
        }
        if (wide && k0 + q < steps) {
          // The row's G products in order, folded by each of its lanes: the
          // shuffles do not wait for the sum, so a step costs G dependent
          // additions.
#pragma unroll
          for (uint32_t i = 0; i < G; i++) {
            const E pi = shfl_value(p, (lane & ~(G - 1)) | i);
            const uint32_t e = (k0 + q) * G + i;
            if (e < len) add(e, pi);
          }
        }
      }
      if (piece && in + U == 8)
        close_piece(k0 >> 3, (deg - (f + (k0 >> 3)) * kPieceEntries + 7) / 8);
    }
    bool present = len > 0, shared = false;
    if (piece) {
      // The whole row is here (combine_pieces' tree over the lanes), or its
      // partials go to the carry slots and the last unit to arrive combines.
      const uint32_t slot0 = unit.d & 0x7fffffffu;
      const uint32_t pieces = (deg + kPieceEntries - 1) / kPieceEntries;
      present = true;
      if (np == pieces) {
        sum = fold_lanes(keep.acc, lane, np);
      } else {
        if (lane < np) carry[slot0 + f + lane] = keep;
        __syncwarp();
        uint32_t arrived = 0;
        if (lane == 0) arrived = arrive_many(A.counters + slot0, np);
        arrived = __shfl_sync(0xffffffffu, arrived, 0);
        shared = arrived + np == pieces;
        emits = emits && shared;
        if (shared) {
          __threadfence();
          sum = combine_pieces<E, ADD, 1>(carry, slot0, pieces, 0, lane).acc;
          if (lane == 0) A.counters[slot0] = 0;
        }
      }
    }
    if (emits) {
      E out{};
      if (present) {
        const int32_t s = sum.value(&out);
        if (s) bad = s;
      }
      epi.row(erow, present, out, pre, shared ? carry + (unit.d & 0x7fffffffu) : nullptr);
    }
    if (bad) raise(err, bad, erow);
    u = u1;
    u1 = u2;
    unit = ahead;
    ahead = after;
    row = row1;
    len = len1;
  }
}

}  // namespace wc
