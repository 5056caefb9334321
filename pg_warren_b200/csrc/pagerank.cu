// pagerank.cu — wc_pagerank: compute/pagerank/mod.rs:96-287 on the device.
//
// The reference runs, per iteration, `spread` (msg = x / out, the dangling
// rank summed), a plus_times pull over the reverse CSR, and `advance`
// (x ← d·(y + dangling·p) + (1−d)·p with the L1 change), each step's
// arithmetic as SQL float8 does it.  Here one kernel per iteration does all
// three: the pull of row i is followed at once by its advance and by the
// spread of the new x_i into the next iteration's message, so the messages
// are read once and x once per iteration.  The two sums (the L1 change and
// the next dangling rank) are reduced per block and then, by the last block
// to finish, in block order, so results do not vary from run to run.  That
// block also applies the stop test (delta < live × tol in SQL order) and
// raises a device flag on which later iterations return at once, so a
// call's iterations are queued without a round trip per iteration.
//
// Floating-point reassociation: rows of more than 256 entries, and the two
// sums, are added in another order than the reference's sequential folds
// (documented; the ranks stay within 1e-12 relative L1).  The seeded
// personalisation's sum is computed in the reference's own order (65536-
// element chunks folded sequentially, combined in order).
#include "lanes.cuh"
#include "operand.h"
#include "pagerank.h"
#include "pull.cuh"
#include "sqlfloat.cuh"
#include "upload.h"

namespace wc {

constexpr uint64_t kChunk = 1 << 16;  // compute/reduce.rs:20



__device__ inline bool tomb_at(const uint64_t* t, uint32_t i) {
  return t && ((t[i >> 6] >> (i & 63)) & 1);
}

// A fixed-order sum of two values over the block: lanes, then warps in
// order.  The result is in thread 0.
__device__ inline void block_sum_two(double& a, double& b) {
  __shared__ double sa[32], sb[32];
  const unsigned lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_down_sync(0xffffffffu, a, o);
    b += __shfl_down_sync(0xffffffffu, b, o);
  }
  __syncthreads();
  if (lane == 0) {
    sa[wid] = a;
    sb[wid] = b;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double ta = 0.0, tb = 0.0;
    for (unsigned w = 0; w < blockDim.x / 32; w++) {
      ta += sa[w];
      tb += sb[w];
    }
    a = ta;
    b = tb;
  }
}

// Sums two values per thread over the block, then over the blocks' sums
// in the last block to arrive (each of its threads folding a fixed stride
// of them, then the block in fixed order), so the totals do not depend on
// which block arrives last.  Returns true in thread 0 of that block, with
// the totals in a, b.
// `more(a, b)`: what each thread of the last block adds to its run of them.
template <class More>
__device__ inline bool reduce_two(double& a, double& b, double* partials, unsigned* counter,
                                  More more) {
  __shared__ bool last;
  block_sum_two(a, b);
  if (threadIdx.x == 0) {
    partials[2 * blockIdx.x] = a;
    partials[2 * blockIdx.x + 1] = b;
    __threadfence();
    last = atomicAdd(counter, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
  double ta = 0.0, tb = 0.0;
  for (unsigned k = threadIdx.x; k < gridDim.x; k += blockDim.x) {
    ta += __ldcg(partials + 2 * k);
    tb += __ldcg(partials + 2 * k + 1);
  }
  more(ta, tb);
  block_sum_two(ta, tb);
  if (threadIdx.x != 0) return false;
  *counter = 0;
  a = ta;
  b = tb;
  return true;
}
__device__ inline bool reduce_two(double& a, double& b, double* partials, unsigned* counter) {
  return reduce_two(a, b, partials, counter, [](double&, double&) {});
}

// The reference's sum of a seed over live rows (reduce.rs:137-153, 266-279):
// each 65536-element chunk folded sequentially from +0.
// Block c sums chunk c of the live seed values in index order: warps 1..
// stage the next 2,048 terms in shared memory while thread 0 adds the
// current ones.  A tombstoned row's term is +0.0, which leaves a sum that
// starts at +0.0 unchanged, as skipping it does.
constexpr uint32_t kSeedStage = 2048;

__global__ void __launch_bounds__(256) seed_chunks_kernel(const double* seed, const uint64_t* tomb,
                                                          uint64_t n, double* partial) {
  __shared__ double stage[2][kSeedStage];
  const uint64_t c0 = (uint64_t)blockIdx.x * kChunk;
  const uint64_t c1 = min(n, c0 + kChunk);
  const uint32_t rounds = (uint32_t)((c1 - c0 + kSeedStage - 1) / kSeedStage);
  auto fill = [&](uint32_t r, uint32_t first) {
    double* st = stage[r & 1];
    for (uint32_t q = threadIdx.x - first; q < kSeedStage; q += blockDim.x - first) {
      const uint64_t i = c0 + (uint64_t)r * kSeedStage + q;
      st[q] = (i < c1 && !tomb_at(tomb, (uint32_t)i)) ? seed[i] : 0.0;
    }
  };
  double sum = 0.0;
  fill(0, 0);
  __syncthreads();
  for (uint32_t r = 0; r < rounds; r++) {
    if (threadIdx.x == 0) {
      const double* st = stage[r & 1];
#pragma unroll 16
      for (uint32_t q = 0; q < kSeedStage; q++) sum = sum + st[q];
    } else if (threadIdx.x >= 32 && r + 1 < rounds) {
      fill(r + 1, 32);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = sum;
}

__global__ void seed_shares_kernel(const double* seed, const uint64_t* tomb, uint32_t n,
                                   const double* partial, uint32_t chunks, double* shares,
                                   DeviceError* err) {
  // total = 1 / (chunk sums added in chunk order); every thread recomputes
  // the short fold so no second launch is needed.
  double sum = 0.0;
  for (uint32_t c = 0; c < chunks; c++) sum = sum + partial[c];
  double total;
  int32_t s = sql_float<F_DIV>(1.0, sum, &total);
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    if (s) {
      raise(err, s);
      return;
    }
    double share = 0.0;
    if (!tomb_at(tomb, i)) {
      int32_t e = sql_float<F_MUL>(seed[i], total, &share);
      if (e) raise(err, e, i);
    }
    shares[i] = share;
  }
}

__device__ __noinline__ void check_spread(double x, double out, DeviceError* err, uint32_t row) {
  double m;
  const int32_t s = sql_float<F_DIV>(x, out, &m);
  if (s) raise(err, s, row);
}

// spread (mod.rs:204-232) for one row: the message, and the row's dangling
// rank (x where out is not above 0 in SQL order).
__device__ inline double spread_row(double x, double out, double* msg, DeviceError* err,
                                    uint32_t row) {
  if (sql_cmp_f(out, 0.0) > 0) {
    const double m = x / out;
    if (m == 0.0 || !isfinite(m)) check_spread(x, out, err, row);  // what a failing one leaves
    *msg = m;
    return 0.0;
  }
  *msg = 0.0;
  return x;
}

// An unweighted row's out-weight is its entry count (the reference's sum of
// that many ones), taken from the forward offsets here: the sum as a product
// took 350 µs of a 5.9 ms solve on R-MAT 22.
__global__ void pr_init_kernel(PrState s) {
  double none = 0.0, dangling = 0.0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < s.n; i += gridDim.x * blockDim.x) {
    double x = tomb_at(s.tomb, i) ? 0.0 : s.start;
    s.x[0][i] = x;
    double out;
    if (s.degrees) {
      const uint32_t id = __ldg(s.order + i);
      out = (double)(s.degrees[id + 1] - s.degrees[id]);
      s.out[i] = out;
    } else {
      out = s.out[i];
    }
    dangling += spread_row(x, out, &s.msg[0][i], s.err, i);
  }
  if (reduce_two(none, dangling, s.partials, s.counter)) {
    s.dangling[0] = dangling;
    *s.iterations = 0;
    *s.done = 0;
  }
}

// A row's next rank by the reference's checked operations.
__device__ __noinline__ double checked_next(double damping, double teleport, DeviceError* err,
                                            uint32_t i, double y, double p, double dangling_in) {
  double dp, flowed, a, b, next = 0.0;
  int32_t e = sql_float<F_MUL>(dangling_in, p, &dp);
  if (!e) e = sql_float<F_ADD>(y, dp, &flowed);
  if (!e) e = sql_float<F_MUL>(damping, flowed, &a);
  if (!e) e = sql_float<F_MUL>(teleport, p, &b);
  if (!e) e = sql_float<F_ADD>(a, b, &next);
  if (e) raise(err, e, i);
  return next;
}

// advance (mod.rs:245-282) and the next spread, for the row the pull ends.
struct PrEpi {
  const PrState* s;
  int cur;
  double dangling_in;
  double delta = 0.0;
  double dangling_out = 0.0;
  // dangling · start and teleport · start, and whether neither failed.
  double uniform_dp = 0.0, uniform_b = 0.0;
  bool uniform_ok = false;
  bool slots = true;  // whether a row's slot takes what it adds to the sums
  __device__ PrEpi(const PrState* st, int c, double in) : s(st), cur(c), dangling_in(in) {
    uniform_ok = sql_float<F_MUL>(in, st->start, &uniform_dp) == 0 &&
                 sql_float<F_MUL>(st->teleport, st->start, &uniform_b) == 0;
  }
  // The row's operands, requested before its pull so they arrive with it.
  struct Pre {
    double old, out, share;
    bool dead;
  };
  __device__ Pre pre(uint32_t i) const {
    const PrState& st = *s;
    Pre p;
    p.dead = tomb_at(st.tomb, i);
    p.share = st.shares ? st.shares[i] : st.start;
    p.old = st.x[cur][i];
    p.out = st.out[i];
    return p;
  }
  typedef Partial<double, semiring_add(WC_PLUS_TIMES)> Slot;
  // With the uniform personalisation two of the products are the launch's.
  // Every failing operation leaves an infinity, a NaN or a zero product, so
  // only a row that shows one goes through the checked operations.  A row
  // finished by whichever warp came last leaves its share of the sums in its
  // slot, for the last block to add in row order.
  __device__ void row(uint32_t i, bool present, double y, const Pre& pr, Slot* slot = nullptr) {
    const PrState& st = *s;
    if (!present) y = 0.0;  // an empty row writes the plus identity
    const double flowed = st.damping * (y + uniform_dp);
    double next = flowed + uniform_b;
    if (pr.dead)
      next = 0.0;
    else if (st.shares || flowed == 0.0 || !isfinite(next) || !uniform_ok)
      next = checked_next(st.damping, st.teleport, st.err, i, y, pr.share, dangling_in);
    const double change = fabs(next - pr.old);
    st.x[cur ^ 1][i] = next;
    const double dangles = spread_row(next, pr.out, &st.msg[cur ^ 1][i], st.err, i);
    if (slots && slot) {
      static_assert(sizeof(Slot) == sizeof(double2), "a slot holds the row's two sums");
      *reinterpret_cast<double2*>(slot) = make_double2(change, dangles);
    } else {
      delta += change;
      dangling_out += dangles;
    }
  }
};

// The caller's cancel word (host memory, mapped), requested by one thread of
// an iteration as it begins and passed to the device's copy as it ends, so the
// round trip over PCIe runs beside the iteration.
__device__ inline int32_t pr_read_cancel(const PrState& s) {
  return blockIdx.x == 0 && threadIdx.x == 32 ? *(volatile const int32_t*)s.cancel : 0;
}
__device__ inline void pr_pass_cancel(const PrState& s, int32_t cancel) {
  if (blockIdx.x == 0 && threadIdx.x == 32) *(volatile int32_t*)s.cancelled = cancel;
}

// The step's close, by the last block of its last kernel: the stop test,
// the cancel word and the progress words.
__device__ inline void pr_close(const PrState& s, uint32_t it, double delta, double dangling) {
  s.delta[it] = delta;
  s.dangling[it + 1] = dangling;
  *s.iterations = it + 1;
  if (s.has_tol && sql_cmp_f(delta, s.threshold) < 0) *s.done = 1;
  // The caller's cancel word was read once, as the iteration began; the next
  // iteration then returns at once.
  if (*(volatile const int32_t*)s.cancelled) {
    raise(s.err, WC_CANCELLED);
    *s.done = 1;
  }
  // Tell the host how far the solve is, so it stops queueing iterations.
  if (s.pace) {
    *(volatile double*)s.last_delta = delta;
    volatile uint32_t* pace = s.pace;
    pace[1] = *s.done;
    pace[0] = it + 1;
  }
}

// The reverse CSR's lane-major copy with its targets in the sorted numbering:
// a slice's rows are consecutive there, so the epilogue's vectors are read and
// written in runs (by dense id they took 32-byte sectors apiece, which cost
// as much again as the gathers: 702 against 465 µs for the product alone).
template <class W> static LaneView<W> ranked_view(const PullLaunch& L, const wc_version* v) {
  LaneView<W> A = lane_view<W>(L);
  A.rows = nullptr;
  A.first_short = v->rev.schedule.long_rows;
  A.numbers = v->loc.perm.as<uint32_t>();
  A.tgt = v->loc.lane_targets.as<uint32_t>();
  A.hot = v->loc.lane_hot.as<uint32_t>();
  return A;
}

// The rows that several warps' pieces make up, [lo, hi) of `longs` (row, first
// slot, pieces) with more than `run` pieces, left their shares of the sums in
// their slots: each thread of the last block adds some, in row order, four
// loads in flight.
__device__ inline void add_slots(double& a, double& b, const uint4* longs, uint32_t lo,
                                 uint32_t hi, uint32_t run, const PrEpi::Slot* carry) {
  constexpr uint32_t U = 4;
  for (uint64_t r0 = lo + threadIdx.x; r0 < hi; r0 += U * blockDim.x) {
    uint4 L[U];
    double2 v[U];
#pragma unroll
    for (uint32_t q = 0; q < U; q++) {
      const uint64_t r = r0 + q * blockDim.x;
      L[q] = r < hi ? __ldg(longs + r) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (uint32_t q = 0; q < U; q++)
      if (L[q].z > run) v[q] = __ldcg(reinterpret_cast<const double2*>(carry + L[q].y));
#pragma unroll
    for (uint32_t q = 0; q < U; q++)
      if (L[q].z > run) {
        a += v[q].x;
        b += v[q].y;
      }
  }
}

// One iteration over the reverse CSR's lane-major copy: one launch, one
// block an SM.
template <class W>
__global__ void __launch_bounds__(kLaneThreads, 1)
    pr_lane_kernel(LaneView<W> A, PrState s, uint32_t it, const uint4* longs, uint32_t long_count,
                   uint32_t run) {
  extern __shared__ __align__(16) double pr_hot[];
  const int cur = it & 1;
  const int32_t done = *(volatile int32_t*)s.done;
  const int32_t cancel = pr_read_cancel(s);
  PrEpi epi(&s, cur, s.dangling[it]);
  lane_fill_hot<double, W>(A, s.msg[cur], pr_hot);
  if (done) return;
  lane_units<double, WC_PLUS_TIMES, W>(A, s.msg[cur], pr_hot, epi, s.err);
  pr_pass_cancel(s, cancel);
  double delta = epi.delta, dangling = epi.dangling_out;
  auto more = [&](double& a, double& b) {
    add_slots(a, b, longs, 0, long_count, run, static_cast<const PrEpi::Slot*>(A.carry));
  };
  if (reduce_two(delta, dangling, s.partials, s.counter, more)) pr_close(s, it, delta, dangling);
}

// The messages that pr_iter_kernel's gathers keep in L1: 64 KB of them, what
// the SM's L1 holds beside four blocks' staging rings.  They are those of the
// rows numbered first, the longest, which a graph of skewed degrees gathers
// most often as well.
constexpr uint32_t kHotRows = 8192;

// One iteration over the row-split schedule of the CSC in row order
// (solve_lanes_pay says when), or over a range of it (a part of a
// row-partitioned solve, which gives no `longs`: its sums take a row in pieces
// as it comes).  Unweighted, four blocks an SM (64 registers) keep more gathers
// in flight; with weights the extra registers would spill, so three.  Bound by
// the latency of the gathers; with plain loads in place of load_x_split's the
// parts of a weighted R-MAT 22 took 1.05 ms whole and 0.30, 0.32 and 0.37
// (first, second and last quarter), with the split 0.97 and 0.29, 0.30 and
// 0.34 (an unweighted one 0.70 and 0.71 whole).
template <class W>
__global__ void __launch_bounds__(kPullThreads, WSize<W>::v == 0 ? 4 : 3)
    pr_iter_kernel(CsrView<W> A, PrState s, uint32_t it, const uint4* longs, uint32_t long_count) {
  extern __shared__ __align__(16) unsigned char smem[];
  if (*(volatile int32_t*)s.done) return;
  const int32_t cancel = pr_read_cancel(s);
  const int cur = it & 1;
  PrEpi epi(&s, cur, s.dangling[it]);
  epi.slots = longs != nullptr;
  PullRing<double, W>* ring = reinterpret_cast<PullRing<double, W>*>(smem) + (threadIdx.x >> 5);
  pull_units<double, WC_PLUS_TIMES, W, PrEpi, true>(A, s.msg[cur], epi, s.err, ring);
  pr_pass_cancel(s, cancel);
  double delta = epi.delta, dangling = epi.dangling_out;
  auto more = [&](double& a, double& b) {
    add_slots(a, b, longs, 0, long_count, 0, static_cast<const PrEpi::Slot*>(A.carry));
  };
  if (reduce_two(delta, dangling, s.partials, s.counter, more)) pr_close(s, it, delta, dangling);
}

template <class W>
static wc_status launch_iter(const PullLaunch& L, const PrState& s, uint32_t it, uint32_t blocks,
                             const wc_version* v) {
  const Schedule& longs = v->rev.schedule;
  static const cudaError_t attr =
      cudaFuncSetAttribute(pr_lane_kernel<W>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)(kHotSlots * sizeof(double)));
  if (attr != cudaSuccess) return cuda_status(attr, L.detail, "pagerank kernel attributes");
  const LaneView<W> A = ranked_view<W>(L, v);
  note_launch(), pr_lane_kernel<W><<<blocks, kLaneThreads, A.hot_count * sizeof(double),
                                     L.stream>>>(A, s, it, longs.long_list.as<uint4>(),
                                                 longs.long_rows, L.lanes->run);
  return WC_OK;
}

template <class W>
static wc_status launch_rows(const PullLaunch& L, const PrState& s, uint32_t it, uint32_t blocks,
                             const Schedule* longs) {
  CsrView<W> A{L.off, L.tgt, static_cast<const W*>(L.weights), L.units, L.unit_count, L.counters,
               L.carry, kHotRows};
  constexpr size_t smem = pull_smem_bytes<double, W>();
  static const cudaError_t attr = cudaFuncSetAttribute(
      pr_iter_kernel<W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (attr != cudaSuccess) return cuda_status(attr, L.detail, "pagerank kernel attributes");
  note_launch(), pr_iter_kernel<W><<<blocks, kPullThreads, smem, L.stream>>>(
      A, s, it, longs ? longs->long_list.as<uint4>() : nullptr, longs ? longs->long_rows : 0);
  return WC_OK;
}

wc_status prepare_pull(Ctx& ctx, DevCsr& csr, int semiring, int weighted_flag, int dtype,
                       uint32_t width, PullLaunch& L);
wc_status launch_pull(const PullLaunch& L, int dtype, const void* x, void* y);

wc_status launch_pr_init(const PrState& s, uint32_t grid, cudaStream_t stream) {
  note_launch(), pr_init_kernel<<<grid, kPullThreads, 0, stream>>>(s);
  return cuda_status(cudaGetLastError(), nullptr, "pagerank init");
}

wc_status launch_row_iteration(const PullLaunch& L, const PrState& s, uint32_t it, uint32_t blocks,
                               const Schedule* longs) {
  if (L.weight_kind == WEIGHTS_F64) return launch_rows<double>(L, s, it, blocks, longs);
  return launch_rows<void>(L, s, it, blocks, longs);
}

uint64_t live_count(const uint64_t* tomb, uint64_t n) {
  uint64_t dead = 0;
  if (tomb)
    for (uint64_t w = 0; w < (n + 63) / 64; w++) {
      uint64_t word = tomb[w];
      if (w == n / 64 && (n & 63)) word &= (1ull << (n & 63)) - 1;
      dead += __builtin_popcountll(word);
    }
  return n - dead;
}

uint32_t pagerank_grid(const DevCsr& csc) {
  return std::max<uint32_t>(1, std::min<uint32_t>((csc.schedule.count + kPullWarps - 1) / kPullWarps,
                                                  max_blocks(8)));
}

wc_status PageRankRun::setup(Ctx& ctx, const wc_pagerank_opts* o, const uint64_t* tomb_host,
                             const double* seed) {
  wc_version* v = ctx.v;
  const uint64_t n = v->n;
  const uint64_t words = (n + 63) / 64;
  opts = *o;
  // Tombstones: the caller's words, on the device.
  std::vector<uint64_t> host_words;
  const uint64_t* th = tomb_host;
  if (tomb_host && is_device_pointer(tomb_host)) {
    host_words.resize(words);
    WC_CUDA(cudaMemcpy(host_words.data(), tomb_host, words * 8, cudaMemcpyDeviceToHost),
            ctx.detail);
    th = host_words.data();
  }
  live = live_count(th, n);
  nodes = (double)live;
  double start;
  WC_TRY((wc_status)sql_float<F_DIV>(1.0, nodes, &start));
  double teleport;
  WC_TRY((wc_status)sql_float<F_SUB>(1.0, o->damping, &teleport));
  double threshold = 0.0;
  if (o->has_tol && o->max_iter > 0) WC_TRY((wc_status)sql_float<F_MUL>(nodes, o->tol, &threshold));
  grid = pagerank_grid(v->loc.csc);
  WC_TRY(ctx.scratch(POOL_PR_X, 2 * n * 8, &x));
  WC_TRY(ctx.scratch(POOL_PR_MSG, 2 * n * 8, &msg));
  WC_TRY(ctx.scratch(POOL_PR_OUT, n * 8, &out));
  const uint64_t scalar_bytes = (2 * (uint64_t)o->max_iter + 8) * 8 + 2 * (uint64_t)grid * 8 + 64;
  WC_TRY(ctx.scratch(POOL_PR_SCALARS, scalar_bytes, &scalars));
  uint64_t* tomb_dev = nullptr;
  if (th) {
    // The words are renumbered into the buffer's second half.
    WC_TRY(ctx.scratch(POOL_PR_TOMB, words * 8 * 2, &tomb));
    WC_CUDA(cudaMemcpyAsync(tomb->ptr, th, words * 8, cudaMemcpyHostToDevice, ctx.stream),
            ctx.detail);
    tomb_dev = tomb->as<uint64_t>();
    WC_TRY(bits_to_locality(v, ctx.stream, tomb_dev, tomb_dev + words));
    tomb_dev += words;
  }
  WC_CUDA(cudaMemsetAsync(scalars->ptr, 0, scalar_bytes, ctx.stream), ctx.detail);
  double* sc = scalars->as<double>();
  s = PrState{};
  s.n = (uint32_t)n;
  s.x[0] = x->as<double>();
  s.x[1] = x->as<double>() + n;
  s.msg[0] = msg->as<double>();
  s.msg[1] = msg->as<double>() + n;
  s.out = out->as<double>();
  s.tomb = tomb_dev;
  s.start = start;
  s.damping = o->damping;
  s.teleport = teleport;
  s.threshold = threshold;
  s.has_tol = o->has_tol != 0;
  s.delta = sc;
  s.dangling = sc + o->max_iter;
  s.partials = sc + 2 * (uint64_t)o->max_iter + 8;
  unsigned char* tail = reinterpret_cast<unsigned char*>(s.partials + 2 * grid);
  s.counter = reinterpret_cast<unsigned*>(tail);
  s.iterations = reinterpret_cast<uint32_t*>(tail + 8);
  s.done = reinterpret_cast<int32_t*>(tail + 16);
  s.cancel = v->cancel_dev;
  s.cancelled = reinterpret_cast<int32_t*>(tail + 24);
  s.pace = v->pace_dev;
  s.err = v->error.as<DeviceError>();
  s.last_delta = reinterpret_cast<double*>(v->stage_dev + kStagePayload);
  WC_TRY(out_weights(ctx));
  // The personalisation, summed in dense-id order (the reference's chunks).
  if (seed) {
    Operand S(POOL_SEED);
    WC_TRY(S.in(ctx, seed, n * 8));
    const double* sd = static_cast<const double*>(S.dev);
    const uint32_t chunks = (uint32_t)((n + kChunk - 1) / kChunk);
    WC_TRY(ctx.scratch(POOL_PR_SHARES, n * 8 * 2 + (uint64_t)chunks * 8, &shares));
    double* partial = shares->as<double>() + n * 2;
    const uint64_t* tomb_ids = th ? tomb->as<uint64_t>() : nullptr;  // dense-id order
    if (chunks)
      note_launch(), seed_chunks_kernel<<<chunks, 256, 0, ctx.stream>>>(sd, tomb_ids, n, partial);
    note_launch(), seed_shares_kernel<<<max_blocks(4), 256, 0, ctx.stream>>>(sd, tomb_ids, (uint32_t)n, partial,
                                                             chunks, shares->as<double>(), s.err);
    WC_TRY(to_locality(v, ctx.stream, shares->as<double>(), shares->as<double>() + n));
    s.shares = shares->as<double>() + n;
  }
  return cuda_status(cudaGetLastError(), ctx.detail, "pagerank setup");
}

// The out-weights, s.out: plus_first over the forward CSR when weighted
// (renumbered through the second message buffer); when not, the rows' entry
// counts, which pr_init_kernel takes from the offsets.
wc_status PageRankRun::out_weights(Ctx& ctx) {
  wc_version* v = ctx.v;
  if (opts.weighted == 0 || !v->weighted) {
    s.degrees = v->fwd.offsets.as<uint32_t>();
    s.order = v->loc.order.as<uint32_t>();
    return WC_OK;
  }
  PullLaunch L;
  WC_TRY(prepare_pull(ctx, v->fwd, WC_PLUS_FIRST, opts.weighted, WC_F64, 1, L));
  WC_TRY(launch_pull(L, WC_F64, s.x[0], s.msg[1]));
  return to_locality(v, ctx.stream, s.msg[1], s.out);
}

__global__ void out_degrees_kernel(PrState s) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < s.n; i += gridDim.x * blockDim.x) {
    const uint32_t id = __ldg(s.order + i);
    s.out[i] = (double)(s.degrees[id + 1] - s.degrees[id]);
  }
}

wc_status PageRankRun::out_now(Ctx& ctx) {
  if (s.degrees && s.n)
    note_launch(), out_degrees_kernel<<<max_blocks(4), 256, 0, ctx.stream>>>(s);
  return cuda_status(cudaGetLastError(), ctx.detail, "out-degrees");
}

// Whether a solve walks the lane-major copy.  Over a skewed graph (one with
// long rows) of few entries its longest slices are what an iteration waits
// for, and the row-split schedule, whose units are all alike, is the faster.
// Solves to 1e-10 over R-MAT graphs of so many nodes and edges, lanes and
// schedule, µs: 4,096 and 28,700 386 and 271 (weighted 440 and 302), 33,000 and
// 157,396 490 and 326 (511 and 340), 65,536 and 954,361 339 and 334 (366 and
// 383), 131,072 and 999,085 468 and 411 (519 and 486), 262,144 and 1,024,319
// 558 and 506.  In longer rows the schedule holds out further: 65,536 and
// 1,818,513 512 and 397, 131,072 and 1,942,324 541 and 474 (weighted 611 and
// 615), but 262,144 and 2,016,841 554 and 568, 524,288 and 2,057,684 620 and
// 663.  G(n, m) graphs have no long row: 65,536 and 262,129 260 and 290.
bool solve_lanes_pay(const wc_version* v, bool weighted) {
  if (!v->rev.schedule.long_rows) return true;
  return v->m >= (!weighted && v->m >= 12 * v->n ? 1u << 21 : 1u << 20);
}

wc_status PageRankRun::run(Ctx& ctx) {
  wc_version* v = ctx.v;
  WC_TRY(launch_pr_init(s, grid, ctx.stream));
  PullLaunch L;
  WC_TRY(prepare_pull(ctx, v->rev, WC_PLUS_TIMES, opts.weighted, WC_F64, 1, L));
  const bool lanes = v->rev.lanes.targets.ptr && v->loc.lane_targets.ptr &&
                     solve_lanes_pay(v, L.weight_kind == WEIGHTS_F64);
  if (lanes) L.lanes = &v->rev.lanes;
  else WC_TRY(prepare_pull(ctx, v->loc.csc, WC_PLUS_TIMES, opts.weighted, WC_F64, 1, L));
  // No more blocks than the step keeps sums for.
  const uint32_t blocks = lanes ? std::min(lane_grid(L), grid) : grid;
  // With a tolerance the solve usually stops well before max_iter: the
  // host keeps at most kAhead iterations queued beyond the last one the
  // device reported, and stops queueing once the device reports the stop,
  // so few launches return at once on the done flag.
  constexpr uint32_t kAhead = 3;
  volatile uint32_t* pace = s.pace ? v->pace_host : nullptr;
  if (pace) {
    pace[0] = 0;
    pace[1] = 0;
  }
  ctx.phase_begin("iteration");
  for (uint32_t it = 0; it < opts.max_iter; it++) {
    // A cancel stops the queueing (the kernels queued read the device's
    // copy of the word, which finish() raises).
    if (ctx.cancelled()) break;
    if (pace && s.has_tol) {
      bool stop = false;
      while (!(stop = pace[1] != 0) && it >= pace[0] + kAhead) {
        if (ctx.cancelled() || cudaStreamQuery(ctx.stream) != cudaErrorNotReady) break;
        std::this_thread::yield();
      }
      if (stop) break;
    }
    if (!lanes) WC_TRY(launch_row_iteration(L, s, it, blocks, &v->loc.csc.schedule));
    else if (L.weight_kind == WEIGHTS_F64) WC_TRY(launch_iter<double>(L, s, it, blocks, v));
    else WC_TRY(launch_iter<void>(L, s, it, blocks, v));
  }
  ctx.phase_end();
  return cuda_status(cudaGetLastError(), ctx.detail, "pagerank iterations");
}

wc_status PageRankRun::result(Ctx& ctx, double* ranks_dev_or_host, uint32_t* iterations_out,
                              double* margin) {
  // A solve that reported its progress left the count and the last change in
  // mapped memory, complete once finish() has waited.
  uint32_t its = 0;
  if (s.pace) its = ctx.v->pace_host[0];
  else WC_CUDA(cudaMemcpy(&its, s.iterations, 4, cudaMemcpyDeviceToHost), ctx.detail);
  if (opts.max_iter == 0) its = 0;
  const double* final_x = s.x[its & 1];
  // Back to dense-id order, through the other rank buffer (free now).
  WC_TRY(from_locality(ctx.v, ctx.stream, final_x, s.x[(its & 1) ^ 1]));
  final_x = s.x[(its & 1) ^ 1];
  WC_CUDA(cudaMemcpyAsync(ranks_dev_or_host, final_x, ctx.v->n * 8, cudaMemcpyDefault, ctx.stream),
          ctx.detail);
  WC_CUDA(cudaStreamSynchronize(ctx.stream), ctx.detail);
  if (iterations_out) *iterations_out = its;
  if (margin && its > 0) {
    double delta = 0.0;
    if (s.pace) std::memcpy(&delta, ctx.v->stage_host + kStagePayload, 8);
    else WC_CUDA(cudaMemcpy(&delta, s.delta + (its - 1), 8, cudaMemcpyDeviceToHost), ctx.detail);
    *margin = s.threshold != 0.0 ? delta / s.threshold : 0.0;
  }
  return WC_OK;
}

}  // namespace wc

using namespace wc;

extern "C" {

wc_status wc_pagerank(wc_version* v, const wc_call* call, const wc_pagerank_opts* o,
                      const uint64_t* tombstones, double* ranks, uint32_t* iterations) {
  if (!v || !o || !ranks) return WC_INVALID_ARGUMENT;
  std::lock_guard<std::recursive_mutex> lock(v->mu);
  WC_CUDA(cudaSetDevice(v->device), call ? call->detail : nullptr);
  Ctx ctx(v, call);
  if (ctx.cancelled()) return WC_CANCELLED;
  WC_TRY(ctx.begin());
  // The two ways to walk the rows add the solve's sums in orders of their own:
  // a solve does not change the way of the next by what it allocates.
  ctx.keep_lanes = true;
  PageRankRun run;
  ctx.phase_begin("setup");
  WC_TRY(run.setup(ctx, o, tombstones, o->seed));
  ctx.phase_end();
  ctx.progress("iterating", 0, o->max_iter);
  WC_TRY(run.run(ctx));
  WC_TRY(locality_status(ctx, ctx.finish()));
  double margin = 0.0;
  WC_TRY(run.result(ctx, ranks, iterations, &margin));
  v->last_margin = margin;
  ctx.progress("iterating", iterations ? *iterations : 0, o->max_iter);
  return WC_OK;
}

double wc_pagerank_last_margin(const wc_version* v) { return v ? v->last_margin : 0.0; }

}  // extern "C"
