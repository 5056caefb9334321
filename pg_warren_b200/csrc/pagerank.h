// pagerank.h — the state of one PageRank solve on the device, shared by
// wc_pagerank, the batched personalised PageRank and the adjoint.
#pragma once

#include "product.h"
#include "runtime.cuh"

namespace wc {

struct PrState {
  uint32_t n;
  double* x[2];
  double* msg[2];
  double* out;
  const uint32_t* degrees;  // unweighted: the forward offsets pr_init takes `out` from
  const uint32_t* order;    //   by the rows' dense ids; else NULL
  const double* shares;  // NULL: uniform, `start` at every live row
  const uint64_t* tomb;
  double start, damping, teleport, threshold;
  bool has_tol;
  double* delta;     // per iteration
  double* dangling;  // per iteration (+1)
  double* partials;  // 2 per block
  unsigned* counter;
  uint32_t* iterations;
  int32_t* done;
  const int32_t* cancel;  // the caller's word, host-mapped
  int32_t* cancelled;     // what an iteration read there as it began
  uint32_t* pace;  // host-mapped: [0] iterations done, [1] stopped
  double* last_delta;  // host-mapped: the last iteration's change (with `pace`)
  DeviceError* err;
};

struct PageRankRun {
  wc_pagerank_opts opts;
  uint64_t live = 0;
  double nodes = 0.0;
  uint32_t grid = 1;
  // The vectors are numbered as the version's CSC in row order (v->loc):
  // setup renumbers its inputs in and result the ranks out.
  DevBuf *x = nullptr, *msg = nullptr, *out = nullptr, *shares = nullptr, *tomb = nullptr,
         *scalars = nullptr;
  PrState s;

  wc_status setup(Ctx& ctx, const wc_pagerank_opts* o, const uint64_t* tomb_host,
                  const double* seed);
  wc_status out_weights(Ctx& ctx);
  // s.out by itself, for a caller that does not run pr_init_kernel.
  wc_status out_now(Ctx& ctx);
  wc_status run(Ctx& ctx);
  wc_status result(Ctx& ctx, double* ranks, uint32_t* iterations, double* margin);
};

// Whether a solve walks the reverse lane-major copy, where it is there.
bool solve_lanes_pay(const wc_version* v, bool weighted);
uint64_t live_count(const uint64_t* tomb, uint64_t n);
// pr_init_kernel: the start vector, its messages and dangling rank.
wc_status launch_pr_init(const PrState& s, uint32_t grid, cudaStream_t stream);
// One iteration (pr_iter_kernel) over L's units; `longs`, for all of them: the
// schedule's long rows, whose shares of the sums are then added in row order.
struct PullLaunch;
wc_status launch_row_iteration(const PullLaunch& L, const PrState& s, uint32_t it, uint32_t blocks,
                               const Schedule* longs);
// Drops a version's partitioned solve (wc_pagerank_part_*) when it is released.
void pagerank_part_forget(const wc_version* v);
// The row-partitioned search's and product's state kept with a version
// (bfs_part.cu), dropped when the version is released.
void bfs_part_forget(const wc_version* v);
// Blocks of an iteration launch over `csc` at the most, each with a block sum.
uint32_t pagerank_grid(const DevCsr& csc);

}  // namespace wc
