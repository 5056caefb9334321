// locality.cu — a version's reverse CSR in row order, for the solvers that
// keep their per-node vectors in an order of their own (PageRank, the batched
// personalised PageRank).
//
// The nodes are renumbered by the length of their reverse rows, longest first
// (equal lengths in dense-id order): the order in which the lane-major copy
// (lanes.cu) deals rows to lanes, so a slice's 32 rows are 32 consecutive
// values of every vector its epilogue reads and writes.  Row k of the
// renumbered CSC is the reverse row of node order[k] with its entries in
// their stored order and each source renumbered perm[source]; a row's fold
// adds the same products in the same order as over the plain CSC, so each
// row's result is the same bit for bit.  A solver renumbers only at the
// boundary: inputs scattered in, results gathered out.
// (The reference's own locality orders, graph/node_order/, renumber the
// stored graph; this one is internal to the device copy.)
#include <algorithm>
#include <vector>

#include <cub/cub.cuh>

#include "operand.h"
#include "runtime.cuh"
#include "upload.h"

namespace wc {

__global__ void degree_keys_kernel(const uint32_t* off, uint32_t n, uint32_t* keys,
                                   uint32_t* ids) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    keys[i] = ~(off[i + 1] - off[i]);  // ascending keys: longest row first
    ids[i] = i;
  }
}

__global__ void invert_kernel(const uint32_t* order, uint32_t n, uint32_t* perm) {
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x)
    perm[order[k]] = k;
}

// New row k's entry count (the last slot, n, is zero for the scan).
__global__ void loc_degrees_kernel(const uint32_t* order, const uint32_t* roff, uint32_t n,
                                   uint32_t* deg) {
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k <= n; k += gridDim.x * blockDim.x)
    deg[k] = k < n ? roff[order[k] + 1] - roff[order[k]] : 0u;
}

// A warp per new row: the old row's entries in order, sources renumbered.
__global__ void loc_entries_kernel(const uint32_t* order, const uint32_t* perm,
                                   const uint32_t* roff, const uint32_t* rtgt, const double* rw,
                                   const uint32_t* noff, uint32_t n, uint32_t* ntgt, double* nw) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < n; k += warps) {
    const uint32_t r = order[k], a = roff[r], b = roff[r + 1], dst = noff[k];
    for (uint32_t e = a + lane; e < b; e += 32) {
      ntgt[dst + (e - a)] = perm[rtgt[e]];
      if (rw) nw[dst + (e - a)] = rw[e];
    }
  }
}

// The lane-major copy's targets and hot nodes in the new numbers (a hot
// target's slot stays).
__global__ void loc_lanes_kernel(const uint32_t* targets, uint64_t places, const uint32_t* hot,
                                 uint32_t hot_count, const uint32_t* perm, uint32_t* new_targets,
                                 uint32_t* new_hot) {
  const uint64_t first = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const uint32_t hot_bit = hot_count ? kHotTarget : 0u;
  for (uint64_t e = first; e < places; e += stride) {
    const uint32_t t = targets[e];
    new_targets[e] = t & hot_bit ? t : perm[t];
  }
  for (uint64_t h = first; h < hot_count; h += stride) new_hot[h] = perm[hot[h]];
}

static uint32_t grid_of(uint64_t items) {
  return (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(max_blocks(8), (items + 255) / 256));
}

wc_status device_locality(wc_version* v, wc_error_detail* detail) {
  const uint64_t n = v->n, m = v->m;
  cudaStream_t st = v->stream;
  Locality& L = v->loc;
  DevCsr& c = L.csc;
  WC_TRY(L.order.alloc(v->budget, std::max<uint64_t>(n, 1) * 4, detail));
  WC_TRY(L.perm.alloc(v->budget, std::max<uint64_t>(n, 1) * 4, detail));
  WC_TRY(c.offsets.alloc(v->budget, (n + 1) * 4 + kBulkPad, detail));
  WC_TRY(c.targets.alloc(v->budget, m * 4 + kBulkPad, detail));
  if (v->weighted) WC_TRY(c.weights.alloc(v->budget, m * 8 + kBulkPad, detail));
  if (n) {
    // Order: a stable radix sort of (¬length, id).
    DevBuf k0, k1, i1, temp;
    WC_TRY(k0.alloc(v->budget, n * 4, detail));
    WC_TRY(k1.alloc(v->budget, n * 4, detail));
    WC_TRY(i1.alloc(v->budget, n * 4, detail));
    note_launch(), degree_keys_kernel<<<grid_of(n), 256, 0, st>>>(
        v->rev.offsets.as<uint32_t>(), (uint32_t)n, k0.as<uint32_t>(), L.order.as<uint32_t>());
    cub::DoubleBuffer<uint32_t> keys(k0.as<uint32_t>(), k1.as<uint32_t>());
    cub::DoubleBuffer<uint32_t> ids(L.order.as<uint32_t>(), i1.as<uint32_t>());
    size_t temp_bytes = 0;
    WC_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, temp_bytes, keys, ids, (int)n, 0, 32, st),
            detail);
    WC_TRY(temp.alloc(v->budget, std::max<size_t>(temp_bytes, 16), detail));
    WC_CUDA(cub::DeviceRadixSort::SortPairs(temp.ptr, temp_bytes, keys, ids, (int)n, 0, 32, st),
            detail);
    if (ids.Current() != L.order.as<uint32_t>())
      WC_CUDA(cudaMemcpyAsync(L.order.ptr, ids.Current(), n * 4, cudaMemcpyDeviceToDevice, st),
              detail);
    note_launch(), invert_kernel<<<grid_of(n), 256, 0, st>>>(L.order.as<uint32_t>(), (uint32_t)n,
                                                              L.perm.as<uint32_t>());
    // Offsets: the new rows' entry counts, scanned (k1 holds the counts).
    DevBuf counts;
    WC_TRY(counts.alloc(v->budget, (n + 1) * 4, detail));
    note_launch(), loc_degrees_kernel<<<grid_of(n + 1), 256, 0, st>>>(
        L.order.as<uint32_t>(), v->rev.offsets.as<uint32_t>(), (uint32_t)n, counts.as<uint32_t>());
    size_t scan_bytes = 0;
    WC_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, counts.as<uint32_t>(),
                                          c.offsets.as<uint32_t>(), (int)(n + 1), st),
            detail);
    if (scan_bytes > temp.bytes) WC_TRY(temp.alloc(v->budget, scan_bytes, detail));
    WC_CUDA(cub::DeviceScan::ExclusiveSum(temp.ptr, scan_bytes, counts.as<uint32_t>(),
                                          c.offsets.as<uint32_t>(), (int)(n + 1), st),
            detail);
    if (m)
      note_launch(), loc_entries_kernel<<<max_blocks(8), 256, 0, st>>>(
          L.order.as<uint32_t>(), L.perm.as<uint32_t>(), v->rev.offsets.as<uint32_t>(),
          v->rev.targets.as<uint32_t>(), v->weighted ? v->rev.weights.as<double>() : nullptr,
          c.offsets.as<uint32_t>(), (uint32_t)n, c.targets.as<uint32_t>(),
          c.weights.as<double>());
    WC_CUDA(cudaStreamSynchronize(st), detail);  // before the transient buffers go
  } else {
    WC_CUDA(cudaMemsetAsync(c.offsets.ptr, 0, 4, st), detail);
  }
  std::vector<uint32_t> off32(n + 1);
  WC_CUDA(cudaMemcpyAsync(off32.data(), c.offsets.ptr, (n + 1) * 4, cudaMemcpyDeviceToHost, st),
          detail);
  WC_CUDA(cudaStreamSynchronize(st), detail);
  std::vector<uint64_t> off(off32.begin(), off32.end());
  WC_TRY(put_schedule(v, c, off, detail));
  return cuda_status(cudaGetLastError(), detail, "locality order");
}

wc_status device_lane_numbers(wc_version* v, uint64_t& room, wc_error_detail* detail) {
  const LaneCsr& lanes = v->rev.lanes;
  Locality& L = v->loc;
  if (!lanes.places) return WC_OK;  // no copy, or no nodes
  const uint64_t bytes = (lanes.places + lanes.hot_count) * 4;
  if (bytes > room) return WC_OUT_OF_MEMORY;
  WC_TRY(L.lane_targets.alloc(v->budget, lanes.places * 4, detail, Room{false}));
  if (lanes.hot_count)
    WC_TRY(L.lane_hot.alloc(v->budget, lanes.hot_count * 4, detail, Room{false}));
  room -= bytes;
  if (v->n)
    note_launch(), loc_lanes_kernel<<<grid_of(lanes.places), 256, 0, v->stream>>>(
        lanes.targets.as<uint32_t>(), lanes.places, lanes.hot.as<uint32_t>(), lanes.hot_count,
        L.perm.as<uint32_t>(), L.lane_targets.as<uint32_t>(), L.lane_hot.as<uint32_t>());
  return cuda_status(cudaStreamSynchronize(v->stream), detail, "lane-major numbers");
}

// ------------------------------------------------- renumbering vectors

__global__ void scatter_f64_kernel(const double* src, const uint32_t* perm, uint32_t n,
                                   double* dst) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    dst[perm[i]] = src[i];
}

__global__ void gather_f64_kernel(const double* src, const uint32_t* perm, uint32_t n,
                                  double* dst) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    dst[i] = src[perm[i]];
}

__global__ void scatter_bits_kernel(const uint64_t* bits, const uint32_t* perm, uint32_t n,
                                    uint64_t* out) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    if ((bits[i >> 6] >> (i & 63)) & 1) {
      const uint32_t k = perm[i];
      atomicOr(reinterpret_cast<unsigned long long*>(out + (k >> 6)), 1ull << (k & 63));
    }
}

wc_status to_locality(const wc_version* v, cudaStream_t st, const double* src, double* dst) {
  if (v->n)
    note_launch(), scatter_f64_kernel<<<grid_of(v->n), 256, 0, st>>>(
        src, v->loc.perm.as<uint32_t>(), (uint32_t)v->n, dst);
  return cuda_status(cudaGetLastError(), nullptr, "renumber in");
}

wc_status from_locality(const wc_version* v, cudaStream_t st, const double* src, double* dst) {
  if (v->n)
    note_launch(), gather_f64_kernel<<<grid_of(v->n), 256, 0, st>>>(
        src, v->loc.perm.as<uint32_t>(), (uint32_t)v->n, dst);
  return cuda_status(cudaGetLastError(), nullptr, "renumber out");
}

wc_status bits_to_locality(const wc_version* v, cudaStream_t st, const uint64_t* src,
                           uint64_t* dst) {
  const uint64_t words = (v->n + 63) / 64;
  WC_CUDA(cudaMemsetAsync(dst, 0, words * 8, st), nullptr);
  if (v->n)
    note_launch(), scatter_bits_kernel<<<grid_of(v->n), 256, 0, st>>>(
        src, v->loc.perm.as<uint32_t>(), (uint32_t)v->n, dst);
  return cuda_status(cudaGetLastError(), nullptr, "renumber bits");
}

wc_status locality_status(Ctx& ctx, wc_status st) {
  if (st == WC_OK || !ctx.device_error || !ctx.detail || ctx.detail->node >= ctx.v->n) return st;
  uint32_t id = 0;
  if (cudaMemcpy(&id, ctx.v->loc.order.as<uint32_t>() + ctx.detail->node, 4,
                 cudaMemcpyDeviceToHost) == cudaSuccess)
    ctx.detail->node = id;
  return st;
}

}  // namespace wc
