// lanes.cu — builds a version's lane-major copies (LaneCsr): each
// orientation's entries laid out so that a warp's lanes walk the rows they
// fold.
//
// The row-major CSR suits kernels that take a row with a warp.  A product
// over one vector does not: a row's fold is sequential (the reference's
// order), so the entries had to be moved from the lanes that gathered them
// to the lane that folds the row, which cost more instructions than the
// gathers themselves.  Here the rows of at most kPieceEntries entries are
// sorted by length and cut into slices: 32 rows of up to 32 entries with a
// lane each, entry k of lane l at base + 32k + l, so a step of the folds
// reads one 128-byte run of targets and nothing is moved.  In a graph too
// small to keep every warp busy past its longest slice, longer rows get
// kWideLanes lanes (entry k of a row in its lane k mod 8) that gather side by
// side and all fold: a fold costs more so, but a slice is shorter.  A row over
// kPieceEntries is cut into the row-split schedule's pieces (256 entries,
// eight consecutive ones a lane), laid out likewise, a few of them a unit.
//
// The nodes gathered most often get slots in a table that each block copies
// to shared memory before it walks (lanes.cuh); their targets are stored as
// kHotTarget | slot.
#include <algorithm>
#include <vector>

#include <cub/cub.cuh>

#include "lanes.h"
#include "operand.h"
#include "runtime.cuh"
#include "upload.h"

namespace wc {

// A node earns a slot when each SM would gather it at least twice (148 SMs):
// filling its slot costs every block one gather.
constexpr uint64_t kHotGathers = 296;

static uint32_t grid_of(uint64_t items) {
  return (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(max_blocks(8), (items + 255) / 256));
}

// Sort keys: short rows by length, longest first; the long rows last.
__global__ void lane_keys_kernel(const uint32_t* off, uint32_t n, uint32_t* keys, uint32_t* ids) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint32_t deg = off[i + 1] - off[i];
    keys[i] = deg > kPieceEntries ? kPieceEntries + 1 : kPieceEntries - deg;
    ids[i] = i;
  }
}

__global__ void gather_keys_kernel(const uint32_t* off, uint32_t n, uint32_t* keys, uint32_t* ids) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    keys[i] = ~(off[i + 1] - off[i]);  // ascending keys: most gathered first
    ids[i] = i;
  }
}

// The slices of rows with kWideLanes lanes, then of those with one: class c
// holds rows [row[c], row[c + 1]) of the sorted order in slices [slice[c],
// slice[c + 1]).
struct LaneClasses {
  uint32_t row[3], slice[3];
};

__global__ void lane_lengths_kernel(const uint32_t* off, const uint32_t* rows, uint32_t shorts,
                                    uint16_t* lengths) {
  for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < shorts; q += gridDim.x * blockDim.x)
    lengths[q] = (uint16_t)(off[rows[q] + 1] - off[rows[q]]);
}

// Each slice's unit, its base left for the scan of the steps.
__global__ void lane_slices_kernel(LaneClasses c, const uint16_t* lengths, LaneUnit* units,
                                   uint32_t* steps) {
  for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < c.slice[2];
       s += gridDim.x * blockDim.x) {
    const uint32_t q = s >= c.slice[1];
    const uint32_t lg = q ? 0u : 3u, per = 32 >> lg;
    const uint32_t a = c.row[q] + (s - c.slice[q]) * per;
    const uint32_t count = min(per, c.row[q + 1] - a);
    const uint32_t st = ((uint32_t)lengths[a] + (1u << lg) - 1) >> lg;  // the longest row's
    const uint32_t least = count < per ? 0u : (uint32_t)lengths[a + count - 1] >> lg;
    steps[s] = st;
    units[s] = LaneUnit{a, st, 0u, lg | count << 8 | least << 16};
  }
}

__global__ void lane_bases_kernel(const uint32_t* bases, uint32_t slices, uint32_t first,
                                  LaneUnit* units) {
  for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < slices; s += gridDim.x * blockDim.x)
    units[s].c = first + bases[s];
}

// Over the nodes: rows of more than `cap` entries (the long ones apart), rows
// without entries, and nodes gathered often enough for a slot.
__global__ void lane_counts_kernel(const uint32_t* off, const uint32_t* other, uint32_t n,
                                   uint32_t cap, uint32_t* counts) {
  uint32_t wide = 0, empty = 0, hot = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint32_t deg = off[i + 1] - off[i];
    wide += deg > cap && deg <= kPieceEntries;
    empty += deg == 0;
    hot += other[i + 1] - other[i] >= kHotGathers;
  }
  wide = __reduce_add_sync(0xffffffffu, wide);
  empty = __reduce_add_sync(0xffffffffu, empty);
  hot = __reduce_add_sync(0xffffffffu, hot);
  if ((threadIdx.x & 31) == 0) {
    if (wide) atomicAdd(counts, wide);
    if (empty) atomicAdd(counts + 1, empty);
    if (hot) atomicAdd(counts + 2, hot);
  }
}

__global__ void hot_slots_kernel(const uint32_t* hot, uint32_t count, uint32_t* slot_of) {
  const uint32_t h = blockIdx.x * blockDim.x + threadIdx.x;
  if (h < count) slot_of[hot[h]] = kHotTarget | h;
}

// A warp per unit: its lanes' entries to their places.  `slot_of` (NULL: no
// hot nodes) holds a hot node's stored target, 0 for the others.
__global__ void lane_entries_kernel(const LaneUnit* units, uint32_t count, const uint32_t* rows,
                                    const uint16_t* lengths, const uint32_t* off,
                                    const uint32_t* tgt, const double* w, const int32_t* wi,
                                    const uint32_t* slot_of, uint32_t* ltgt, double* lw,
                                    int32_t* lwi) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  auto put = [&](size_t to, uint32_t e) {
    uint32_t t = tgt[e];
    if (slot_of) {
      const uint32_t h = slot_of[t];
      if (h) t = h;
    }
    ltgt[to] = t;
    if (lw) lw[to] = w[e];
    if (lwi) lwi[to] = wi[e];
  };
  for (uint32_t u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; u < count; u += warps) {
    const LaneUnit d = units[u];
    const size_t base = (size_t)d.c * 32;
    if (!(d.d >> 31)) {
      const uint32_t lg = d.d & 255, g = 1u << lg, r = lane >> lg;
      if (r >= ((d.d >> 8) & 255)) continue;
      const uint32_t e0 = off[rows[d.a + r]], len = lengths[d.a + r];
      for (uint32_t k = lane & (g - 1); k < len; k += g) put(base + 32 * (k >> lg) + lane, e0 + k);
    } else {
      const uint32_t e0 = off[d.a], deg = off[d.a + 1] - e0;
      const uint32_t f = d.b >> 8, np = d.b & 255;
      for (uint32_t p = 0; p < np; p++)
        for (uint32_t q = 0; q < 8; q++) {
          const uint32_t k = (f + p) * kPieceEntries + 8 * lane + q;
          if (k < deg) put(base + p * kPieceEntries + 32 * q + lane, e0 + k);
        }
    }
  }
}

wc_status device_lanes(wc_version* v, DevCsr& d, const std::vector<uint64_t>& off,
                       const DevCsr& other, uint64_t& room, wc_error_detail* detail) {
  const uint64_t n = v->n, m = v->m;
  cudaStream_t st = v->stream;
  const Room ask{false};  // no other version's copies for these
  LaneCsr& L = d.lanes;
  const uint32_t shorts = (uint32_t)n - d.schedule.long_rows;
  // Rows by width, the hot nodes, and the long rows' units: runs of pieces,
  // each piece a place of kPieceEntries entries.
  const uint32_t run = std::max<uint32_t>(
      1, std::min<uint32_t>(kGroupPieces, d.schedule.slots / kGroupSpread));
  L.run = run;
  // A slice's steps at most: half the steps a warp gets in all, so that one
  // slice cannot be what the last warp is busy with.
  uint64_t cap = 32;
  while (cap < kPieceEntries && m / 32 >= 2 * (2 * cap) * kLaneWarps) cap *= 2;
  std::vector<LaneUnit> groups;
  std::vector<uint4> longs(d.schedule.long_rows);  // row, first slot, pieces
  uint32_t counts[3] = {0, 0, 0};
  DevBuf tally;
  WC_TRY(tally.alloc(v->budget, sizeof counts, detail, ask));
  WC_CUDA(cudaMemsetAsync(tally.ptr, 0, sizeof counts, st), detail);
  if (n)
    note_launch(), lane_counts_kernel<<<grid_of(n), 256, 0, st>>>(
        d.offsets.as<uint32_t>(), other.offsets.as<uint32_t>(), (uint32_t)n, (uint32_t)cap,
        tally.as<uint32_t>());
  WC_CUDA(cudaMemcpyAsync(counts, tally.ptr, sizeof counts, cudaMemcpyDeviceToHost, st), detail);
  if (!longs.empty())
    WC_CUDA(cudaMemcpyAsync(longs.data(), d.schedule.long_list.ptr, longs.size() * sizeof(uint4),
                            cudaMemcpyDeviceToHost, st), detail);
  WC_CUDA(cudaStreamSynchronize(st), detail);
  uint64_t long_entries = 0;
  const uint32_t slot = d.schedule.slots;
  for (const uint4& l : longs) {
    long_entries += off[l.x + 1] - off[l.x];
    for (uint32_t f = 0; f < l.z; f += run)
      groups.push_back(LaneUnit{l.x, f << 8 | std::min(run, l.z - f),
                                (l.y + f) * (kPieceEntries / 32), 1u << 31 | l.y});
  }
  LaneClasses cls{};
  const uint64_t hot_nodes = counts[2];
  cls.row[1] = counts[0];
  cls.row[2] = L.filled = shorts - counts[1];
  L.shorts = shorts;
  for (uint32_t q = 0; q < 2; q++) {
    const uint32_t per = q ? 32 : 32 / kWideLanes;
    cls.slice[q + 1] = cls.slice[q] + (cls.row[q + 1] - cls.row[q] + per - 1) / per;
  }
  const uint32_t slices = cls.slice[2];
  const uint32_t first = slot * (kPieceEntries / 32);  // the slices' entries follow
  L.groups = (uint32_t)groups.size();
  L.count = L.groups + slices;
  // A slice ends at its longest row, at most the shortest of the slice
  // before, so a class wastes at most one slice's entries, and less than a
  // step a slice where a row's lanes do not come out even.
  const uint64_t places = L.places =
      (uint64_t)first * 32 + (m - long_entries) + 32 * cap + 1024 + 32 * (uint64_t)cls.slice[1];
  L.hot_count = n < kHotTarget ? (uint32_t)std::min<uint64_t>(hot_nodes, kHotSlots) : 0;
  const uint64_t bytes = L.count * sizeof(LaneUnit) + n * 4 + shorts * 2ull +
                         places * (4 + (d.weights.ptr ? 8 : 0) + (d.iweights.ptr ? 4 : 0));
  if (bytes > room) return WC_OUT_OF_MEMORY;
  room -= bytes;
  WC_TRY(L.units.alloc(v->budget, std::max<uint64_t>(L.count, 1) * sizeof(LaneUnit), detail, ask));
  WC_TRY(L.rows.alloc(v->budget, std::max<uint64_t>(n, 1) * 4, detail, ask));
  WC_TRY(L.lengths.alloc(v->budget, std::max<uint32_t>(shorts, 1) * 2, detail, ask));
  WC_TRY(L.targets.alloc(v->budget, places * 4, detail, ask));
  if (d.weights.ptr) WC_TRY(L.weights.alloc(v->budget, places * 8, detail, ask));
  if (d.iweights.ptr) WC_TRY(L.iweights.alloc(v->budget, places * 4, detail, ask));
  if (L.hot_count) WC_TRY(L.hot.alloc(v->budget, L.hot_count * 4, detail, ask));
  if (!n) return WC_OK;
  // One transient buffer: two key and two id buffers of n words, the sorts'
  // and the scan's temporary memory behind them.  (The rows are sorted into
  // place by a copy.)
  size_t sort_bytes = 0, scan_bytes = 0;
  {
    cub::DoubleBuffer<uint32_t> none(nullptr, nullptr);
    uint32_t* nowhere = nullptr;
    WC_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, none, none, (int)n, 0, 32, st),
            detail);
    WC_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, nowhere, nowhere, (int)slices, st),
            detail);
  }
  const uint64_t words = (n + 63) / 64 * 64, ids_at = 2 * words;
  const uint64_t temp_at = (ids_at + std::max<uint64_t>(words, 2 * slices) + 63) / 64 * 64;
  size_t temp_bytes = std::max<size_t>({sort_bytes, scan_bytes, 16});
  DevBuf transient;
  WC_TRY(transient.alloc(v->budget, temp_at * 4 + temp_bytes, detail, ask));
  uint32_t* k0 = transient.as<uint32_t>();
  uint32_t* ids = k0 + ids_at;
  void* temp = k0 + temp_at;
  cub::DoubleBuffer<uint32_t> kb(k0, k0 + words);
  cub::DoubleBuffer<uint32_t> ib(L.rows.as<uint32_t>(), ids);
  // The hot nodes: the front of the nodes sorted by gathers.
  uint32_t* slot_of = nullptr;
  if (L.hot_count) {
    note_launch(), gather_keys_kernel<<<grid_of(n), 256, 0, st>>>(
        other.offsets.as<uint32_t>(), (uint32_t)n, kb.Current(), ib.Current());
    WC_CUDA(cub::DeviceRadixSort::SortPairs(temp, temp_bytes, kb, ib, (int)n, 0, 32, st),
            detail);
    WC_CUDA(cudaMemcpyAsync(L.hot.ptr, ib.Current(), L.hot_count * 4, cudaMemcpyDeviceToDevice, st),
            detail);
  }
  // The short rows, longest first.
  note_launch(), lane_keys_kernel<<<grid_of(n), 256, 0, st>>>(
      d.offsets.as<uint32_t>(), (uint32_t)n, kb.Current(), ib.Current());
  WC_CUDA(cub::DeviceRadixSort::SortPairs(temp, temp_bytes, kb, ib, (int)n, 0, 9, st), detail);
  if (ib.Current() != L.rows.as<uint32_t>())
    WC_CUDA(cudaMemcpyAsync(L.rows.ptr, ib.Current(), n * 4, cudaMemcpyDeviceToDevice, st), detail);
  if (!groups.empty())
    WC_CUDA(cudaMemcpyAsync(L.units.ptr, groups.data(), groups.size() * sizeof(LaneUnit),
                            cudaMemcpyHostToDevice, st), detail);
  if (slices) {
    uint32_t *steps = ids, *bases = steps + slices;
    LaneUnit* units = L.units.as<LaneUnit>() + groups.size();
    note_launch(), lane_lengths_kernel<<<grid_of(shorts), 256, 0, st>>>(
        d.offsets.as<uint32_t>(), L.rows.as<uint32_t>(), shorts, L.lengths.as<uint16_t>());
    note_launch(), lane_slices_kernel<<<grid_of(slices), 256, 0, st>>>(
        cls, L.lengths.as<uint16_t>(), units, steps);
    WC_CUDA(cub::DeviceScan::ExclusiveSum(temp, temp_bytes, steps, bases, (int)slices, st),
            detail);
    note_launch(), lane_bases_kernel<<<grid_of(slices), 256, 0, st>>>(bases, slices, first, units);
  }
  if (L.hot_count) {
    slot_of = k0;
    WC_CUDA(cudaMemsetAsync(slot_of, 0, n * 4, st), detail);
    note_launch(), hot_slots_kernel<<<(L.hot_count + 255) / 256, 256, 0, st>>>(
        L.hot.as<uint32_t>(), L.hot_count, slot_of);
  }
  WC_CUDA(cudaMemsetAsync(L.targets.ptr, 0, places * 4, st), detail);
  if (m)
    note_launch(), lane_entries_kernel<<<max_blocks(8), 256, 0, st>>>(
        L.units.as<LaneUnit>(), L.count, L.rows.as<uint32_t>(), L.lengths.as<uint16_t>(),
        d.offsets.as<uint32_t>(), d.targets.as<uint32_t>(), d.weights.as<double>(),
        d.iweights.as<int32_t>(), slot_of, L.targets.as<uint32_t>(), L.weights.as<double>(),
        L.iweights.as<int32_t>());
  WC_CUDA(cudaGetLastError(), detail);
  // Before the transient buffers and the host's units go.
  return cuda_status(cudaStreamSynchronize(st), detail, "lane-major copy");
}

}  // namespace wc
