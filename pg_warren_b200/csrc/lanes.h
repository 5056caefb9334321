// lanes.h — the constants of the lane-major layout that its builder and its
// walkers share.
#pragma once

#include <cstdint>

namespace wc {

// Pieces of one long row that a unit takes at most (a warp folds them
// without leaving registers; a row of no more pieces needs no carry at all):
// the version's pieces over kGroupSpread (16 warps an SM), so that a small
// graph's long rows spread over the chip.
constexpr uint32_t kGroupPieces = 8;
constexpr uint32_t kGroupSpread = 2368;
// The warps that walk a lane-major copy: 24 an SM, 148 SMs.
constexpr uint32_t kLaneWarps = 3552;
// The lanes of a row longer than a version's slices are (lanes.cu).
constexpr uint32_t kWideLanes = 8;
// Slots of the shared-memory table of hot values: 64 KB of 8-byte elements.
// The rest of an SM's 256 KB is the L1 that the other gathers' lines wait in:
// 16,384 slots are level on PageRank and 2% slower on R-MAT 22's weighted
// product, 22,528 take 5% and 21% longer.
constexpr uint32_t kHotSlots = 8192;

}  // namespace wc
