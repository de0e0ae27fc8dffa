// The tap plan of a level (taps.cu writes it, conv_taps.cuh reads it).
#pragma once

#include "common.cuh"

namespace ocnn {

constexpr int kTapTile = 128;             // nodes per tile

// order[tile * 128 + r]: the row (rank among the non-empty nodes) that tile row r stands for, -1: none.
// mask[tile]: bit t is set where a row of the tile has a neighbour at tap t = 9x + 3y + z.
// table[(tile * 27 + j) * 128 + tap_slot(r)]: row r's neighbour at the j-th set tap, -1: none.
struct TapPlanView {
  const int* order;
  const uint32_t* mask;
  const int* table;
  int tiles;
};
TapPlanView tap_plan_view(const void* plan, int rows);

// A gather thread copies rows k, k + 4, ... of its warp's 32: their entries lie next to each other.
__host__ __device__ __forceinline__ int tap_slot(int r) { return (r & ~31) + ((r & 3) << 3) + ((r >> 2) & 7); }

}  // namespace ocnn
