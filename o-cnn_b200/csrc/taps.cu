// Tap plan: the non-empty nodes of octree levels ordered by which of their 27 neighbours exist.
//
// On the non-empty nodes of a scene a node has 2.4 (depth 9) to 12 (depth 5) of 27 neighbours, but 128 nodes
// in Morton order have all 27 between them, so a convolution tile walks every tap: products of zeros and
// weight tiles fetched for them.  Sorted by the set of taps they have, 128 nodes share 7 (depth 9), 12 (depth 8)
// or 16 taps (200 k points), and the convolution (conv_taps.cuh) walks only those.
//
// The sort key is the Gray rank of the 26-bit neighbour set with corners above edges above faces (neighbours in
// that order differ by few taps: 4.8 / 10.6 taps a tile in full order, 5.1 / 11.3 without the Gray code, 5.2 /
// 14.6 with faces on top).  The order need not be exact: nodes are binned by the key's upper 13 bits over the
// whole level and sorted in full in windows of 2048 (6.9 / 12.4 taps).  Which of several equal places a node
// takes is left to atomics: a node's result does not depend on it, only on the node's own rows.
//
// Four launches for all levels together (115 us for the five levels of a U-Net on 200 k points, 254 k sibling groups
// and 443 k nodes; with 34 of its convolutions on the plan the pass is 0.85 ms shorter, plan included), each bound by latency and scattered 4-byte reads of L2: keys and
// histogram (a sibling group's 64 neighbours are read once for its up to eight nodes), binning,
// window sort, tables.  The tables hold the gathered rows' indices per tile and present tap, in the order in
// which the convolution's threads read them.
#include "taps.cuh"

namespace ocnn {
namespace {

constexpr int kLevels = 8;               // levels per call
constexpr int kBinBits = 13, kBins = 1 << kBinBits, kLowBits = 26 - kBinBits;
constexpr int kWindow = 2048;
constexpr int kKeyThreads = 256, kGroupsPerBlock = 128;
constexpr int kBinThreads = 256, kBinChunk = 2048;
constexpr int kSortThreads = 512;

struct PlanLevel {
  const int* neigh;
  const int* child;
  int groups, rows;
  int at;                                // first slot in the arrays over all levels (a multiple of kWindow)
  int key_block, bin_block, sort_block, tile_block;   // first block of each launch
  int* order;
  uint32_t* mask;
  int* table;
};
struct PlanArgs {
  PlanLevel level[kLevels];
  int levels;
  int* hist;                             // [levels][kBins]
  int* cursor;                           // [levels][kBins]
  uint32_t* key;                         // by slot: the level's nodes in rank order
  int* node;
  uint32_t* key2;                        // binned
  int* node2;
};

template <int PlanLevel::*FIRST>
__device__ __forceinline__ int level_of(const PlanArgs& a, int block) {
  int l = 0;
  while (l + 1 < a.levels && block >= a.level[l + 1].*FIRST) ++l;
  return l;
}

// Position of the key's bit for tap t (tap = 9x + 3y + z, the centre has none): corners 18..25, edges 6..17, faces 0..5.
__host__ __device__ constexpr int tap_class(int t) {
  return (t / 9 != 1) + ((t / 3) % 3 != 1) + (t % 3 != 1);
}
__host__ __device__ constexpr int key_bit(int t) {
  int below = 0;
  for (int u = 0; u < 27; ++u)
    if (u != 13 && (tap_class(u) < tap_class(t) || (tap_class(u) == tap_class(t) && u > t))) ++below;
  return below;
}
struct BitTable { signed char bit[27]; };
constexpr BitTable make_bits() {
  BitTable b = {};
  for (int t = 0; t < 27; ++t) b.bit[t] = t == 13 ? -1 : (signed char)key_bit(t);
  return b;
}
__constant__ BitTable kBit = make_bits();

// A warp takes four sibling groups at a time: lane l < 32 stands for two positions of each group's 4x4x4
// neighbour block in the look-ups, and for node l & 7 of group l >> 3 after them.
__global__ void __launch_bounds__(kKeyThreads) tap_key_kernel(const __grid_constant__ PlanArgs a) {
  __shared__ int hist[kBins];
  __shared__ uint32_t slab[3][512];      // key bits of the nine taps at x = 0, 1, 2
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int i = tid; i < kBins / 4; i += kKeyThreads) reinterpret_cast<int4*>(hist)[i] = make_int4(0, 0, 0, 0);
  for (int i = tid; i < 3 * 512; i += kKeyThreads) {
    uint32_t bits = 0;
    for (int j = 0; j < 9; ++j) {
      const int bit = kBit.bit[(i >> 9) * 9 + j];
      if (((i >> j) & 1) && bit >= 0) bits |= 1u << bit;
    }
    slab[i >> 9][i & 511] = bits;
  }
  const int l = level_of<&PlanLevel::key_block>(a, blockIdx.x);
  const PlanLevel& lv = a.level[l];
  grid_dependency_wait();
  __syncthreads();
  const int g0 = (blockIdx.x - lv.key_block) * kGroupsPerBlock;
  const int g1 = min(g0 + kGroupsPerBlock, lv.groups);
  constexpr int kAhead = 4;
  const int o = lane & 7, u_own = lane >> 3;
  const int shift = ((o & 4) << 2) | ((o & 2) << 1) | (o & 1);       // where the octant's 3x3x3 window starts
  for (int g = g0 + warp * kAhead; g < g1; g += kKeyThreads / 32 * kAhead) {
    int n[kAhead][2];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const bool in = g + u < g1;
      n[u][0] = in ? lv.neigh[((long long)(g + u) << 6) + lane] : -1;
      n[u][1] = in ? lv.neigh[((long long)(g + u) << 6) + 32 + lane] : -1;
    }
    const int rank = g + u_own < g1 ? lv.child[8 * g + lane] : -1;   // of this lane's node
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      if (n[u][0] >= 0) n[u][0] = lv.child[n[u][0]];
      if (n[u][1] >= 0) n[u][1] = lv.child[n[u][1]];
    }
    uint32_t lo = 0, hi = 0;
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const uint32_t b0 = __ballot_sync(0xffffffffu, n[u][0] >= 0), b1 = __ballot_sync(0xffffffffu, n[u][1] >= 0);
      if (u == u_own) { lo = b0; hi = b1; }
    }
    const unsigned long long window = (((unsigned long long)hi << 32) | lo) >> shift;
    uint32_t set = 0;
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      const uint32_t v = (uint32_t)(window >> (16 * x));                       // rows of four, three of each
      set |= slab[x][(v & 7u) | ((v >> 1) & 0x38u) | ((v >> 2) & 0x1c0u)];
    }
    uint32_t gray = set;                                                       // Gray rank: prefix XOR from the top
    gray ^= gray >> 1; gray ^= gray >> 2; gray ^= gray >> 4; gray ^= gray >> 8; gray ^= gray >> 16;
    if (rank >= 0 && rank < lv.rows) {
      a.key[lv.at + rank] = gray;
      a.node[lv.at + rank] = 8 * g + lane;
      atomicAdd(&hist[gray >> kLowBits], 1);
    }
  }
  __syncthreads();
  for (int i = tid; i < kBins; i += kKeyThreads)
    if (hist[i]) atomicAdd(a.hist + l * kBins + i, hist[i]);
  grid_dependency_trigger();    // at the end: the successor's blocks should not sit on SM slots early
}

// (clamped here and below: a node count in the header that the child array does not bear out leaves keys unwritten)
__device__ __forceinline__ int bin_of(uint32_t key) { return min((int)(key >> kLowBits), kBins - 1); }

__global__ void __launch_bounds__(kBinThreads) tap_bin_kernel(const __grid_constant__ PlanArgs a) {
  extern __shared__ int bin_smem[];
  int* first = bin_smem;                 // [kBins] first slot of a bin, then of this block's share of it
  int* count = bin_smem + kBins;         // [kBins] this block's
  __shared__ int warp_sum[kBinThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int kPer = kBins / kBinThreads;
  for (int i = tid; i < kBins; i += kBinThreads) count[i] = 0;
  const int l = level_of<&PlanLevel::bin_block>(a, blockIdx.x);
  const PlanLevel& lv = a.level[l];
  grid_dependency_wait();
  // every block scans the level's histogram for itself: 32 KB from L2 against a launch of its own
  int v[kPer], sum = 0;
#pragma unroll
  for (int q = 0; q < kPer; q += 4) {
    const int4 h = *reinterpret_cast<const int4*>(a.hist + l * kBins + tid * kPer + q);
    v[q] = h.x; v[q + 1] = h.y; v[q + 2] = h.z; v[q + 3] = h.w;
  }
#pragma unroll
  for (int q = 0; q < kPer; ++q) { const int t = v[q]; v[q] = sum; sum += t; }
  int inc = sum;
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) warp_sum[warp] = inc;
  __syncthreads();
  int base = inc - sum;
  for (int w = 0; w < warp; ++w) base += warp_sum[w];
#pragma unroll
  for (int q = 0; q < kPer; ++q) first[tid * kPer + q] = base + v[q];
  // this block's nodes
  const int i0 = (blockIdx.x - lv.bin_block) * kBinChunk;
  constexpr int kItems = kBinChunk / kBinThreads;
  uint32_t key[kItems];
  int node[kItems], rank[kItems];
#pragma unroll
  for (int u = 0; u < kItems; ++u) {
    const int i = i0 + u * kBinThreads + tid;
    key[u] = i < lv.rows ? a.key[lv.at + i] : 0xffffffffu;
    node[u] = i < lv.rows ? a.node[lv.at + i] : 0;
  }
#pragma unroll
  for (int u = 0; u < kItems; ++u)
    rank[u] = key[u] != 0xffffffffu ? atomicAdd(&count[bin_of(key[u])], 1) : -1;
  __syncthreads();
  for (int i = tid; i < kBins; i += kBinThreads)
    if (count[i]) first[i] += atomicAdd(a.cursor + l * kBins + i, count[i]);
  __syncthreads();
#pragma unroll
  for (int u = 0; u < kItems; ++u) {
    if (rank[u] < 0) continue;
    const int to = lv.at + min(first[bin_of(key[u])] + rank[u], lv.rows - 1);
    a.key2[to] = key[u];
    a.node2[to] = node[u];
  }
  grid_dependency_trigger();
}

// Bitonic sort of a window, four neighbouring elements a thread: strides 1 and 2 in registers, up to 64 by
// shuffles, the ten steps beyond a warp's 128 elements through shared memory.
__device__ __forceinline__ void order_pair(unsigned long long& a, unsigned long long& b, bool up) {
  const unsigned long long lo = a < b ? a : b, hi = a < b ? b : a;
  a = up ? lo : hi;
  b = up ? hi : lo;
}
__global__ void __launch_bounds__(kSortThreads) tap_sort_kernel(const __grid_constant__ PlanArgs a) {
  static_assert(kWindow == 4 * kSortThreads, "four elements a thread");
  __shared__ unsigned long long s[kWindow];
  const int tid = threadIdx.x, lane = tid & 31;
  const PlanLevel& lv = a.level[level_of<&PlanLevel::sort_block>(a, blockIdx.x)];
  const int w0 = (blockIdx.x - lv.sort_block) * kWindow;
  grid_dependency_wait();
  unsigned long long e[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int i = w0 + 4 * tid + q;
    e[q] = i < lv.rows ? ((unsigned long long)a.key2[lv.at + i] << 32) | (uint32_t)a.node2[lv.at + i] : ~0ull;
  }
#pragma unroll 1
  for (int k = 2; k <= kWindow; k <<= 1) {
#pragma unroll 1
    for (int j = k >> 1; j > 0; j >>= 1) {
      if (j >= 128) {
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 4; ++q) s[q * kSortThreads + tid] = e[q];        // element 4 tid + q
        __syncthreads();
        const int other = tid ^ (j >> 2);
        const bool up = ((4 * tid) & k) == 0, lower = (tid & (j >> 2)) == 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const unsigned long long o = s[q * kSortThreads + other];
          e[q] = (lower == up) == (o < e[q]) ? o : e[q];
        }
      } else if (j >= 4) {
        const bool up = ((4 * tid) & k) == 0, lower = (lane & (j >> 2)) == 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const unsigned long long o = __shfl_xor_sync(0xffffffffu, e[q], j >> 2);
          e[q] = (lower == up) == (o < e[q]) ? o : e[q];
        }
      } else if (j == 2) {
        order_pair(e[0], e[2], ((4 * tid) & k) == 0);
        order_pair(e[1], e[3], ((4 * tid) & k) == 0);
      } else {
        order_pair(e[0], e[1], ((4 * tid) & k) == 0);
        order_pair(e[2], e[3], ((4 * tid + 2) & k) == 0);
      }
    }
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int i = w0 + 4 * tid + q;
    if (i < lv.rows) a.node[lv.at + i] = (int)(uint32_t)e[q];
  }
  grid_dependency_trigger();
}

__global__ void __launch_bounds__(kTapTile) tap_table_kernel(const __grid_constant__ PlanArgs a) {
  __shared__ uint32_t warp_mask[kTapTile / 32];
  const int tid = threadIdx.x;
  const PlanLevel& lv = a.level[level_of<&PlanLevel::tile_block>(a, blockIdx.x)];
  const int tile = blockIdx.x - lv.tile_block, row = tile * kTapTile + tid;
  grid_dependency_wait();
  const bool live = row < lv.rows;
  const int h = live ? max(0, min(a.node[lv.at + row], 8 * lv.groups - 1)) : 0;
  const int* block = lv.neigh + ((long long)(h >> 3) << 6) + (((h & 4) << 2) | ((h & 2) << 1) | (h & 1));
  int p[27];
  uint32_t set = 0;
#pragma unroll
  for (int t = 0; t < 27; ++t) p[t] = live ? block[((t / 9) << 4) | (((t / 3) % 3) << 2) | (t % 3)] : -1;
#pragma unroll
  for (int t = 0; t < 27; ++t)
    if (p[t] >= 0) p[t] = lv.child[p[t]];
#pragma unroll
  for (int t = 0; t < 27; ++t) set |= (uint32_t)(p[t] >= 0) << t;
  set = __reduce_or_sync(0xffffffffu, set);
  if ((tid & 31) == 0) warp_mask[tid >> 5] = set;
  __syncthreads();
  set = warp_mask[0] | warp_mask[1] | warp_mask[2] | warp_mask[3];
  lv.order[row] = live ? p[13] : -1;
  if (tid == 0) lv.mask[tile] = set;
  int* out = lv.table + (long long)tile * (27 * kTapTile) + tap_slot(tid);
  int j = 0;
#pragma unroll
  for (int t = 0; t < 27; ++t)
    if ((set >> t) & 1u) out[(j++) * kTapTile] = p[t];
  grid_dependency_trigger();
}

size_t round_up(size_t v, size_t to) { return (v + to - 1) / to * to; }

struct PlanWork {
  size_t slots, bytes;
};
PlanWork plan_work(const ocnn_tap_level* levels, int count) {
  PlanWork w = {0, 0};
  for (int l = 0; l < count; ++l) w.slots += round_up((size_t)levels[l].rows, kWindow);
  w.bytes = (size_t)count * kBins * 8 + w.slots * 16;
  return w;
}

}  // namespace

TapPlanView tap_plan_view(const void* plan, int rows) {
  TapPlanView v;
  v.tiles = ceil_div(rows, kTapTile);
  v.order = static_cast<const int*>(plan);
  v.mask = reinterpret_cast<const uint32_t*>(v.order + (size_t)v.tiles * kTapTile);
  v.table = v.order + (size_t)v.tiles * kTapTile + round_up((size_t)v.tiles, 32);
  return v;
}

}  // namespace ocnn

extern "C" {

size_t ocnn_tap_plan_bytes(int rows) {
  using namespace ocnn;
  if (rows <= 0) return 0;
  const size_t tiles = ceil_div(rows, kTapTile);
  return 4 * (tiles * kTapTile + round_up(tiles, 32) + tiles * 27 * kTapTile);
}

size_t ocnn_tap_plan_workspace_bytes(const ocnn_tap_level* levels, int count) {
  using namespace ocnn;
  if (levels == nullptr || count <= 0) return 0;
  return plan_work(levels, count).bytes;
}

int ocnn_tap_plan(const ocnn_tap_level* levels, int count, void* workspace, size_t workspace_bytes, void* stream) {
  using namespace ocnn;
  OCNN_REQUIRE(levels != nullptr && count > 0 && count <= kLevels, "ocnn_tap_plan: 1 to %d levels (got %d)", kLevels,
               count);
  const PlanWork w = plan_work(levels, count);
  OCNN_REQUIRE(workspace != nullptr && workspace_bytes >= w.bytes && (uintptr_t)workspace % 16 == 0,
               "ocnn_tap_plan: the workspace needs %zu bytes on a 16-byte boundary", w.bytes);
  OCNN_REQUIRE(w.slots < (1u << 31), "ocnn_tap_plan: %zu nodes are too many", w.slots);
  PlanArgs a = {};
  int at = 0, key_blocks = 0, bin_blocks = 0, sort_blocks = 0, tiles = 0;
  for (int l = 0; l < count; ++l) {
    const ocnn_tap_level& in = levels[l];
    OCNN_REQUIRE(in.neigh_dev && in.child_dev && in.plan_dev && in.rows > 0 && in.nodes > 0 && in.nodes % 8 == 0,
                 "ocnn_tap_plan: level %d: null pointer, no rows or a node count (%d) that is no multiple of 8", l,
                 in.nodes);
    OCNN_REQUIRE((uintptr_t)in.plan_dev % 32 == 0, "ocnn_tap_plan: plans lie on 32-byte boundaries");
    PlanLevel& lv = a.level[l];
    lv.neigh = in.neigh_dev; lv.child = in.child_dev;
    lv.groups = in.nodes / 8; lv.rows = in.rows; lv.at = at;
    lv.key_block = key_blocks; lv.bin_block = bin_blocks; lv.sort_block = sort_blocks; lv.tile_block = tiles;
    const TapPlanView v = tap_plan_view(in.plan_dev, in.rows);
    lv.order = const_cast<int*>(v.order);
    lv.mask = const_cast<uint32_t*>(v.mask);
    lv.table = const_cast<int*>(v.table);
    at += (int)round_up((size_t)in.rows, kWindow);
    key_blocks += ceil_div(lv.groups, kGroupsPerBlock);
    bin_blocks += ceil_div(in.rows, kBinChunk);
    sort_blocks += ceil_div(in.rows, kWindow);
    tiles += v.tiles;
  }
  a.levels = count;
  a.hist = static_cast<int*>(workspace);
  a.cursor = a.hist + (size_t)count * kBins;
  a.key = reinterpret_cast<uint32_t*>(a.cursor + (size_t)count * kBins);
  a.node = reinterpret_cast<int*>(a.key + w.slots);
  a.key2 = reinterpret_cast<uint32_t*>(a.node + w.slots);
  a.node2 = reinterpret_cast<int*>(a.key2 + w.slots);
  static PerDeviceOnce attr_once;
  const int limits = attr_once.run([&]() -> int {
    OCNN_CUDA_OK(cudaFuncSetAttribute(tap_bin_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 8 * kBins));
    return OCNN_OK;
  });
  if (limits != OCNN_OK) return limits;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  OCNN_CUDA_OK(cudaMemsetAsync(workspace, 0, (size_t)count * kBins * 8, st));
  OCNN_CUDA_OK(launch_chained(tap_key_kernel, dim3(key_blocks), dim3(kKeyThreads), 0, st, a));
  OCNN_CUDA_OK(launch_chained(tap_bin_kernel, dim3(bin_blocks), dim3(kBinThreads), 8 * kBins, st, a));
  OCNN_CUDA_OK(launch_chained(tap_sort_kernel, dim3(sort_blocks), dim3(kSortThreads), 0, st, a));
  OCNN_CUDA_OK(launch_chained(tap_table_kernel, dim3(tiles), dim3(kTapTile), 0, st, a));
  OCNN_LAUNCHES_OK("tap plan", 4);
  return OCNN_OK;
}

}  // extern "C"
