// points -> octree on the device, for a whole batch of clouds at once.
//
// What the reference does per cloud on one CPU core (Octree::build, octree/octree/octree.cpp:74-121)
// and then per batch (merge_octrees, octree/octree/merge_octrees.cpp:7-198) is done here in one
// pass over all clouds: every point gets the composite key  (cloud << 3*depth) | morton(cell), the
// clouds' own key bits are radix-sorted (the clouds already lie one behind the other, so the sort is
// segmented by cloud and never looks at the cloud bits, unless there are many small clouds: by_cloud; equal
// to the reference's std::sort of (key, index) pairs per cloud), and every level is a segmented "unique" of the
// sorted keys.
// The composite key of a level-d node is also its rank basis: ranks in the batch-wide unique list
// are exactly the rebased child indices that merge_octrees produces.
//
// Phase 1 (plan) leaves in the workspace, for d = full..depth, the sorted unique composite keys
// Kd of the non-empty nodes and, for each such node, where its children (or its points, at the
// finest level) start in the list below.  The per-level counts reach the host through a mapped
// word; the caller allocates the exact output.  Phase 2 (emit) writes header, keys, children, split
// labels, finest-level signal and — for a merged batch — the neighbour table.
//
// All scans are reduce-then-scan over a fixed grid (no inter-block waiting anywhere).
// This file is compiled with --fmad=false: the signal must round exactly like the reference's
// separate multiplies and adds (octree.cpp:330-348).
//
// A small cloud's keys, sort and unique are one launch (small_build_kernel).  A depth-6 batch is 15 launches and a memset: encode + first histogram, two sort passes of 9 bits (five
// launches), count and compact for all levels at once, averages, emit, five for the neighbour tables.  (A
// count and a compact launch per level, a sort over the cloud bits too and separate header / table copies
// made it 29, most of them shorter than their launch.)
#include <cstring>
#include <vector>

#include "header.h"

namespace ocnn {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kScanItems = 4;
constexpr int kScanTile = kThreads * kScanItems;
constexpr int kMaxScanGrid = kSMs * 4;   // 592 blocks: 4 CTAs of 256 threads per SM
constexpr int kSortItems = 8;            // keys per thread per sort tile
constexpr int kSortTile = kThreads * kSortItems;   // 2048 keys

// One entry per cloud (plus a sentinel holding the totals).
struct CloudRef {
  const float* xyz;
  const float* normal;
  const float* feat;
  const float* label;
  long long offset;     // index of the cloud's first point in the batch-wide numbering
  int chunk0;           // first sort chunk (= sort CTA) of the cloud: a chunk never crosses clouds
  int pad;
};
constexpr int kCloudPoints = 7000;       // see by_cloud
constexpr int kInlineClouds = 63;        // a table of this many clouds rides in the launch parameters

// ---- workspace layout --------------------------------------------------------------------------
struct Layout {
  int64_t n;            // total points
  int batch, depth, full;
  int key_bytes;        // 4 or 8: width of the composite keys
  int segments;         // of the sort: the clouds, or 1 (by_cloud)
  int radix_bits, passes;
  int max_chunks;       // sort: bound on the number of chunks, whatever the clouds' sizes
  int64_t cap[OCNN_MAX_DEPTH + 1];   // capacity of Kd
  size_t off_clouds, off_counts, off_bintot, off_blockcnt, off_hist, off_avg;
  size_t zero_bytes;    // counts + digit totals, cleared together
  size_t off_keys[2], off_idx[2];
  size_t off_K[OCNN_MAX_DEPTH + 1], off_start[OCNN_MAX_DEPTH + 2];
  size_t total;
};

size_t align_up(size_t v, size_t a = 256) { return (v + a - 1) / a * a; }

int bits_for(int64_t v) {  // number of bits needed to represent values 0..v-1
  int b = 0;
  while ((1LL << b) < v) ++b;
  return b;
}

// Points per sort chunk: one tile until the batch has four tiles per SM, several tiles then.
int chunk_points(int64_t n) {
  const int64_t tiles = (n + kSortTile - 1) / kSortTile;
  const int64_t per = (tiles + kSMs * 4 - 1) / (kSMs * 4);
  return (int)((per < 1 ? 1 : per) * kSortTile);
}

// Whether the sort runs cloud by cloud or over the whole batch, cloud bits and all.  By cloud saves the passes
// over the cloud bits, but every cloud costs a chunk, a digit row per warp and its digit totals, whatever
// it holds, so the cost of many small clouds has no bound: 60000 clouds of 8 points at depth 6 took 21 ms and
// cleared 246 MB of totals; over the whole batch 3.5 ms.  Measured at depths 5 to 8 (us, by cloud /
// over the batch): 65 clouds of 200 to 32000 points 102 / 116 to 631 / 659, by cloud at nearly every size; 128
// of 500 140 / 127; 256 of 1000 224 / 188, of 6000 498 / 467, of 8000 302 / 311 and 566 / 564, of 12000 364 / 384; 512 of
// 1000 385 / 296; 1024 of 2000 945 / 787.
bool by_cloud(int64_t n, int batch) { return batch <= 64 || n >= (int64_t)batch * kCloudPoints; }

Layout make_layout(int64_t n, int batch, int depth, int full) {
  Layout L;
  memset(&L, 0, sizeof(L));
  L.n = n; L.batch = batch; L.depth = depth; L.full = full;
  L.key_bytes = (3 * depth + bits_for(batch) <= 32) ? 4 : 8;
  L.segments = by_cloud(n, batch) ? batch : 1;
  const int bits = 3 * depth + (L.segments == batch ? 0 : bits_for(batch));
  // 9-bit digits where they save a pass over 8-bit ones (depth 6: two passes instead of three,
  // depth 9: three instead of four)
  const int p8 = (bits + 7) / 8, p9 = (bits + 8) / 9;
  L.radix_bits = p9 < p8 ? 9 : 8;
  L.passes = p9 < p8 ? p9 : p8;
  const int bins = 1 << L.radix_bits;
  // (a bound that grows with n although the chunks do too, so that the workspace of n points serves fewer)
  L.max_chunks = (int)(n / kSortTile < kSMs * 4 ? n / kSortTile : kSMs * 4) + L.segments;
  size_t o = 0;
  auto take = [&](size_t bytes) { size_t at = o; o = align_up(o + bytes); return at; };
  L.off_clouds = take(sizeof(CloudRef) * (size_t)(batch + 3));    // the clouds, then the one segment of all of them
  L.off_counts = take(sizeof(int) * 32);
  L.off_bintot = take(sizeof(int) * (size_t)bins * L.segments * L.passes);   // digit totals per pass and segment
  L.zero_bytes = o - L.off_counts;
  L.off_blockcnt = take(sizeof(int) * kMaxScanGrid * (OCNN_MAX_DEPTH + 1));
  L.off_hist = take(sizeof(int) * (size_t)bins * L.max_chunks);
  for (int i = 0; i < 2; ++i) L.off_keys[i] = take((size_t)L.key_bytes * (size_t)n);
  for (int i = 0; i < 2; ++i) L.off_idx[i] = take(sizeof(uint32_t) * (size_t)n);
  for (int d = full; d <= depth; ++d) {
    int64_t full_nodes = d >= 20 ? INT64_MAX : (int64_t)batch << (3 * d);
    L.cap[d] = n < full_nodes ? n : full_nodes;
    L.off_K[d] = take((size_t)L.key_bytes * (size_t)L.cap[d]);
    // start[d][a]: first entry, in the list below Kd (K(d+1), or the sorted points for d = depth),
    // that belongs to node a of Kd
    L.off_start[d] = take(sizeof(int) * (size_t)(L.cap[d] + 1));
  }
  L.off_avg = take(3 * sizeof(float) * (size_t)L.cap[depth]);   // averaged normals of the finest nodes
  L.total = o;
  return L;
}

// ---- Morton -------------------------------------------------------------------------------------
// bit i of v -> bit 3i for v < 2^21 (octree/octree/octree_nn.cpp:551-560 interleaves x,y,z so)
__device__ __forceinline__ uint64_t spread3(uint32_t v) {
  uint64_t x = v & 0x1fffffu;
  x = (x | (x << 32)) & 0x001f00000000ffffULL;
  x = (x | (x << 16)) & 0x001f0000ff0000ffULL;
  x = (x | (x << 8)) & 0x100f00f00f00f00fULL;
  x = (x | (x << 4)) & 0x10c30c30c30c30c3ULL;
  x = (x | (x << 2)) & 0x1249249249249249ULL;
  return x;
}

// A table of the sort's segments has the form of the table of clouds: first point and first chunk of each, and a
// sentinel.  It is that table where the sort runs cloud by cloud.

// The segment that sort chunk `chunk` belongs to.
__device__ __forceinline__ int segment_of_chunk(const CloudRef* clouds, int batch, int chunk) {
  int lo = 0, hi = batch;          // clouds[lo].chunk0 <= chunk < clouds[hi].chunk0
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (clouds[mid].chunk0 <= chunk) lo = mid; else hi = mid;
  }
  return lo;
}

// The cloud that point i belongs to, between clouds lo and hi.
__device__ __forceinline__ int cloud_of_point(const CloudRef* clouds, int lo, int hi, long long i) {
  while (hi > lo) {                // clouds[lo].offset <= i < clouds[hi + 1].offset
    const int mid = (lo + hi + 1) >> 1;
    if (clouds[mid].offset <= i) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// One chunk of one segment: its points, and where its digit counts go (hist holds, segment by segment, a
// [digit][chunk of the segment] table).
struct Chunk {
  int segment, first, chunks;      // segment, index inside it, the segment's number of chunks
  long long beg, end;
};
__device__ __forceinline__ Chunk chunk_of(const CloudRef* clouds, int batch, int chunk_pts) {
  Chunk c;
  c.segment = segment_of_chunk(clouds, batch, blockIdx.x);
  const CloudRef a = clouds[c.segment];
  const long long next = clouds[c.segment + 1].offset;
  c.first = (int)blockIdx.x - a.chunk0;
  c.chunks = clouds[c.segment + 1].chunk0 - a.chunk0;
  c.beg = a.offset + (long long)c.first * chunk_pts;
  c.end = c.beg + chunk_pts < next ? c.beg + chunk_pts : next;
  return c;
}

// Per-warp digit counters of a CTA, summed and published: hist gets the chunk's counts, bintot the
// segment's totals (integer additions: their order does not matter).
template <int RB>
__device__ __forceinline__ void publish_counts(int (&sh)[kWarps][1 << RB], const Chunk& c, int chunk0,
                                               int* __restrict__ hist, int* __restrict__ bintot) {
  constexpr int kBins = 1 << RB;
  __syncthreads();
  int* to = hist + (long long)chunk0 * kBins + c.first;
#pragma unroll
  for (int d = threadIdx.x; d < kBins; d += kThreads) {
    int total = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) total += sh[w][d];
    to[(long long)d * c.chunks] = total;
    if (total) atomicAdd(&bintot[c.segment * kBins + d], total);
  }
}

// Adds one digit per lane to the warp's counters. Keys that are close in memory often share the
// digit: a run of equal digits in consecutive lanes is added once, by its first lane.  Lanes without
// a key pass `none`, which no counter has.
__device__ __forceinline__ void count_digit(int* counters, int digit, int none) {
  const int lane = threadIdx.x & 31;
  const int prev = __shfl_up_sync(0xffffffffu, digit, 1);
  const bool head = lane == 0 || prev != digit;
  const unsigned heads = __ballot_sync(0xffffffffu, head);
  if (head && digit != none) {
    const unsigned later = lane == 31 ? 0u : (heads >> (lane + 1));
    atomicAdd(&counters[digit], later ? __ffs(later) : 32 - lane);
  }
}

struct EncodeArgs {
  const CloudRef* table;    // device table (written by this kernel when the clouds ride along)
  const CloudRef* segments; // WHOLE: the one segment
  int inline_clouds;        // 1: `clouds` holds them
  int batch, depth, chunk_pts;
  float bbmin[3];
  float mul;
  CloudRef clouds[kInlineClouds + 1];
};

// normalize_pts + sort_keys' key computation (octree.cpp:155-170, 180-186): cell = trunc((p -
// bbmin) * mul), only `depth` bits per axis enter the key.
__device__ __forceinline__ uint64_t cell_key(const EncodeArgs& a, const float (&p)[3], uint64_t top) {
  const uint32_t mask = (1u << a.depth) - 1u;
  uint32_t cell[3];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const float s = (p[j] - a.bbmin[j]) * a.mul;
    cell[j] = (uint32_t)s & mask;
  }
  return top | (spread3(cell[0]) << 2) | (spread3(cell[1]) << 1) | spread3(cell[2]);
}

// One CTA per sort chunk, whose cloud is the
// CTA's (WHOLE: each of its points is looked up among the chunk's clouds); the first sort pass's digits are
// counted on the way.
template <typename KeyT, int RB, bool WHOLE>
__global__ void __launch_bounds__(kThreads) encode_kernel(const __grid_constant__ EncodeArgs a,
                                                          KeyT* __restrict__ keys, int* __restrict__ hist,
                                                          int* __restrict__ bintot) {
  __shared__ int sh[kWarps][1 << RB];
  for (int d = threadIdx.x; d < (1 << RB); d += kThreads)
#pragma unroll
    for (int w = 0; w < kWarps; ++w) sh[w][d] = 0;
  grid_dependency_wait();       // launched as a programmatic dependent: see common.cuh
  const CloudRef* clouds = a.inline_clouds ? a.clouds : a.table;
  if (a.inline_clouds && blockIdx.x == 0)
    for (int i = threadIdx.x; i <= a.batch; i += kThreads) const_cast<CloudRef*>(a.table)[i] = a.clouds[i];
  const Chunk c = WHOLE ? chunk_of(a.segments, 1, a.chunk_pts) : chunk_of(clouds, a.batch, a.chunk_pts);
  __shared__ int range[2];      // WHOLE: the chunk's first and last cloud
  if (WHOLE && (threadIdx.x & 31) == 0 && threadIdx.x < 64)
    range[threadIdx.x >> 5] = cloud_of_point(clouds, 0, a.batch - 1, threadIdx.x == 0 ? c.beg : c.end - 1);
  const float* xyz = WHOLE ? nullptr : clouds[c.segment].xyz - 3 * clouds[c.segment].offset;
  uint64_t top = (uint64_t)c.segment << (3 * a.depth);
  __syncthreads();
  for (long long i0 = c.beg; i0 < c.end; i0 += 4 * kThreads) {
    float p[4][3];
    int cloud[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long long i = i0 + u * kThreads + threadIdx.x;
      const float* from = xyz;
      if (WHOLE && i < c.end) {
        cloud[u] = cloud_of_point(clouds, range[0], range[1], i);
        from = clouds[cloud[u]].xyz - 3 * clouds[cloud[u]].offset;
      }
#pragma unroll
      for (int j = 0; j < 3; ++j) p[u][j] = i < c.end ? from[3 * i + j] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long long i = i0 + u * kThreads + threadIdx.x;
      if (WHOLE) top = i < c.end ? (uint64_t)cloud[u] << (3 * a.depth) : 0;
      // (with the cloud's bits: the top digit of a shallow tree reaches into them, here as in the scatter)
      const uint64_t key = cell_key(a, p[u], top);
      if (i < c.end) keys[i] = (KeyT)key;
      count_digit(sh[threadIdx.x >> 5], i < c.end ? (int)(key & ((1 << RB) - 1)) : (1 << RB), 1 << RB);
    }
  }
  publish_counts<RB>(sh, c, WHOLE ? 0 : clouds[c.segment].chunk0, hist, bintot);
  grid_dependency_trigger();    // at the end: the successor's blocks should not sit on SM slots early
}

// ---- stable LSD radix sort, RB bits per pass, by segments (the clouds, or the batch: by_cloud) ---------
// Each CTA owns one chunk of one segment.  A pass is: per-CTA digit histogram -> exclusive scan over
// (digit, chunk) inside the segment -> stable scatter.  The scatter works in tiles of 2048 keys: every
// warp ranks its 256 keys 32 at a time with ballots (stable inside the warp), the per-warp digit counts
// are prefixed across warps and digits, the tile is written to shared memory in digit order, and
// only then copied out — consecutive threads then write consecutive global addresses of one digit
// run, so the 4-byte scatter of the naive formulation becomes coalesced runs.
template <typename KeyT, int RB>
__global__ void __launch_bounds__(kThreads) sort_hist_kernel(const KeyT* __restrict__ keys,
                                                             const CloudRef* __restrict__ clouds, int batch,
                                                             int chunk_pts, int shift, int* __restrict__ hist,
                                                             int* __restrict__ bintot) {
  // one private histogram per warp (shared-memory atomics never cross warps), summed at the end
  __shared__ int sh[kWarps][1 << RB];
  for (int d = threadIdx.x; d < (1 << RB); d += kThreads)
#pragma unroll
    for (int w = 0; w < kWarps; ++w) sh[w][d] = 0;
  grid_dependency_wait();       // launched as a programmatic dependent: see common.cuh
  const Chunk c = chunk_of(clouds, batch, chunk_pts);
  __syncthreads();
  for (long long i0 = c.beg; i0 < c.end; i0 += 8 * kThreads) {
    KeyT k[8];                  // all requested before the first is counted
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const long long i = i0 + u * kThreads + threadIdx.x;
      k[u] = i < c.end ? keys[i] : 0;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const long long i = i0 + u * kThreads + threadIdx.x;
      count_digit(sh[threadIdx.x >> 5], i < c.end ? (int)((k[u] >> shift) & ((1 << RB) - 1)) : (1 << RB), 1 << RB);
    }
  }
  publish_counts<RB>(sh, c, clouds[c.segment].chunk0, hist, bintot);
  grid_dependency_trigger();    // at the end: the successor's blocks should not sit on SM slots early
}

__device__ __forceinline__ int block_exclusive_scan(int v, int* total) {
  // exclusive prefix of v over the CTA's kThreads threads
  __shared__ int wsum[kWarps];
  __shared__ int wtot;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int inc = v;
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  __syncthreads();   // protects wsum/wtot of a previous call
  if (lane == 31) wsum[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    int w = lane < kWarps ? wsum[lane] : 0;
    int winc = w;
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, winc, o);
      if (lane >= o) winc += t;
    }
    if (lane < kWarps) wsum[lane] = winc - w;
    if (lane == kWarps - 1) wtot = winc;
  }
  __syncthreads();
  *total = wtot;
  return inc - v + wsum[warp];
}

// Exclusive scan of every segment's hist[digit][chunk] in that order, starting at the segment's first
// point: one warp per (segment, digit) row.
template <int RB>
__global__ void __launch_bounds__(kThreads) sort_rowscan_kernel(int* __restrict__ hist,
                                                                const CloudRef* __restrict__ clouds, int batch,
                                                                const int* __restrict__ bintot) {
  constexpr int kBins = 1 << RB;
  grid_dependency_wait();       // launched as a programmatic dependent: see common.cuh
  const int lane = threadIdx.x & 31;
  const long long row = (long long)blockIdx.x * kWarps + (threadIdx.x >> 5);
  if (row < (long long)batch * kBins) {
    const int b = (int)(row >> RB), digit = (int)(row & (kBins - 1));
    const CloudRef c = clouds[b];
    const int chunks = clouds[b + 1].chunk0 - c.chunk0;
    // first slot of this digit = number of the segment's keys with a smaller digit
    int below = 0;
    for (int d = lane; d < digit; d += 32) below += bintot[b * kBins + d];
    for (int o = 16; o > 0; o >>= 1) below += __shfl_xor_sync(0xffffffffu, below, o);
    int base = (int)c.offset + below;
    int* at = hist + (long long)c.chunk0 * kBins + (long long)digit * chunks;
    for (int i0 = 0; i0 < chunks; i0 += 32) {
      const int i = i0 + lane;
      const int v = i < chunks ? at[i] : 0;
      int inc = v;
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
      }
      if (i < chunks) at[i] = base + inc - v;
      base += __shfl_sync(0xffffffffu, inc, 31);
    }
  }
  grid_dependency_trigger();    // at the end: the successor's blocks should not sit on SM slots early
}

// The lanes of `mask` whose RB-bit digit equals this lane's: one ballot per bit.  (Measured several
// times faster here than match.any.)
template <int RB>
__device__ __forceinline__ unsigned match_digit(unsigned mask, int digit) {
  unsigned peers = mask;
#pragma unroll
  for (int b = 0; b < RB; ++b) {
    const bool bit = (digit >> b) & 1;
    const unsigned with = __ballot_sync(mask, bit);
    peers &= bit ? with : ~with;
  }
  return peers;
}

template <typename KeyT, bool FIRST, int RB>
__global__ void __launch_bounds__(kThreads) sort_scatter_kernel(
    const KeyT* __restrict__ keys_in, const uint32_t* __restrict__ idx_in,
    KeyT* __restrict__ keys_out, uint32_t* __restrict__ idx_out, const CloudRef* __restrict__ clouds, int batch,
    int chunk_pts, int shift, const int* __restrict__ hist) {
  constexpr int kBins = 1 << RB, kPer = kBins / kThreads;     // digits per thread: 1 or 2, neighbours
  __shared__ int cnt[kWarps][kBins];      // per-warp digit counts, then per-warp digit bases
  __shared__ int tile_start[kBins];       // first slot of each digit inside the sorted tile
  __shared__ int gofs[kBins];             // next global slot of each digit for this CTA
  __shared__ KeyT skey[kSortTile];
  __shared__ uint32_t sidx[kSortTile];
  grid_dependency_wait();       // launched as a programmatic dependent: see common.cuh
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const Chunk c = chunk_of(clouds, batch, chunk_pts);
  {
    const int* from = hist + (long long)clouds[c.segment].chunk0 * kBins + c.first;
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
      const int d = threadIdx.x * kPer + q;
      gofs[d] = from[(long long)d * c.chunks];
    }
  }
  for (long long t0 = c.beg; t0 < c.end; t0 += kSortTile) {
    const int tile_n = (int)((c.end - t0) < kSortTile ? (c.end - t0) : kSortTile);
    for (int d = threadIdx.x; d < kBins; d += kThreads)
#pragma unroll
      for (int w = 0; w < kWarps; ++w) cnt[w][d] = 0;
    __syncthreads();
    // 1. rank inside the warp's 256 keys (index order = rank order: stable)
    KeyT key[kSortItems];
    uint32_t idx[kSortItems];
    int rank[kSortItems];
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {      // all loads of the tile first: one latency, not 8
      const int local = warp * (32 * kSortItems) + r * 32 + lane;
      key[r] = 0;
      idx[r] = 0;
      if (local < tile_n) {
        key[r] = keys_in[t0 + local];
        idx[r] = FIRST ? (uint32_t)(t0 + local) : idx_in[t0 + local];
      }
    }
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
      const int local = warp * (32 * kSortItems) + r * 32 + lane;
      const bool valid = local < tile_n;
      const unsigned mask = __ballot_sync(0xffffffffu, valid);
      rank[r] = -1;
      if (valid) {
        const int digit = (int)((key[r] >> shift) & (kBins - 1));
        const unsigned peers = match_digit<RB>(mask, digit);
        const int before = __popc(peers & ((1u << lane) - 1));
        rank[r] = cnt[warp][digit] + before;
        __syncwarp(mask);
        if (before == 0) cnt[warp][digit] += __popc(peers);
      }
      __syncwarp();
    }
    __syncthreads();
    // 2. every thread: prefix its digits over the warps, then over the digits
    int total_d[kPer], sum = 0;
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
      const int d = threadIdx.x * kPer + q;
      int t = 0;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {
        const int v = cnt[w][d];
        cnt[w][d] = t;
        t += v;
      }
      total_d[q] = t;
      sum += t;
    }
    int tile_total;
    int start_d = block_exclusive_scan(sum, &tile_total);
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
      tile_start[threadIdx.x * kPer + q] = start_d;
      start_d += total_d[q];
    }
    __syncthreads();
    // 3. tile into shared memory in digit order
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
      if (rank[r] >= 0) {
        const int digit = (int)((key[r] >> shift) & (kBins - 1));
        const int pos = tile_start[digit] + cnt[warp][digit] + rank[r];
        skey[pos] = key[r];
        sidx[pos] = idx[r];
      }
    }
    __syncthreads();
    // 4. copy out: slot i of the sorted tile goes to gofs[digit] + (i - tile_start[digit])
    for (int i = threadIdx.x; i < tile_n; i += kThreads) {
      const KeyT k = skey[i];
      const int digit = (int)((k >> shift) & (kBins - 1));
      const long long pos = (long long)gofs[digit] + (i - tile_start[digit]);
      keys_out[pos] = k;
      idx_out[pos] = sidx[i];
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kPer; ++q) gofs[threadIdx.x * kPer + q] += total_d[q];
    __syncthreads();
  }
  grid_dependency_trigger();    // at the end: the successor's blocks should not sit on SM slots early
}

// ---- unique for every level at once (reduce, then scan) -------------------------------------------
// In the sorted composite keys, point i opens a new node at level d iff its key differs from the one
// before it above bit 3 (depth - d); a node opened at one level opens one at every finer level too,
// so a point is described by the coarsest level it opens (`levels` = none).  Level l = 0 is the full
// level, l = levels - 1 the finest.  K_l[rank] = key >> 3 (levels - 1 - l), start_l[rank] = the rank the
// same point has one level finer (the point itself at the finest), so that a node's children are
// start_l[a] .. start_l[a + 1].
template <typename KeyT>
struct UniqueArgs {
  const KeyT* keys;
  long long n;
  int depth, full, levels;
  int wide;                 // 32-bit keys on a 16-byte boundary (the workspace may lie on 8)
  int* blockcnt;            // [levels][blocks]
  int* counts;              // by depth
  int* host_counts;         // the same in mapped host memory
  KeyT* K[OCNN_MAX_DEPTH + 1];
  int* start[OCNN_MAX_DEPTH + 1];
};

__device__ __forceinline__ int top_bit(uint32_t v) { return 31 - __clz(v); }
__device__ __forceinline__ int top_bit(uint64_t v) { return 63 - __clzll((long long)v); }

template <typename KeyT>
__device__ __forceinline__ int opened_level(const UniqueArgs<KeyT>& a, KeyT key, KeyT prev, bool first) {
  if (first) return 0;
  const KeyT x = key ^ prev;
  if (x == 0) return a.levels;
  const int l = a.depth - top_bit(x) / 3 - a.full;
  return l < 0 ? 0 : l;
}

__device__ __forceinline__ void scan_range(long long n, long long* beg, long long* end) {
  long long chunk = (n + gridDim.x - 1) / gridDim.x;
  chunk = (chunk + kScanTile - 1) / kScanTile * kScanTile;
  *beg = (long long)blockIdx.x * chunk;
  if (*beg > n) *beg = n;
  const long long e = *beg + chunk;
  *end = e < n ? e : n;
}

// Four consecutive keys per thread (one 16-byte read where `wide`) and the key before them.
template <typename KeyT>
__device__ __forceinline__ void load_items(const UniqueArgs<KeyT>& a, long long i0, long long end,
                                           KeyT (&key)[kScanItems], int (&lvl)[kScanItems]) {
  KeyT prev = (i0 > 0 && i0 < end) ? a.keys[i0 - 1] : 0;
  if (sizeof(KeyT) == 4 && a.wide && i0 + kScanItems <= end) {
    const uint4 q = *reinterpret_cast<const uint4*>(a.keys + i0);
    key[0] = (KeyT)q.x; key[1] = (KeyT)q.y; key[2] = (KeyT)q.z; key[3] = (KeyT)q.w;
  } else {
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) key[k] = i0 + k < end ? a.keys[i0 + k] : 0;
  }
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    lvl[k] = i0 + k < end ? opened_level(a, key[k], prev, i0 + k == 0) : a.levels;
    prev = key[k];
  }
}

template <typename KeyT, int LV>       // LV: bound on the levels
__global__ void __launch_bounds__(kThreads) unique_count_kernel(const __grid_constant__ UniqueArgs<KeyT> a) {
  __shared__ int red[kWarps][LV];
  grid_dependency_wait();       // launched as a programmatic dependent: see common.cuh
  long long beg, end;
  scan_range(a.n, &beg, &end);
  int cnt[LV];
#pragma unroll
  for (int l = 0; l < LV; ++l) cnt[l] = 0;
  for (long long t0 = beg; t0 < end; t0 += kScanTile) {
    KeyT key[kScanItems];
    int lvl[kScanItems];
    load_items(a, t0 + (long long)threadIdx.x * kScanItems, end, key, lvl);
#pragma unroll
    for (int k = 0; k < kScanItems; ++k)
#pragma unroll
      for (int l = 0; l < LV; ++l) cnt[l] += (lvl[k] <= l && lvl[k] < a.levels) ? 1 : 0;
  }
#pragma unroll
  for (int l = 0; l < LV; ++l) {
    for (int o = 16; o > 0; o >>= 1) cnt[l] += __shfl_down_sync(0xffffffffu, cnt[l], o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][l] = cnt[l];
  }
  __syncthreads();
  if (threadIdx.x < a.levels) {
    int t = 0;
    for (int w = 0; w < kWarps; ++w) t += red[w][threadIdx.x];
    a.blockcnt[threadIdx.x * gridDim.x + blockIdx.x] = t;
  }
  grid_dependency_trigger();    // at the end: the successor's blocks should not sit on SM slots early
}

template <typename KeyT, int LV>
__global__ void __launch_bounds__(kThreads) unique_compact_kernel(const __grid_constant__ UniqueArgs<KeyT> a) {
  constexpr int W = (LV + 1) / 2;         // two levels' counts per word, 16 bits each (a tile has 1024 keys)
  __shared__ int s_base[LV];              // nodes of the level in all tiles before this one
  __shared__ unsigned s_warp[kWarps][W];
  grid_dependency_wait();       // launched as a programmatic dependent: see common.cuh
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int l = warp; l < a.levels; l += kWarps) {
    int c = 0;
    for (int g = lane; g < (int)blockIdx.x; g += 32) c += a.blockcnt[l * gridDim.x + g];
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if (lane == 0) s_base[l] = c;
  }
  __syncthreads();
  long long beg, end;
  scan_range(a.n, &beg, &end);
  for (long long t0 = beg; t0 < end; t0 += kScanTile) {
    const long long i0 = t0 + (long long)threadIdx.x * kScanItems;
    KeyT key[kScanItems];
    int lvl[kScanItems];
    load_items(a, i0, end, key, lvl);
    unsigned own[W], inc[W];
#pragma unroll
    for (int w = 0; w < W; ++w) {
      own[w] = 0;
#pragma unroll
      for (int k = 0; k < kScanItems; ++k)
        if (lvl[k] < a.levels)
          own[w] += (lvl[k] <= 2 * w ? 1u : 0u) + (lvl[k] <= 2 * w + 1 ? 0x10000u : 0u);
      inc[w] = own[w];
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(0xffffffffu, inc[w], o);
        if (lane >= o) inc[w] += t;
      }
      if (lane == 31) s_warp[warp][w] = inc[w];
    }
    __syncthreads();
    int rank[LV];
#pragma unroll
    for (int w = 0; w < W; ++w) {
      unsigned before = inc[w] - own[w];
      for (int v = 0; v < warp; ++v) before += s_warp[v][w];
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (2 * w + h < LV) rank[2 * w + h] = (2 * w + h < a.levels ? s_base[2 * w + h] : 0) +
                                              (int)((before >> (16 * h)) & 0xffffu);
    }
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
      if (lvl[k] >= a.levels) continue;
#pragma unroll
      for (int l = 0; l < LV; ++l) {
        if (l < lvl[k] || l >= a.levels) continue;
        a.K[l][rank[l]] = key[k] >> (3 * (a.levels - 1 - l));
        a.start[l][rank[l]] = l == a.levels - 1 ? (int)(i0 + k) : rank[l + 1 < LV ? l + 1 : l];
      }
#pragma unroll
      for (int l = 0; l < LV; ++l)
        if (l >= lvl[k]) ++rank[l];
    }
    __syncthreads();
    if (threadIdx.x < a.levels) {
      unsigned t = 0;
      for (int v = 0; v < kWarps; ++v) t += (s_warp[v][threadIdx.x >> 1] >> (16 * (threadIdx.x & 1))) & 0xffffu;
      s_base[threadIdx.x] += (int)t;
    }
    __syncthreads();
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x < a.levels) {
    const int l = threadIdx.x, c = s_base[l];
    a.counts[a.full + l] = c;
    a.host_counts[a.full + l] = c;
    a.start[l][c] = l == a.levels - 1 ? (int)a.n : s_base[l + 1];
  }
  grid_dependency_trigger();    // at the end: the successor's blocks should not sit on SM slots early
}

// ---- a small cloud in one launch ----------------------------------------------------------------
// Keys, sort and unique of a cloud that one CTA holds, in the workspace form that the launches above leave
// (sorted indices, K and start of every level, counts, the table of clouds).  What bounds it: a chain of steps
// that each run once, so latency and the fetching of code; the loops are rolled (unrolled over a thread's eight
// keys and ten levels the kernel took 26 to 31 us at 5000 points, 20 us so; as nine launches, each 3 to 7 us for a
// few blocks of work, it was 39 us of a data loader's 78 us a sample).
//
// Keys and indices lie in shared memory, twice.  A warp owns a run of rows of 32 keys; a pass counts its digits per
// warp, prefixes the counts over the warps and the digits, and moves the keys row by row (ranks inside a row by
// ballots: match_digit), which keeps equal digits in order.
constexpr int kSmallThreads = 1024, kSmallWarps = 32, kSmallBins = 256, kSmallPoints = 6144;
size_t small_smem(int64_t n) {
  return (size_t)((n + 31) / 32 * 32) * 12 + (size_t)kSmallWarps * kSmallBins * 4 + (4 + 1) * kSmallBins * 4;
}

__global__ void __launch_bounds__(kSmallThreads) small_build_kernel(const __grid_constant__ EncodeArgs e,
                                                                    const __grid_constant__ UniqueArgs<uint32_t> a,
                                                                    uint32_t* __restrict__ idx_out, int passes) {
  extern __shared__ __align__(16) uint8_t small_raw[];
  const int n = (int)a.n, cap = (n + 31) & ~31;
  uint32_t* key = reinterpret_cast<uint32_t*>(small_raw);            // [2][cap]
  int* cnt = reinterpret_cast<int*>(key + 2 * cap);                  // [warp][digit]
  int* part = cnt + kSmallWarps * kSmallBins;                        // [4][digit]
  int* first = part + 4 * kSmallBins;                                // [digit]
  uint16_t* idx = reinterpret_cast<uint16_t*>(first + kSmallBins);   // [2][cap]
  __shared__ int s_scan[kSmallWarps], s_level[kSmallWarps][32], s_total[32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rows = (cap / 32 + kSmallWarps - 1) / kSmallWarps;       // rows a warp owns
  const int run0 = min(warp * rows * 32, cap), run1 = min(run0 + rows * 32, cap);
  const unsigned below = (1u << lane) - 1u;
  grid_dependency_wait();       // launched as a programmatic dependent: see common.cuh
  if (tid < 2) const_cast<CloudRef*>(e.table)[tid] = e.clouds[tid];
#pragma unroll 4
  for (int i = tid; i < n; i += kSmallThreads) {
    const float* from = e.clouds[0].xyz + 3 * i;
    const float p[3] = {from[0], from[1], from[2]};
    key[i] = (uint32_t)cell_key(e, p, 0);
    idx[i] = (uint16_t)i;
  }
  int from = 0;
#pragma unroll 1
  for (int pass = 0; pass < passes; ++pass, from ^= 1) {
    const uint32_t* kin = key + from * cap;
    const uint16_t* iin = idx + from * cap;
    uint32_t* kout = key + (from ^ 1) * cap;
    uint16_t* iout = idx + (from ^ 1) * cap;
    int* mine = cnt + warp * kSmallBins;
    for (int d = lane; d < kSmallBins; d += 32) mine[d] = 0;
    __syncthreads();
#pragma unroll 1
    for (int i = run0 + lane; i < run1; i += 32) {
      const int digit = i < n ? (int)((kin[i] >> (8 * pass)) & (kSmallBins - 1)) : kSmallBins;
      count_digit(mine, digit, kSmallBins);
    }
    __syncthreads();
    {                                    // a digit's counts over the warps: four threads a digit, eight warps each
      const int digit = tid & (kSmallBins - 1), q = tid >> 8;
      int* c = cnt + q * 8 * kSmallBins + digit;
      int v[8], sum = 0;
#pragma unroll
      for (int w = 0; w < 8; ++w) {
        v[w] = c[w * kSmallBins];
        sum += v[w];
      }
      part[q * kSmallBins + digit] = sum;
      __syncthreads();
      int at = 0;
      for (int p = 0; p < q; ++p) at += part[p * kSmallBins + digit];
#pragma unroll
      for (int w = 0; w < 8; ++w) {
        c[w * kSmallBins] = at;
        at += v[w];
      }
      // the digits' totals, prefixed by the last quarter's warps
      int inc = at;
      if (q == 3) {
        for (int o = 1; o < 32; o <<= 1) {
          const int t = __shfl_up_sync(0xffffffffu, inc, o);
          if (lane >= o) inc += t;
        }
        if (lane == 31) s_scan[warp - 24] = inc;
      }
      __syncthreads();
      if (q == 3) {
        int base = inc - at;
        for (int w = 0; w < warp - 24; ++w) base += s_scan[w];
        first[digit] = base;
      }
    }
    __syncthreads();
#pragma unroll 1
    for (int i = run0 + lane; i < run1; i += 32) {
      const unsigned mask = __ballot_sync(0xffffffffu, i < n);
      if (i < n) {
        const uint32_t k = kin[i];
        const int digit = (int)((k >> (8 * pass)) & (kSmallBins - 1));
        const unsigned peers = match_digit<8>(mask, digit);
        const int before = __popc(peers & below), at = mine[digit];
        __syncwarp(mask);
        if (before == 0) mine[digit] = at + __popc(peers);
        kout[first[digit] + at + before] = k;
        iout[first[digit] + at + before] = iin[i];
      }
      __syncwarp();
    }
    __syncthreads();
  }
  const uint32_t* sorted = key + from * cap;
  for (int i = tid; i < n; i += kSmallThreads) idx_out[i] = idx[from * cap + i];
  // Nodes opened per level: a level's nodes of a row are its ballot; lane l keeps level l's count.
  auto opened = [&](int i) { return i < n ? opened_level(a, sorted[i], i > 0 ? sorted[i - 1] : 0u, i == 0) : a.levels; };
  int count = 0;
#pragma unroll 1
  for (int i = run0 + lane; i < run1; i += 32) {
    const int lvl = opened(i);
#pragma unroll 1
    for (int l = 0; l < a.levels; ++l) {
      const int c = __popc(__ballot_sync(0xffffffffu, lvl <= l));
      if (lane == l) count += c;
    }
  }
  s_level[warp][lane] = count;
  __syncthreads();
  if (warp < a.levels) {                 // warp l: the prefix of level l over the warps
    const int v = s_level[lane][warp];
    int t = v;
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += u;
    }
    s_level[lane][warp] = t - v;
    if (lane == 31) s_total[warp] = t;
  }
  __syncthreads();
  count = s_level[warp][lane];
#pragma unroll 1
  for (int i = run0 + lane; i < run1; i += 32) {
    const int lvl = opened(i);
    int finer = i;                       // this node's first entry one level finer
#pragma unroll 1
    for (int l = a.levels - 1; l >= 0; --l) {
      const unsigned opens = __ballot_sync(0xffffffffu, lvl <= l);
      const int rank = __shfl_sync(0xffffffffu, count, l) + __popc(opens & below);
      if (lvl <= l) {
        a.K[l][rank] = sorted[i] >> (3 * (a.levels - 1 - l));
        a.start[l][rank] = finer;
      }
      finer = rank;
      if (lane == l) count += __popc(opens);
    }
  }
  if (tid < a.levels) {
    a.counts[a.full + tid] = s_total[tid];
    a.host_counts[a.full + tid] = s_total[tid];
    a.start[tid][s_total[tid]] = tid == a.levels - 1 ? n : s_total[tid + 1];
  }
  grid_dependency_trigger();
}

// ---- emit ------------------------------------------------------------------------------------
struct EmitLevel {
  long long off_key, off_child, off_split;   // byte offsets of this level (split < 0: absent)
  long long nnum;
  const void* Kp;            // K(d-1), levels above the full ones only
  const void* Kc;            // Kd
  const int* start;          // first entry of Kc under each parent
  int d, block0;             // first block of the level
};
struct EmitAll {
  uint8_t* out;              // octree buffer
  int nlev, batch, full, depth, key_bytes;
  const void* K_full;        // the full level's non-empty nodes, for its children
  const int* count_full;
  float* feat;               // finest level's feature block, [channels, nnum]; NULL: written elsewhere
  int channels;
  const float* avg[6];       // a channel's values on the non-empty finest nodes
  EmitLevel lev[OCNN_MAX_DEPTH + 1];
  uint8_t header[OCNN_HEADER_BYTES];
};

__device__ __forceinline__ void store_key(uint8_t* base, long long off, long long i, uint64_t local,
                                          int b, int key_bytes) {
  // batch index into the top lane of the key: byte 3 of a 32-bit key, uint16 lane 3 of a 64-bit
  // key (merge_octrees.cpp:127-131); a single octree has b = 0.
  if (key_bytes == 8) {
    reinterpret_cast<uint64_t*>(base + off)[i] = (local & 0x0000ffffffffffffULL) | ((uint64_t)(b & 0xffff) << 48);
  } else {
    reinterpret_cast<uint32_t*>(base + off)[i] = ((uint32_t)local & 0x00ffffffu) | ((uint32_t)(b & 0xff) << 24);
  }
}

constexpr int kEmitNodes = kThreads * 8;      // nodes per block: 32 parents per warp
// Nodes per lane whose averages are read before any of them is written: the compiler may not move a read
// over the stores (both are plain float pointers), so one node at a time was eight memory latencies per warp
// (3.3 TB/s, 24 of 30 stall cycles waiting for a load).  Four: build of 64 x 100k at depth 8 916 -> 876 us,
// of 200 k points at depth 9 130 -> 121 us.
constexpr int kEmitAhead = 4;

// All levels in one launch, a block serves one level.
// Levels 0..full hold every node: key = index inside its octree, child = itself below the full level
// (octree.cpp:210-224); at the full level the rank of the node in K_full, whose composite key IS the
// batch-wide node index (octree.cpp:277-282 + the rebasing of merge_octrees.cpp:136-144).
// Level d > full: node 8a+j is the j-th child slot of the a-th non-empty node of level d-1
// (octree.cpp:226-273).  A lane fetches one parent and the octants of its children as a bit mask; its
// 8 nodes are then written by the warp 32 at a time, in order.  Everything a warp's 256 nodes need is
// requested before the first of them is written (one node per thread was a chain of three reads per
// 12 bytes written: 258 us for 23 M nodes).
template <typename KeyT>
__global__ void __launch_bounds__(kThreads) emit_levels_kernel(const __grid_constant__ EmitAll A) {
  grid_dependency_wait();       // launched as a programmatic dependent: see common.cuh
  if (blockIdx.x == 0)
    for (int i = threadIdx.x; i < OCNN_HEADER_BYTES / 4; i += kThreads)
      reinterpret_cast<int*>(A.out)[i] = reinterpret_cast<const int*>(A.header)[i];
  int li = 0;
  while (li + 1 < A.nlev && (int)blockIdx.x >= A.lev[li + 1].block0) ++li;
  const EmitLevel& a = A.lev[li];
  const int lane = threadIdx.x & 31;
  const long long i0 = (long long)((int)blockIdx.x - a.block0) * kEmitNodes;
  int* child = reinterpret_cast<int*>(A.out + a.off_child);
  float* split = a.off_split >= 0 ? reinterpret_cast<float*>(A.out + a.off_split) : nullptr;
  const bool with_feat = A.feat != nullptr && a.d == A.depth;
  if (a.d <= A.full) {
    const long long per = 1LL << (3 * a.d);
    const KeyT* K = static_cast<const KeyT*>(A.K_full);
    const int nk = a.d == A.full && K != nullptr ? *A.count_full : 0;
    for (long long i = i0 + threadIdx.x; i < i0 + kEmitNodes && i < a.nnum; i += kThreads) {
      const int b = (int)(i / per);
      store_key(A.out, a.off_key, i, (uint64_t)(i - b * per), b, A.key_bytes);
      int ch = a.d < A.full ? (int)i : -1;
      if (nk > 0) {
        int lo = 0, hi = nk;
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if ((long long)K[mid] < i) lo = mid + 1; else hi = mid;
        }
        if (lo < nk && (long long)K[lo] == i) ch = lo;
      }
      child[i] = ch;
      if (split) split[i] = ch < 0 ? 0.f : 1.f;
      if (with_feat)            // (the full level is the finest: no node has a signal)
        for (int c = 0; c < A.channels; ++c) A.feat[c * a.nnum + i] = 0.f;
    }
  } else {
    const KeyT* __restrict__ Kp = static_cast<const KeyT*>(a.Kp);
    const KeyT* __restrict__ Kc = static_cast<const KeyT*>(a.Kc);
    const long long w0 = i0 + (threadIdx.x & ~31) * 8;          // the warp's first node
    const long long p = (w0 >> 3) + lane, np = a.nnum >> 3;
    KeyT pk = 0;
    int s0 = 0, s1 = 0;
    if (p < np) {
      pk = Kp[p];
      s0 = a.start[p];
      s1 = a.start[p + 1];
    }
    unsigned octants = 0;
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (s0 + u < s1) octants |= 1u << (int)(Kc[s0 + u] & 7);
    const uint64_t local_mask = (1ULL << (3 * (a.d - 1))) - 1ULL;
    const int o = lane & 7;
#pragma unroll
    for (int half = 0; half < 8; half += kEmitAhead) {
      int ch[kEmitAhead];
      float v[kEmitAhead][6];
#pragma unroll
      for (int t = 0; t < kEmitAhead; ++t) {
        const int src = (half + t) * 4 + (lane >> 3);
        const int first = __shfl_sync(0xffffffffu, s0, src);
        const unsigned have = __shfl_sync(0xffffffffu, octants, src);
        ch[t] = (have >> o) & 1 ? first + __popc(have & ((1u << o) - 1)) : -1;   // (none beyond the level)
        if (with_feat) {
#pragma unroll
          for (int c = 0; c < 6; ++c)
            v[t][c] = c < A.channels && ch[t] >= 0 ? A.avg[c][ch[t]] : 0.f;
        }
      }
#pragma unroll
      for (int t = 0; t < kEmitAhead; ++t) {
        const long long i = w0 + (half + t) * 32 + lane;
        const KeyT key = __shfl_sync(0xffffffffu, pk, (half + t) * 4 + (lane >> 3));
        if (i >= a.nnum) continue;       // (whole sibling groups leave together; shuffles of all lanes precede)
        store_key(A.out, a.off_key, i, (((uint64_t)key & local_mask) << 3) | (uint64_t)o,
                  (int)((uint64_t)key >> (3 * (a.d - 1))), A.key_bytes);
        child[i] = ch[t];
        if (split) split[i] = ch[t] < 0 ? 0.f : 1.f;
        if (with_feat) {
#pragma unroll
          for (int c = 0; c < 6; ++c)
            if (c < A.channels) A.feat[c * a.nnum + i] = v[t][c];
        }
      }
    }
  }
  grid_dependency_trigger();    // at the end: the successor's blocks should not sit on SM slots early
}

// finest-level signal, octree.cpp:312-452 restated per node.  Rows of the feature block, in
// order: normals, displacement, point features, average points (octree.cpp:916-926).
template <typename KeyT>
struct SignalArgs {
  const int* child;          // level `depth` children = index into seg
  const int* seg;            // point segment starts per non-empty finest node
  const uint32_t* sorted_idx;
  const KeyT* K;             // composite keys of the non-empty finest nodes (cloud in the top bits)
  const CloudRef* clouds;
  int depth;
  int has_normal, has_feat;
  float* f_out;              // feature block of the finest level, [C, nnum]
  float* l_out;              // label block or NULL
  long long nnum;
  int cf, node_dis, save_pts;
  float bbmin[3];
  float mul;
  float* avg[6];             // signal_average_kernel: where each channel goes
  int nodes;                 // ... and the number of non-empty nodes
};

// Normals and / or point features (no displacement, labels or average points), averaged per
// non-empty node into compact arrays that the emit kernel spreads over the level's nodes.  Two nodes
// per thread in lock step, every stage of the chain segment -> point index -> values requested for
// both before any is used.  The arithmetic and its order are signal_kernel's: bit-identical.
template <typename KeyT>
__global__ void __launch_bounds__(256) signal_average_kernel(const __grid_constant__ SignalArgs<KeyT> a) {
  grid_dependency_wait();       // launched as a programmatic dependent: see common.cuh
  constexpr int U = 2;
  const int stride = gridDim.x * blockDim.x;
  for (int r0 = blockIdx.x * blockDim.x + threadIdx.x; r0 < a.nodes; r0 += stride * U) {
    int s0[U], s1[U];
    KeyT key[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int r = r0 + u * stride;
      s0[u] = s1[u] = 0;
      key[u] = 0;
      if (r < a.nodes) { s0[u] = a.seg[r]; s1[u] = a.seg[r + 1]; key[u] = a.K[r]; }
    }
    long long h0[U];
    const float* normals[U];
    const float* feats[U];
    long long base[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      h0[u] = 0; normals[u] = feats[u] = nullptr; base[u] = 0;
      if (s1[u] > s0[u]) {
        const CloudRef& cl = a.clouds[(int)((uint64_t)key[u] >> (3 * a.depth))];
        normals[u] = cl.normal;
        feats[u] = cl.feat;
        base[u] = cl.offset;
        h0[u] = a.sorted_idx[s0[u]] - base[u];
      }
    }
    float first[U][3];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int c = 0; c < 3; ++c) first[u][c] = (a.has_normal && s1[u] > s0[u]) ? normals[u][3 * h0[u] + c] : 0.f;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int r = r0 + u * stride;
      if (s1[u] <= s0[u]) continue;
      if (a.has_normal) {
        float nrm[3] = {0.f, 0.f, 0.f};
        nrm[0] += first[u][0]; nrm[1] += first[u][1]; nrm[2] += first[u][2];
        for (int j = s0[u] + 1; j < s1[u]; ++j) {
          const long long h = a.sorted_idx[j] - base[u];
          nrm[0] += normals[u][3 * h]; nrm[1] += normals[u][3 * h + 1]; nrm[2] += normals[u][3 * h + 2];
        }
        float len = 0.f;
        len += nrm[0] * nrm[0]; len += nrm[1] * nrm[1]; len += nrm[2] * nrm[2];
        float factor = sqrtf(len);
        if (factor < 1.0e-6f) {
          nrm[0] = first[u][0]; nrm[1] = first[u][1]; nrm[2] = first[u][2];
          len = 0.f;
          len += nrm[0] * nrm[0]; len += nrm[1] * nrm[1]; len += nrm[2] * nrm[2];
          factor = sqrtf(len) + 1.0e-30f;
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) a.avg[c][r] = nrm[c] / factor;
      }
      const float cnt = (float)(unsigned)(s1[u] - s0[u]) + 1.0e-30f;
      for (int c = 0; c < a.cf; ++c) {
        float acc = 0.f;
        for (int j = s0[u]; j < s1[u]; ++j) acc += feats[u][(long long)a.cf * (a.sorted_idx[j] - base[u]) + c];
        a.avg[(a.has_normal ? 3 : 0) + c][r] = acc / cnt;
      }
    }
  }
  grid_dependency_trigger();    // at the end: the successor's blocks should not sit on SM slots early
}

template <typename KeyT>
__global__ void signal_kernel(const __grid_constant__ SignalArgs<KeyT> a) {
  grid_dependency_wait();       // launched as a programmatic dependent: see common.cuh
  const long long nn = a.nnum;
  const int cn = a.has_normal ? 3 : 0;
  const int cdis = a.node_dis ? (a.has_normal ? 1 : 4) : 0;
  float* f_normal = a.f_out;
  float* f_dis = f_normal + cn * nn;
  float* f_feat = f_dis + cdis * nn;
  float* f_pts = f_feat + (long long)a.cf * nn;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nn;
       i += (long long)gridDim.x * blockDim.x) {
    const int t = a.child[i];
    if (t < 0) {
      const int ctot = cn + cdis + a.cf + (a.save_pts ? 3 : 0);
      for (int c = 0; c < ctot; ++c) a.f_out[c * nn + i] = 0.f;
      if (a.l_out) a.l_out[i] = -1.f;
      continue;
    }
    const int s0 = a.seg[t], s1 = a.seg[t + 1];
    // every point of a node comes from the node's own cloud; sorted_idx is batch-wide
    const CloudRef cl = a.clouds[(int)((uint64_t)a.K[t] >> (3 * a.depth))];
    const float* normals = cl.normal;
    const float* feats = cl.feat;
    const float* labels = cl.label;
    const float* xyz = cl.xyz;
    const long long base = cl.offset;
    float nrm[3] = {0.f, 0.f, 0.f};
    if (a.has_normal) {
      for (int j = s0; j < s1; ++j) {
        const long long h = a.sorted_idx[j] - base;
        nrm[0] += normals[3 * h]; nrm[1] += normals[3 * h + 1]; nrm[2] += normals[3 * h + 2];
      }
      float len = 0.f;
      len += nrm[0] * nrm[0]; len += nrm[1] * nrm[1]; len += nrm[2] * nrm[2];
      float factor = sqrtf(len);
      if (factor < 1.0e-6f) {
        const long long h = a.sorted_idx[s0] - base;
        nrm[0] = normals[3 * h]; nrm[1] = normals[3 * h + 1]; nrm[2] = normals[3 * h + 2];
        len = 0.f;
        len += nrm[0] * nrm[0]; len += nrm[1] * nrm[1]; len += nrm[2] * nrm[2];
        factor = sqrtf(len) + 1.0e-30f;
      }
      for (int c = 0; c < 3; ++c) { nrm[c] = nrm[c] / factor; f_normal[c * nn + i] = nrm[c]; }
    }
    const float cnt = (float)(unsigned)(s1 - s0) + 1.0e-30f;
    for (int c = 0; c < a.cf; ++c) {
      float acc = 0.f;
      for (int j = s0; j < s1; ++j) acc += feats[(long long)a.cf * (a.sorted_idx[j] - base) + c];
      f_feat[c * nn + i] = acc / cnt;
    }
    if (a.l_out) {
      // majority vote over labels >= 0, smallest label on ties (octree.cpp:376-401)
      int best = -1, best_cnt = 0;
      for (int j = s0; j < s1; ++j) {
        const int l = (int)labels[a.sorted_idx[j] - base];
        if (l < 0) continue;
        int c = 0;
        for (int k = s0; k < s1; ++k) c += ((int)labels[a.sorted_idx[k] - base] == l) ? 1 : 0;
        if (c > best_cnt || (c == best_cnt && l < best)) { best = l; best_cnt = c; }
      }
      a.l_out[i] = best < 0 ? -1.f : (float)best;
    }
    if (a.node_dis || a.save_pts) {
      float avg[3] = {0.f, 0.f, 0.f}, dis[4] = {0.f, 0.f, 0.f, 0.f};
      for (int j = s0; j < s1; ++j) {
        const long long h = a.sorted_idx[j] - base;
        for (int c = 0; c < 3; ++c) avg[c] += (xyz[3 * h + c] - a.bbmin[c]) * a.mul;
      }
      for (int c = 0; c < 3; ++c) {
        avg[c] = avg[c] / cnt;
        float ip;
        dis[c] = modff(avg[c], &ip) - 0.5f;
        if (a.has_normal) dis[3] += dis[c] * nrm[c]; else dis[3] = 1.f;
        if (a.save_pts) f_pts[c * nn + i] = avg[c];
      }
      if (a.node_dis) {
        if (a.has_normal) {
          f_dis[i] = dis[3] * 1.1547f;
        } else {
          for (int c = 0; c < 3; ++c) f_dis[c * nn + i] = dis[c];
          f_dis[3 * nn + i] = dis[3] * 1.1547f;
        }
      }
    }
  }
  grid_dependency_trigger();    // at the end: the successor's blocks should not sit on SM slots early
}

// ---- host drivers -----------------------------------------------------------------------------
// The counts' way back: a mapped, pinned word per host thread, written by the last kernel of the plan.
struct HostCounts {
  int* host = nullptr;
  ~HostCounts() {
    if (host) cudaFreeHost(host);
  }
  int* get() {
    if (host == nullptr) {
      void* p = nullptr;
      if (cudaHostAlloc(&p, 32 * sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
      }
      host = static_cast<int*>(p);
    }
    return host;
  }
};

float cell_scale(const ocnn_build_params* prm) {
  float width = prm->bbmax[0] - prm->bbmin[0];
  for (int j = 1; j < 3; ++j) {
    const float w = prm->bbmax[j] - prm->bbmin[j];
    if (w > width) width = w;
  }
  if (width == 0.0f) width = 1.0e-10f;
  return (float)(1 << prm->depth) / width;
}

template <typename KeyT, int RB>
int sort_keys(const EncodeArgs& ea, const Layout& L, int chunks, uint8_t* ws, cudaStream_t st) {
  constexpr int kBins = 1 << RB;
  KeyT* keys[2] = {reinterpret_cast<KeyT*>(ws + L.off_keys[0]), reinterpret_cast<KeyT*>(ws + L.off_keys[1])};
  uint32_t* idx[2] = {reinterpret_cast<uint32_t*>(ws + L.off_idx[0]), reinterpret_cast<uint32_t*>(ws + L.off_idx[1])};
  const bool whole = L.segments != L.batch;
  const CloudRef* segs = reinterpret_cast<const CloudRef*>(ws + L.off_clouds) + (whole ? L.batch + 1 : 0);
  int* hist = reinterpret_cast<int*>(ws + L.off_hist);
  OCNN_CUDA_OK(launch_chained(whole ? encode_kernel<KeyT, RB, true> : encode_kernel<KeyT, RB, false>, dim3(chunks),
                              dim3(kThreads), 0, st, ea, keys[0], hist, reinterpret_cast<int*>(ws + L.off_bintot)));
  OCNN_LAUNCH_OK("encode_kernel");
  const int rows = ceil_div((long long)L.segments * kBins, kWarps);
  int cur = 0;
  for (int p = 0; p < L.passes; ++p) {
    const int shift = RB * p;
    int* bintot = reinterpret_cast<int*>(ws + L.off_bintot) + (size_t)p * L.segments * kBins;
    if (p > 0)
      OCNN_CUDA_OK(launch_chained(sort_hist_kernel<KeyT, RB>, dim3(chunks), dim3(kThreads), 0, st,
                                  (const KeyT*)keys[cur], segs, L.segments, ea.chunk_pts, shift, hist, bintot));
    OCNN_CUDA_OK(launch_chained(sort_rowscan_kernel<RB>, dim3(rows), dim3(kThreads), 0, st, hist, segs, L.segments,
                                (const int*)bintot));
    if (p == 0)
      OCNN_CUDA_OK(launch_chained(sort_scatter_kernel<KeyT, true, RB>, dim3(chunks), dim3(kThreads), 0, st,
                                  (const KeyT*)keys[cur], (const uint32_t*)nullptr, keys[cur ^ 1], idx[cur ^ 1],
                                  segs, L.segments, ea.chunk_pts, shift, (const int*)hist));
    else
      OCNN_CUDA_OK(launch_chained(sort_scatter_kernel<KeyT, false, RB>, dim3(chunks), dim3(kThreads), 0, st,
                                  (const KeyT*)keys[cur], (const uint32_t*)idx[cur], keys[cur ^ 1], idx[cur ^ 1],
                                  segs, L.segments, ea.chunk_pts, shift, (const int*)hist));
    OCNN_LAUNCHES_OK("radix sort pass", p == 0 ? 2 : 3);
    cur ^= 1;
  }
  return OCNN_OK;
}

template <typename KeyT>
UniqueArgs<KeyT> unique_args(const Layout& L, uint8_t* ws, int* host_counts) {
  UniqueArgs<KeyT> u;
  memset(&u, 0, sizeof(u));
  u.keys = reinterpret_cast<const KeyT*>(ws + L.off_keys[L.passes & 1]);
  u.wide = sizeof(KeyT) == 4 && (uintptr_t)u.keys % 16 == 0;
  u.n = L.n; u.depth = L.depth; u.full = L.full; u.levels = L.depth - L.full + 1;
  u.blockcnt = reinterpret_cast<int*>(ws + L.off_blockcnt);
  u.counts = reinterpret_cast<int*>(ws + L.off_counts);
  u.host_counts = host_counts;
  for (int l = 0; l < u.levels; ++l) {
    u.K[l] = reinterpret_cast<KeyT*>(ws + L.off_K[L.full + l]);
    u.start[l] = reinterpret_cast<int*>(ws + L.off_start[L.full + l]);
  }
  return u;
}

// Whether one CTA sorts: one cloud with 32-bit keys, and as many points as it sorts in no more time than the launches
// over the whole GPU.  A whole build in us, one CTA / several launches: 1000 points 37 / 53 at depth 5, 45 / 66 at
// depth 8; 4000 points 46 / 57, 58 / 70; 8000 points 58 / 57, 76 / 73; 12288 points 71 / 58, 93 / 74.  (Several
// clouds add a look-up per point: 32 of 380 points 90 / 66.)
bool one_cta(const Layout& L) { return L.batch == 1 && L.key_bytes == 4 && L.n <= kSmallPoints; }

int small_build(const EncodeArgs& ea, const Layout& L, uint8_t* ws, int* host_counts, cudaStream_t st) {
  const UniqueArgs<uint32_t> u = unique_args<uint32_t>(L, ws, host_counts);
  const int passes = (3 * L.depth + 7) / 8;
  uint32_t* idx = reinterpret_cast<uint32_t*>(ws + L.off_idx[L.passes & 1]);      // where the emit looks for it
  static PerDeviceOnce attr_once;
  const int limits = attr_once.run([&]() -> int {
    OCNN_CUDA_OK(cudaFuncSetAttribute(small_build_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)small_smem(kSmallPoints)));
    return OCNN_OK;
  });
  if (limits != OCNN_OK) return limits;
  OCNN_CUDA_OK(launch_chained(small_build_kernel, dim3(1), dim3(kSmallThreads), small_smem(L.n), st, ea, u, idx, passes));
  OCNN_LAUNCH_OK("small_build_kernel");
  return OCNN_OK;
}

template <typename KeyT>
int sort_and_unique(const EncodeArgs& ea, const Layout& L, int chunks, uint8_t* ws, int* host_counts,
                    cudaStream_t st) {
  const int rc = L.radix_bits == 9 ? sort_keys<KeyT, 9>(ea, L, chunks, ws, st) : sort_keys<KeyT, 8>(ea, L, chunks, ws, st);
  if (rc != OCNN_OK) return rc;
  const UniqueArgs<KeyT> u = unique_args<KeyT>(L, ws, host_counts);
  const int grid = grid_for(L.n, kScanTile, 4) < kMaxScanGrid ? grid_for(L.n, kScanTile, 4) : kMaxScanGrid;
  if (u.levels <= 8) {
    OCNN_CUDA_OK(launch_chained(unique_count_kernel<KeyT, 8>, dim3(grid), dim3(kThreads), 0, st, u));
    OCNN_CUDA_OK(launch_chained(unique_compact_kernel<KeyT, 8>, dim3(grid), dim3(kThreads), 0, st, u));
  } else {
    OCNN_CUDA_OK(launch_chained(unique_count_kernel<KeyT, 14>, dim3(grid), dim3(kThreads), 0, st, u));
    OCNN_CUDA_OK(launch_chained(unique_compact_kernel<KeyT, 14>, dim3(grid), dim3(kThreads), 0, st, u));
  }
  OCNN_LAUNCHES_OK("unique", 2);
  return OCNN_OK;
}

template <typename KeyT>
int emit_impl(const ocnn_points_batch* pts, const ocnn_build_params* prm, const ocnn_octree_meta* meta,
              const Layout& L, uint8_t* ws, uint8_t* o, const uint8_t (&hdr)[OCNN_HEADER_BYTES], cudaStream_t st) {
  const int D = prm->depth, F = prm->full_depth;
  SignalArgs<KeyT> sa;
  memset(&sa, 0, sizeof(sa));
  sa.seg = reinterpret_cast<const int*>(ws + L.off_start[D]);
  sa.sorted_idx = reinterpret_cast<const uint32_t*>(ws + L.off_idx[L.passes & 1]);
  sa.K = reinterpret_cast<const KeyT*>(ws + L.off_K[D]);
  sa.clouds = reinterpret_cast<const CloudRef*>(ws + L.off_clouds);
  sa.depth = D;
  sa.has_normal = pts->normal_dev != nullptr;
  sa.has_feat = pts->feature_dev != nullptr;
  sa.nnum = meta->nnum[D];
  sa.cf = pts->feature_dev ? pts->feature_channels : 0;
  sa.node_dis = prm->node_dis; sa.save_pts = prm->save_pts;
  sa.mul = cell_scale(prm);
  for (int j = 0; j < 3; ++j) sa.bbmin[j] = prm->bbmin[j];
  sa.f_out = reinterpret_cast<float*>(o + ocnn_prop_offset(meta, OCNN_PROP_FEATURE, D));
  sa.l_out = pts->label_dev ? reinterpret_cast<float*>(o + ocnn_prop_offset(meta, OCNN_PROP_LABEL, D)) : nullptr;
  sa.nodes = D > F ? meta->nnum_nempty[D] : 0;
  // Normals and features alone (up to six channels): averaged per non-empty node, spread by the emit
  // kernel. The sort's buffers are free by now and hold the channels beyond the first three.
  const int channels = (sa.has_normal ? 3 : 0) + sa.cf;
  const bool compact = channels >= 1 && channels <= 6 && sa.l_out == nullptr && !sa.node_dis && !sa.save_pts;
  if (compact) {
    float* avg = reinterpret_cast<float*>(ws + L.off_avg);
    for (int c = 0; c < 3; ++c) sa.avg[c] = avg + (size_t)c * L.cap[D];
    sa.avg[3] = reinterpret_cast<float*>(ws + L.off_keys[0]);
    sa.avg[4] = reinterpret_cast<float*>(ws + L.off_keys[1]);
    sa.avg[5] = reinterpret_cast<float*>(ws + L.off_idx[(L.passes & 1) ^ 1]);
    if (sa.nodes > 0) {
      OCNN_CUDA_OK(launch_chained(signal_average_kernel<KeyT>, dim3(grid_for((sa.nodes + 1) / 2, 256, 8)), dim3(256), 0,
                                  st, sa));
      OCNN_LAUNCH_OK("signal_average_kernel");
    }
  }

  EmitAll all;
  memset(&all, 0, sizeof(all));
  all.out = o; all.batch = L.batch; all.full = F; all.depth = D; all.key_bytes = prm->key_bits / 8;
  if (D > F && meta->nnum_nempty[F] > 0) {
    all.K_full = ws + L.off_K[F];
    all.count_full = reinterpret_cast<const int*>(ws + L.off_counts) + F;
  }
  if (compact) {
    all.feat = sa.f_out;
    all.channels = channels;
    for (int c = 0; c < 6; ++c) all.avg[c] = sa.avg[c];
  }
  memcpy(all.header, hdr, OCNN_HEADER_BYTES);
  int blocks = 0;
  for (int d = 0; d <= D; ++d) {
    if (meta->nnum[d] == 0) continue;
    EmitLevel& a = all.lev[all.nlev++];
    a.off_key = ocnn_prop_offset(meta, OCNN_PROP_KEY, d);
    a.off_child = ocnn_prop_offset(meta, OCNN_PROP_CHILD, d);
    a.off_split = meta->channels[OCNN_PROP_SPLIT] ? ocnn_prop_offset(meta, OCNN_PROP_SPLIT, d) : -1;
    a.d = d;
    a.nnum = meta->nnum[d];
    a.block0 = blocks;
    blocks += ceil_div(a.nnum, kEmitNodes);
    if (d > F) {
      a.Kp = ws + L.off_K[d - 1];
      a.Kc = ws + L.off_K[d];
      a.start = reinterpret_cast<const int*>(ws + L.off_start[d - 1]);
    }
  }
  OCNN_CUDA_OK(launch_chained(emit_levels_kernel<KeyT>, dim3(blocks), dim3(kThreads), 0, st, all));
  OCNN_LAUNCH_OK("emit_levels_kernel");

  if (meta->nnum[D] > 0 && !compact) {
    sa.child = reinterpret_cast<const int*>(o + ocnn_prop_offset(meta, OCNN_PROP_CHILD, D));
    OCNN_CUDA_OK(launch_chained(signal_kernel<KeyT>, dim3(grid_for(sa.nnum, 256, 8)), dim3(256), 0, st, sa));
    OCNN_LAUNCH_OK("signal_kernel");
  }
  return OCNN_OK;
}

int check_args(const ocnn_points_batch* pts, const ocnn_build_params* prm, const char* who) {
  OCNN_REQUIRE(pts && prm, "%s: null argument", who);
  OCNN_REQUIRE(pts->batch >= 1 && pts->offsets_host && pts->xyz_dev, "%s: empty batch", who);
  for (int b = 0; b < pts->batch; ++b)
    OCNN_REQUIRE(pts->xyz_dev[b] && (!pts->normal_dev || pts->normal_dev[b]) &&
                     (!pts->feature_dev || pts->feature_dev[b]) &&
                     (!pts->label_dev || pts->label_dev[b]),
                 "%s: cloud %d lacks a property the batch declares", who, b);
  OCNN_REQUIRE(prm->key_bits == 32 || prm->key_bits == 64, "%s: key_bits must be 32 or 64", who);
  // the header's 16-entry nnum_cum array must hold index depth + 2
  const int max_depth = prm->key_bits == 64 ? 13 : 8;
  OCNN_REQUIRE(prm->depth >= 1 && prm->depth <= max_depth,
               "%s: depth %d outside [1, %d] for %d-bit keys", who, prm->depth, max_depth,
               prm->key_bits);
  OCNN_REQUIRE(prm->full_depth >= 1 && prm->full_depth <= prm->depth,
               "%s: full_depth %d outside [1, depth]", who, prm->full_depth);
  OCNN_REQUIRE(prm->full_depth <= 7, "%s: full_depth %d too large", who, prm->full_depth);
  OCNN_REQUIRE(pts->batch <= (prm->key_bits == 64 ? 65535 : 255),
               "%s: batch %d does not fit the batch lane of a %d-bit key", who, pts->batch,
               prm->key_bits);
  OCNN_REQUIRE(prm->merged || pts->batch == 1, "%s: an un-merged build takes one cloud", who);
  OCNN_REQUIRE(pts->offsets_host[0] == 0, "%s: offsets must start at 0", who);
  for (int b = 0; b < pts->batch; ++b)
    OCNN_REQUIRE(pts->offsets_host[b + 1] > pts->offsets_host[b],
                 "%s: cloud %d is empty (the reference rejects empty point clouds)", who, b);
  OCNN_REQUIRE(pts->normal_dev || pts->feature_dev,
               "%s: points need normals or features (or both)", who);
  OCNN_REQUIRE(pts->feature_dev == nullptr || pts->feature_channels > 0,
               "%s: feature_channels must be positive", who);
  OCNN_REQUIRE(3 * prm->depth + bits_for(pts->batch) <= 64, "%s: composite key overflow", who);
  return OCNN_OK;
}

void fill_static_meta(const ocnn_points_batch* pts, const ocnn_build_params* prm,
                      ocnn_octree_meta* m) {
  memset(m, 0, sizeof(*m));
  m->key_bits = prm->key_bits;
  m->batch_size = prm->merged ? pts->batch : 1;
  m->depth = prm->depth;
  m->full_depth = prm->full_depth;
  m->has_node_dis = prm->node_dis != 0;
  m->save_pts = prm->save_pts != 0;
  // OctreeInfo::initialize, octree_info.cpp:28-64
  m->channels[OCNN_PROP_KEY] = 1; m->locations[OCNN_PROP_KEY] = -1;
  m->channels[OCNN_PROP_CHILD] = 1; m->locations[OCNN_PROP_CHILD] = -1;
  if (prm->merged) { m->channels[OCNN_PROP_NEIGH] = 8; m->locations[OCNN_PROP_NEIGH] = -1; }
  int cfeat = (pts->normal_dev ? 3 : 0) + (pts->feature_dev ? pts->feature_channels : 0);
  if (prm->node_dis) cfeat += pts->normal_dev ? 1 : 4;
  if (prm->save_pts) cfeat += 3;
  m->channels[OCNN_PROP_FEATURE] = cfeat; m->locations[OCNN_PROP_FEATURE] = prm->depth;
  if (pts->label_dev) { m->channels[OCNN_PROP_LABEL] = 1; m->locations[OCNN_PROP_LABEL] = prm->depth; }
  if (prm->split_label) { m->channels[OCNN_PROP_SPLIT] = 1; m->locations[OCNN_PROP_SPLIT] = -1; }
}

}  // namespace
}  // namespace ocnn

extern "C" {

size_t ocnn_octree_build_workspace_bytes(int64_t total_points, int batch, int depth,
                                         int full_depth) {
  if (total_points < 1 || batch < 1 || depth < 1 || depth >= OCNN_MAX_DEPTH || full_depth < 1 ||
      full_depth > depth)
    return 0;
  return ocnn::make_layout(total_points, batch, depth, full_depth).total;
}

int ocnn_octree_build_plan(const ocnn_points_batch* pts, const ocnn_build_params* prm,
                           void* workspace, size_t workspace_bytes, ocnn_octree_meta* meta,
                           void* stream) {
  using namespace ocnn;
  if (int s = check_args(pts, prm, "ocnn_octree_build_plan")) return s;
  OCNN_REQUIRE(workspace && meta, "ocnn_octree_build_plan: null workspace or meta");
  const int64_t n = pts->offsets_host[pts->batch];
  OCNN_REQUIRE(n < (1LL << 31), "ocnn_octree_build_plan: too many points");
  const Layout L = make_layout(n, pts->batch, prm->depth, prm->full_depth);
  if (workspace_bytes < L.total)
    return fail(OCNN_ERR_CAPACITY, "ocnn_octree_build_plan: workspace of %zu bytes, need %zu",
                workspace_bytes, L.total);
  static thread_local HostCounts host_counts;
  int* counts = host_counts.get();
  if (counts == nullptr)
    return fail(OCNN_ERR_CUDA, "ocnn_octree_build_plan: no pinned memory for the node counts");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  uint8_t* ws = static_cast<uint8_t*>(workspace);

  EncodeArgs ea;
  ea.table = reinterpret_cast<const CloudRef*>(ws + L.off_clouds);
  ea.segments = ea.table + pts->batch + 1;
  ea.inline_clouds = pts->batch <= kInlineClouds ? 1 : 0;
  ea.batch = pts->batch; ea.depth = prm->depth; ea.chunk_pts = chunk_points(n);
  ea.mul = cell_scale(prm);
  for (int j = 0; j < 3; ++j) ea.bbmin[j] = prm->bbmin[j];
  std::vector<CloudRef> big(ea.inline_clouds ? 0 : (size_t)pts->batch + 3);
  CloudRef* table = ea.inline_clouds ? ea.clouds : big.data();
  int chunks = 0;
  for (int b = 0; b <= pts->batch; ++b) {
    CloudRef& c = table[b];
    const bool real = b < pts->batch;
    c.xyz = real ? pts->xyz_dev[b] : nullptr;
    c.normal = real && pts->normal_dev ? pts->normal_dev[b] : nullptr;
    c.feat = real && pts->feature_dev ? pts->feature_dev[b] : nullptr;
    c.label = real && pts->label_dev ? pts->label_dev[b] : nullptr;
    c.offset = pts->offsets_host[b];
    c.chunk0 = chunks;
    c.pad = 0;
    if (real) chunks += ceil_div(pts->offsets_host[b + 1] - pts->offsets_host[b], ea.chunk_pts);
  }
  if (L.segments != L.batch) {           // one segment of all clouds (by_cloud: more than ride along)
    chunks = ceil_div(n, ea.chunk_pts);
    for (int e = 0; e < 2; ++e) {
      CloudRef& c = big[pts->batch + 1 + e];
      memset(&c, 0, sizeof(c));
      c.offset = e == 0 ? 0 : n;
      c.chunk0 = e == 0 ? 0 : chunks;
    }
  }
  // (pageable source: the runtime stages it before returning, so `big` may go out of scope)
  if (!ea.inline_clouds)
    OCNN_CUDA_OK(cudaMemcpyAsync(ws + L.off_clouds, big.data(), sizeof(CloudRef) * big.size(),
                                 cudaMemcpyHostToDevice, st));
  int s;
  if (one_cta(L)) {
    s = small_build(ea, L, ws, counts, st);
  } else {
    OCNN_CUDA_OK(cudaMemsetAsync(ws + L.off_counts, 0, L.zero_bytes, st));
    s = L.key_bytes == 4 ? sort_and_unique<uint32_t>(ea, L, chunks, ws, counts, st)
                         : sort_and_unique<uint64_t>(ea, L, chunks, ws, counts, st);
  }
  if (s != OCNN_OK) return s;
  OCNN_CUDA_OK(cudaStreamSynchronize(st));

  fill_static_meta(pts, prm, meta);
  const int D = prm->depth, F = prm->full_depth, B = pts->batch;
  for (int d = 0; d <= D; ++d) {
    if (d <= F) {
      meta->nnum[d] = B << (3 * d);
      meta->nnum_nempty[d] = d < F ? meta->nnum[d] : (D > F ? counts[F] : 0);
    } else {
      meta->nnum[d] = 8 * counts[d - 1];
      meta->nnum_nempty[d] = counts[d];
    }
  }
  for (int d = F; d <= D; ++d)
    OCNN_REQUIRE(counts[d] > 0 && (int64_t)counts[d] <= L.cap[d],
                 "ocnn_octree_build_plan: inconsistent node count %d at level %d", counts[d], d);
  finish_meta(meta);
  OCNN_REQUIRE(meta->ptr_dis[OCNN_PROP_COUNT] < (1LL << 31),
               "ocnn_octree_build_plan: octree of %lld bytes exceeds the format's 2 GiB limit",
               (long long)meta->ptr_dis[OCNN_PROP_COUNT]);
  return OCNN_OK;
}

int ocnn_octree_build_emit(const ocnn_points_batch* pts, const ocnn_build_params* prm,
                           const ocnn_octree_meta* meta, void* workspace, size_t workspace_bytes,
                           void* out, size_t out_bytes, void* header_host_out, void* stream) {
  using namespace ocnn;
  if (int s = check_args(pts, prm, "ocnn_octree_build_emit")) return s;
  OCNN_REQUIRE(workspace && meta && out, "ocnn_octree_build_emit: null argument");
  const int64_t n = pts->offsets_host[pts->batch];
  const Layout L = make_layout(n, pts->batch, prm->depth, prm->full_depth);
  if (workspace_bytes < L.total)
    return fail(OCNN_ERR_CAPACITY, "ocnn_octree_build_emit: workspace too small");
  if ((int64_t)out_bytes < meta->ptr_dis[OCNN_PROP_COUNT])
    return fail(OCNN_ERR_CAPACITY, "ocnn_octree_build_emit: output of %zu bytes, need %lld",
                out_bytes, (long long)meta->ptr_dis[OCNN_PROP_COUNT]);
  uint8_t hdr[OCNN_HEADER_BYTES];
  HeaderExtras ex;
  ex.adp_depth = prm->adp_depth;
  ex.th_distance = prm->th_distance;
  ex.th_normal = prm->th_normal;
  for (int j = 0; j < 3; ++j) { ex.bbmin[j] = prm->bbmin[j]; ex.bbmax[j] = prm->bbmax[j]; }
  write_header(meta, ex, hdr);
  if (header_host_out) memcpy(header_host_out, hdr, OCNN_HEADER_BYTES);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  uint8_t* o = static_cast<uint8_t*>(out);
  const int s = L.key_bytes == 4 ? emit_impl<uint32_t>(pts, prm, meta, L, ws, o, hdr, st)
                                 : emit_impl<uint64_t>(pts, prm, meta, L, ws, o, hdr, st);
  if (s != OCNN_OK) return s;
  if (prm->merged) return ocnn_calc_neigh(out, meta, stream);
  return OCNN_OK;
}

}  // extern "C"
