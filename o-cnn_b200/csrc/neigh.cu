// Neighbour table: for every sibling group of a level, the 4x4x4 block of node indices around it.
//
// Algorithmic traffic of a split level d: read child[d-1] (4 B/node) and neigh[d-1] (32 B/node),
// write neigh[d] (32 B/node): the kernels below are HBM-bound integer kernels; each warp writes
// 128 contiguous bytes, every lookup inside a parent's block hits one 256-byte line.
#include "common.cuh"

namespace ocnn {
namespace {

__device__ __forceinline__ unsigned spread3(unsigned v) {
  // bit i of v -> bit 3i (v < 2^10 is enough: full levels never exceed depth 10 in practice)
  unsigned r = 0;
#pragma unroll
  for (int i = 0; i < 10; ++i) r |= ((v >> i) & 1u) << (3 * i);
  return r;
}

__device__ __forceinline__ unsigned gather3(unsigned key) {
  unsigned r = 0;
#pragma unroll
  for (int i = 0; i < 10; ++i) r |= ((key >> (3 * i)) & 1u) << i;
  return r;
}

// Full level: one thread per output int; out[(n*per + g)*8 + j], j = (X<<4)|(Y<<2)|Z.
// Restates calc_neigh_cpu(neigh, depth, batch), octree/octree/octree_nn.cpp:382-424.
__global__ void neigh_full_kernel(int* __restrict__ out, int depth, long long per,
                                  long long total) {
  grid_dependency_wait();       // launched as a programmatic dependent: see common.cuh
  const int side = 1 << depth;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int j = (int)(i & 63);
    const long long blk = i >> 6;                  // sibling group over the whole batch
    const long long n = (blk << 3) / per;          // batch item
    const unsigned g = (unsigned)((blk << 3) - n * per);   // first node of the group
    const int x = (int)gather3(g >> 2) + (j >> 4) - 1;
    const int y = (int)gather3(g >> 1) + ((j >> 2) & 3) - 1;
    const int z = (int)gather3(g) + (j & 3) - 1;
    int v = -1;
    if (x >= 0 && y >= 0 && z >= 0 && x < side && y < side && z < side)
      v = (int)((spread3(x) << 2) | (spread3(y) << 1) | spread3(z)) + (int)(n * per);
    out[i] = v;
  }
  grid_dependency_trigger();    // at the end: the successor's blocks should not sit on SM slots early
}

// Levels 0 .. full of a batch octree in one launch: level d's table is out + 8 * 8^d-node prefix, i.e.
// the levels lie one behind the other. Level 0 has no neighbour table; the reference leaves its slot
// zero-filled (merge_octrees.cpp:108-112 resizes a fresh vector, the loop at :184 starts at d = 1).
__global__ void neigh_full_levels_kernel(int* __restrict__ out, int batch, int full, long long total) {
  grid_dependency_wait();       // launched as a programmatic dependent: see common.cuh
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    long long at = i;
    int depth = 0;
    while (depth < full && at >= 8LL * batch << (3 * depth)) { at -= 8LL * batch << (3 * depth); ++depth; }
    if (depth == 0) { out[i] = 0; continue; }
    const int per = 1 << (3 * depth), side = 1 << depth;
    const int j = (int)(at & 63);
    const long long node = at >> 6 << 3;           // first node of the sibling group, over the batch
    const int n = (int)(node / per);
    const unsigned g = (unsigned)(node - (long long)n * per);
    const int x = (int)gather3(g >> 2) + (j >> 4) - 1;
    const int y = (int)gather3(g >> 1) + ((j >> 2) & 3) - 1;
    const int z = (int)gather3(g) + (j & 3) - 1;
    int v = -1;
    if (x >= 0 && y >= 0 && z >= 0 && x < side && y < side && z < side)
      v = (int)((spread3(x) << 2) | (spread3(y) << 1) | spread3(z)) + n * per;
    out[i] = v;
  }
  grid_dependency_trigger();    // at the end: the successor's blocks should not sit on SM slots early
}

// Split level, one warp per sibling group of PARENT nodes.  The eight parents of a group share one
// 4x4x4 neighbour block at their own level, and every entry any of their children's blocks needs
// is "the child group of one of those 64 cells".  So the warp reads the group's 64 neighbour
// entries (256 contiguous bytes) and the 64 child pointers behind them ONCE (two gathers per
// lane), keeps them in shared memory, and then writes the 64-int block of each non-empty parent:
// 8 child gathers per parent instead of the 64 of the one-thread-per-output formulation.
// WIDE (the output on a 16-byte boundary: a level's table starts 12 * batch bytes past one with
// 64-bit keys, so batches of a multiple of four): two parents, z-neighbours, at a time, 16 lanes each,
// a lane writes the four z positions of one (x, y) from one 16-byte read of the parents' block.  A
// quarter of the stores and reads of the other form, one int per lane and store, which was bound
// by instruction issue.  Depth 8 of 64 clouds of 100k points: 190 -> 178 us, 916 MB of DRAM traffic
// at 5.1 TB/s (79 % of a copy).  Restates calc_neigh_cpu(neigh_split, neigh, children,
// node_num), octree/octree/octree_nn.cpp:357-380, with the parent/displacement tables
// (octree_nn.cpp:53-81) in arithmetic form.
constexpr int kNeighWarps = 8;

template <bool WIDE>
__global__ void __launch_bounds__(kNeighWarps * 32) neigh_split_kernel(
    int* __restrict__ out, const int* __restrict__ neigh, const int* __restrict__ child,
    long long ngroups) {
  grid_dependency_wait();       // launched as a programmatic dependent: see common.cuh
  // 8 * child group of each cell of the parents' block, -1 where there is none: an output is that
  // value | octant either way
  __shared__ __align__(16) int cblk[kNeighWarps][64];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // child-level block position j = (x,y,z) in 0..3 -> which parent-level cell (tap, as a
  // (tx<<4)|(ty<<2)|tz code relative to the parent) and which octant inside it; two per lane
  int tapcode[2], oct[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int j = lane + 32 * k;
    const int x = (j >> 4) + 1, y = ((j >> 2) & 3) + 1, z = (j & 3) + 1;
    tapcode[k] = ((x >> 1) << 4) | ((y >> 1) << 2) | (z >> 1);
    oct[k] = ((x & 1) << 2) | ((y & 1) << 1) | (z & 1);
  }
  // WIDE: the lane's (x, y) and half = the z bit of its parent
  const int half = lane >> 4, wx = ((lane >> 2) & 3) + 1, wy = (lane & 3) + 1;
  const int rowcode = ((wx >> 1) << 4) | ((wy >> 1) << 2), rowoct = ((wx & 1) << 2) | ((wy & 1) << 1);
  // Three stages in flight per warp: the block of the group after next is requested, then the child
  // pointers behind the next group's block, then this group's tables are written.  (One group at a
  // time was a chain of two reads per 700 bytes written: 3.7 TB/s where the writes alone go at 7.4.)
  const long long stride = (long long)gridDim.x * kNeighWarps;
  const long long first = blockIdx.x * (long long)kNeighWarps + warp;
  auto cells = [&](long long g, int (&cell)[2], int& mine) {
    cell[0] = cell[1] = mine = -1;
    if (g >= ngroups) return;
    const int* blk = neigh + (g << 6);
    cell[0] = blk[lane];
    cell[1] = blk[lane + 32];
    if (lane < 8) mine = child[(g << 3) + lane];     // the eight parents themselves
  };
  auto kids = [&](const int (&cell)[2], int (&kid)[2]) {
#pragma unroll
    for (int k = 0; k < 2; ++k) kid[k] = cell[k] >= 0 ? child[cell[k]] : -1;
  };
  int cell[2], kid[2], mine, mine_next;
  cells(first, cell, mine);
  kids(cell, kid);
  cells(first + stride, cell, mine_next);
  for (long long g = first; g < ngroups; g += stride) {
#pragma unroll
    for (int k = 0; k < 2; ++k) cblk[warp][lane + 32 * k] = kid[k] >= 0 ? kid[k] << 3 : -1;
    __syncwarp();
    kids(cell, kid);
    int mine_after;
    cells(g + 2 * stride, cell, mine_after);
    if constexpr (WIDE) {
#pragma unroll
      for (int pair = 0; pair < 4; ++pair) {
        const int l0 = __shfl_sync(0xffffffffu, mine, 2 * pair + half);
        if (l0 < 0) continue;                                   // empty parent: no block
        const int4 c = *reinterpret_cast<const int4*>(&cblk[warp][rowcode + ((pair & 2) << 3) + ((pair & 1) << 2)]);
        const int lo = half ? c.y : c.x, mid = half ? c.z : c.y, hi = half ? c.w : c.z;
        *reinterpret_cast<int4*>(out + ((long long)l0 << 6) + ((lane & 15) << 2)) =
            make_int4(lo | rowoct | 1, mid | rowoct, mid | rowoct | 1, hi | rowoct);
      }
    } else {
#pragma unroll
      for (int o = 0; o < 8; ++o) {
        const int l0 = __shfl_sync(0xffffffffu, mine, o);
        if (l0 < 0) continue;                                     // empty parent: no block
        const int octcode = ((o & 4) << 2) | ((o & 2) << 1) | (o & 1);
        int* dst = out + ((long long)l0 << 6);
#pragma unroll
        for (int k = 0; k < 2; ++k) dst[lane + 32 * k] = cblk[warp][tapcode[k] + octcode] | oct[k];
      }
    }
    mine = mine_next;
    mine_next = mine_after;
    __syncwarp();
  }
  grid_dependency_trigger();    // at the end: the successor's blocks should not sit on SM slots early
}

}  // namespace
}  // namespace ocnn

extern "C" {

int ocnn_calc_neigh_full(int32_t* neigh, int depth, int batch, void* stream) {
  using namespace ocnn;
  OCNN_REQUIRE(neigh != nullptr, "ocnn_calc_neigh_full: null output");
  OCNN_REQUIRE(depth >= 1 && depth <= 10 && batch >= 1, "ocnn_calc_neigh_full: depth %d / batch %d "
               "out of range", depth, batch);
  const long long per = 1LL << (3 * depth);
  const long long total = per * batch * 8;
  OCNN_REQUIRE(per * batch < (1LL << 31), "ocnn_calc_neigh_full: level too large for int32 indices");
  OCNN_CUDA_OK(launch_chained(neigh_full_kernel, dim3(grid_for(total, 256)), dim3(256), 0, static_cast<cudaStream_t>(stream), neigh, depth, per, total));
  OCNN_LAUNCH_OK("neigh_full_kernel");
  return OCNN_OK;
}

int ocnn_calc_neigh_split(int32_t* neigh_child, const int32_t* neigh, const int32_t* child,
                          int nnum_parent, void* stream) {
  using namespace ocnn;
  if (nnum_parent == 0) return OCNN_OK;
  OCNN_REQUIRE(neigh_child && neigh && child, "ocnn_calc_neigh_split: null pointer");
  OCNN_REQUIRE(nnum_parent > 0 && nnum_parent % 8 == 0,
               "ocnn_calc_neigh_split: parent level must hold whole sibling groups (got %d nodes)",
               nnum_parent);
  const long long ngroups = nnum_parent / 8;
  const bool wide = (uintptr_t)neigh_child % 16 == 0;
  OCNN_CUDA_OK(launch_chained(wide ? neigh_split_kernel<true> : neigh_split_kernel<false>,
                              dim3(grid_for(ngroups, kNeighWarps, 16)), dim3(kNeighWarps * 32), 0,
                              static_cast<cudaStream_t>(stream), neigh_child, neigh, child, ngroups));
  OCNN_LAUNCH_OK("neigh_split_kernel");
  return OCNN_OK;
}

int ocnn_calc_neigh(void* octree_dev, const ocnn_octree_meta* m, void* stream) {
  using namespace ocnn;
  OCNN_REQUIRE(octree_dev != nullptr && m != nullptr, "ocnn_calc_neigh: null argument");
  OCNN_REQUIRE(m->channels[OCNN_PROP_NEIGH] == 8 && m->locations[OCNN_PROP_NEIGH] == -1,
               "ocnn_calc_neigh: the octree has no neighbour block (not a merged batch)");
  OCNN_REQUIRE(m->channels[OCNN_PROP_CHILD] == 1 && m->locations[OCNN_PROP_CHILD] == -1,
               "ocnn_calc_neigh: the octree has no child block");
  uint8_t* base = static_cast<uint8_t*>(octree_dev);
  const int full = m->full_depth < m->depth ? m->full_depth : m->depth;
  OCNN_REQUIRE(full >= 0 && full <= 10, "ocnn_calc_neigh: full depth %d out of range", full);
  long long total = 0;
  for (int d = 0; d <= full; ++d) {
    OCNN_REQUIRE(m->nnum[d] == (long long)m->batch_size << (3 * d), "ocnn_calc_neigh: level %d is not full", d);
    total += 8LL * m->nnum[d];
  }
  int* all = reinterpret_cast<int*>(base + ocnn_prop_offset(m, OCNN_PROP_NEIGH, 0));
  OCNN_CUDA_OK(launch_chained(neigh_full_levels_kernel, dim3(grid_for(total, 256)), dim3(256), 0,
                              static_cast<cudaStream_t>(stream), all, m->batch_size, full, total));
  OCNN_LAUNCH_OK("neigh_full_levels_kernel");
  for (int d = full + 1; d <= m->depth; ++d) {
    const int s = ocnn_calc_neigh_split(
        reinterpret_cast<int32_t*>(base + ocnn_prop_offset(m, OCNN_PROP_NEIGH, d)),
        reinterpret_cast<const int32_t*>(base + ocnn_prop_offset(m, OCNN_PROP_NEIGH, d - 1)),
        reinterpret_cast<const int32_t*>(base + ocnn_prop_offset(m, OCNN_PROP_CHILD, d - 1)), m->nnum[d - 1],
        stream);
    if (s != OCNN_OK) return s;
  }
  return OCNN_OK;
}

}  // extern "C"
