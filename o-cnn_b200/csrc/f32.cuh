// What the fp32 kernels on the tensor cores share (conv_f32.cu, conv_f32_wgrad.cu): the three-part
// representation, its row layout, and the swizzled operand tiles.
#pragma once

#include "tc.cuh"

namespace ocnn {
namespace {

constexpr int kF32Rows = 128;                    // tile rows = TMEM lanes
constexpr int kF32K = 32;                        // K values per K-block: one 64-byte row per part
constexpr int kF32PartA = kF32Rows * 64;         // bytes of one part's A tile
constexpr int kF32Threads = 320;
constexpr int kF32TableStride = 132;             // ints between taps in the neighbour table: the lanes'
                                                 // 16-byte reads of different taps spread over the banks

// Accumulation.  The tensor core cuts a sum to fp32 after every instruction instead of rounding it, a
// bias of about 2^-27 of the running sum each time (measured on positive data: 1.2e-6 after the 54
// instructions of 32 channels x 27 taps, where a chain of rounded FMAs is off by 4e-7).  So no
// accumulator runs for more than kChunk K-blocks: the high product's accumulator is double
// buffered, the epilogue warps drain the finished one into registers (rounded additions) while the
// other fills, and the chains stay short enough to be at least as accurate as the FMAs.  The two
// accumulators of the small products are 2^-8 of the sum and below and run through.
constexpr int kChunk = 8;                  // K-blocks per chunk: 16 accumulations

// 64-byte-swizzled K-major operand: 8-row groups of 512 bytes, 16-byte chunk c of row r at
// c ^ ((r >> 1) & 3); layout type SWIZZLE_64B = 4.
__device__ __forceinline__ uint64_t smem_desc_sw64(uint32_t addr) {
  return (uint64_t)((addr & 0x3ffffu) >> 4) | (1ull << 16) | ((uint64_t)(512 >> 4) << 32) |
         (1ull << 46) | (4ull << 61);
}

// The three bf16 parts of v.  Rounding to nearest keeps the dropped products small and of either
// sign; a value that would round up to infinity is cut instead, and an infinity or NaN stays in the
// high part alone.
__device__ __forceinline__ void split3(float v, uint16_t& hi, uint16_t& mid, uint16_t& lo) {
  __nv_bfloat16 h = __float2bfloat16(v);
  uint16_t hb = __bfloat16_as_ushort(h);
  mid = 0;
  lo = 0;
  if ((hb & 0x7f80u) == 0x7f80u) {
    if ((__float_as_uint(v) & 0x7f800000u) == 0x7f800000u) { hi = hb; return; }
    hb = (uint16_t)(__float_as_uint(v) >> 16);
    h = __ushort_as_bfloat16(hb);
  }
  hi = hb;
  const float r1 = v - __bfloat162float(h);
  const __nv_bfloat16 m = __float2bfloat16(r1);
  mid = __bfloat16_as_ushort(m);
  lo = __bfloat16_as_ushort(__float2bfloat16(r1 - __bfloat162float(m)));
}

// Chunk i of a [C, H] (or node-major [H, C]) fp32 tensor as parts: rows of 6 Cp bytes, per block of 32
// channels [high | middle | low].  One thread per (8-channel chunk, node): eight reads and three 16-byte stores.  Of a
// channel-major tensor a warp takes 8 nodes by 4 chunks: whole 32-byte sectors on either side, 64 contiguous bytes per
// part and node (32 nodes of one chunk wrote half sectors 6 Cp bytes apart: 64 channels x 218 k rows 77 us, 32 so).
__device__ __forceinline__ void split_chunk(const float* __restrict__ x, long long h, int c8, long long rows,
                                            int channels, int node_major, uint4 (&part)[3]) {
  float v[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int c = c8 * 8 + j;
    v[j] = (c < channels && h < rows) ? (node_major ? x[h * channels + c] : x[(long long)c * rows + h]) : 0.f;
  }
  uint32_t w[3][4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    uint16_t p0[3], p1[3];
    split3(v[2 * j], p0[0], p0[1], p0[2]);
    split3(v[2 * j + 1], p1[0], p1[1], p1[2]);
#pragma unroll
    for (int q = 0; q < 3; ++q) w[q][j] = (uint32_t)p0[q] | ((uint32_t)p1[q] << 16);
  }
#pragma unroll
  for (int q = 0; q < 3; ++q) part[q] = make_uint4(w[q][0], w[q][1], w[q][2], w[q][3]);
}

// (chunk, node) number i of a channel-major tensor: blocks of up to four chunks, nodes, chunks of the block.
__device__ __forceinline__ void chunk_of_block(long long i, long long rows, int chunks, int& c8, long long& h) {
  const int block = (int)(i / (4 * rows));
  const uint32_t left = (uint32_t)min(4, chunks - 4 * block);
  const long long rest = i - 4 * rows * block;
  h = left == 4 ? rest >> 2 : rest / left;
  c8 = 4 * block + (int)(rest - h * left);
}

__device__ __forceinline__ void split_rows(const float* __restrict__ x, uint8_t* __restrict__ xs, long long i,
                                           long long rows, int channels, int cp, int node_major) {
  const int chunks = cp >> 3;
  long long h;
  int c8;
  if (node_major) { h = i / chunks; c8 = (int)(i - h * chunks); }
  else chunk_of_block(i, rows, chunks, c8, h);
  uint4 part[3];
  split_chunk(x, h, c8, rows, channels, node_major, part);
  const int block = c8 >> 2, width = min(4, chunks - 4 * block) * 16;
  uint8_t* dst = xs + h * ((long long)cp * 6) + block * 192 + (c8 & 3) * 16;
#pragma unroll
  for (int q = 0; q < 3; ++q) *reinterpret_cast<uint4*>(dst + q * width) = part[q];
}

// The sum of all products from that of the high ones and those of the small ones.  A sum that is infinite
// or NaN is so because of its operands (or has overflowed) and the high products alone say which, as a chain of fp32
// multiply-adds would: the small ones hold inf * 0 there (the lower parts of a value that bf16 holds are 0)
// and infinities of either sign.  What is left: an infinity times a value below 2^-134, whose high part
// is 0, gives NaN instead of an infinity.
__device__ __forceinline__ float join_products(float high, float mid, float low) {
  return fabsf(high) < __int_as_float(0x7f800000) ? high + (low + mid) : high;
}

// Offset of 16-byte chunk cc (of cpt per row) of part q in such a row: base + q * width.
__device__ __forceinline__ void chunk_place(int cc, int cpt, uint32_t& base, uint32_t& width) {
  const uint32_t block = (uint32_t)cc >> 2;
  width = (uint32_t)min(4, cpt - 4 * (int)block) * 16u;
  base = block * 192u + ((uint32_t)cc & 3u) * 16u;
}

// Blocks of `npad` rows in a weight image: [Bh | Bm | Bl], and Bh once more where Ah takes all of them
// in one instruction (3 N <= 256 columns; see the kernel).
__host__ __device__ constexpr int f32_stacks(int npad) { return 3 * npad <= 256 ? 4 : 3; }

}  // namespace
}  // namespace ocnn
