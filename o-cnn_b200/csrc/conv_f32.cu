// Octree convolution in fp32 on the tensor cores (tcgen05 + TMEM): every fp32 value is carried as the sum
// of three bf16 values and the product as six bf16 products accumulated in fp32 (a published method: G. Henry,
// P. T. P. Tang, A. Heinecke, "Leveraging the bfloat16 Artificial Intelligence Datatype For Higher-Precision
// Computations", 2019).
//
//     x = xh + xm + xl,  w = wh + wm + wl       (each part the rounded rest of the ones before: 8 bits
//                                                of significand each, together the 24 of an fp32)
//     x * w = xh wh  +  (xh wm + xm wh)  +  (xh wl + xm wm + xl wh)  +  terms below 2^-24 |x w|
//
// The three groups go to accumulators of their own, so a small term is never rounded against a
// large partial sum; the epilogue adds them smallest first.
//
// Two launches: conv_f32_prepare_kernel rewrites the input rows node-major and split (per row and
// block of 32 channels the three parts side by side; Cin rounded up to 8) and packs the weights;
// conv_f32_kernel is the implicit GEMM of conv_tc.cu on K-blocks of 32: the stage of a K-block
// holds three A tiles [128 rows x 64 bytes] (the gathered rows' high, middle and low parts) and one B image of the
// weights' parts stacked, so that
//     Ah x [Bh | Bm | Bl] -> [D0 | D1 | D2],   Am x [Bh | Bm] -> [D1 | D2],   Al x Bh -> D2
// are three instructions per 16 K values (four where 3 N columns exceed an instruction's 256).
//
// Bound: the L2 -> SM gather (6 Cin bytes per node and tap at about 37 bytes per clock and SM) up to
// 64 output channels, gather and tensor pipe alike at 128.  The CUDA-core kernel (conv_simt.cu)
// ran these layers at 14-15 TFLOP/s.
#include "f32.cuh"

namespace ocnn {
namespace {

struct F32Args {
  const uint8_t* xs;       // split input rows [h_in][3][cp] bf16
  const uint8_t* wp;       // packed weights, per slice and K-block a [3 * npad rows x 64 bytes] image
  float* y;
  float* partial;          // K-split launches: one fp32 copy of y per split, reduced afterwards
  const int* neigh;
  const int* child;
  const int* ichild;
  int h_in, h_out, cp, cout, npad, T, stride, identity, up;
  int tiles, slices, splits, nkb, kb_per_split, stages, tmem_cols, node_major;
  int vec4;                // node-major rows of whole float4 on a 16-byte boundary
  long long y_elems;
  ChannelAffine aff;
  const float* residual;
  int relu;
  int* status;
  signed char tap[27];
};

struct PrepareArgs {
  const float* x;
  uint8_t* xs;
  const float* w;
  uint8_t* wp;
  int h_in, cin, cp, node_major;
  int cout, npad, T, nkb, transposed;
  long long x_items;       // (node, 8-channel chunk) pairs
  int x_blocks;            // blocks that split x; the rest pack the weights
  long long w_items;       // (slice, K-block, column, 8-value chunk) quadruples
};

// Input rows and weights, split, in one launch.  A pure stream: 4 bytes read and 6 written per value.
__global__ void __launch_bounds__(256) conv_f32_prepare_kernel(const PrepareArgs a) {
  grid_dependency_trigger();
  grid_dependency_wait();
  if ((int)blockIdx.x < a.x_blocks) {
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= a.x_items) return;
    split_rows(a.x, a.xs, i, a.h_in, a.cin, a.cp, a.node_major);
    return;
  }
  const long long i = (long long)(blockIdx.x - a.x_blocks) * 256 + threadIdx.x;
  if (i >= a.w_items) return;
  const int c = (int)(i & 3);                       // 16-byte chunk of the K-block's 64-byte row
  long long r = i >> 2;
  const int n = (int)(r % a.npad);
  r /= a.npad;
  const int kb = (int)(r % a.nkb), slice = (int)(r / a.nkb);
  const int g = kb * 4 + c, cpt = a.cp >> 3;        // K walks tap-major in chunks of 8 channels
  const int t = g / cpt, ci0 = (g - t * cpt) * 8;
  const int co = slice * a.npad + n;
  uint32_t part[3][4] = {};
  if (t < a.T && co < a.cout) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int ci = ci0 + j;
      if (ci >= a.cin) break;
      const float v = a.transposed ? a.w[((long long)ci * a.cout + co) * a.T + t]
                                   : a.w[((long long)co * a.cin + ci) * a.T + t];
      uint16_t p[3];
      split3(v, p[0], p[1], p[2]);
#pragma unroll
      for (int q = 0; q < 3; ++q) part[q][j >> 1] |= (uint32_t)p[q] << (16 * (j & 1));
    }
  }
  const int stacks = f32_stacks(a.npad);
  uint8_t* dst = a.wp + ((long long)slice * a.nkb + kb) * (a.npad * 64 * stacks);
#pragma unroll
  for (int b = 0; b < 4; ++b) {                     // high, middle, low (and high again)
    if (b >= stacks) break;
    const int q = b == 3 ? 0 : b, row = b * a.npad + n;
    *reinterpret_cast<uint4*>(dst + row * 64 + ((c ^ ((row >> 1) & 3)) << 4)) =
        make_uint4(part[q][0], part[q][1], part[q][2], part[q][3]);
  }
}

// Persistent: a CTA walks (tile, slice, split) items.  Warps 0-3 fill the item's neighbour table and
// gather, warps 4-7 drain the accumulators and store, warp 8 owns TMEM and issues the MMAs, warp 9
// streams the weight images; two CTAs share an SM up to 64 columns, so that one's table look-ups
// (three dependent reads) run under the other's copies.  The ring and its phases run on across items.
// TMEM columns: chunk accumulators D0 at [0, N) and [3N, 4N), the small products' D1, D2 between them.
template <int NG>                          // N / 16
__global__ void __launch_bounds__(kF32Threads, NG <= 4 ? 2 : 1) conv_f32_kernel(const F32Args a) {
  constexpr int N = 16 * NG;
  constexpr bool kOne = f32_stacks(N) == 4;  // Ah meets all three weight parts in one instruction
  constexpr int kBytesB = N * 64 * f32_stacks(N);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* sA = smem;                                    // stage s: high, middle, low tiles
  uint8_t* sB = sA + a.stages * (3 * kF32PartA);
  int* nbr = reinterpret_cast<int*>(sB + a.stages * kBytesB);
  float2* s_aff = reinterpret_cast<float2*>(nbr + a.T * kF32TableStride);   // [slices * N]
  uint64_t* full = reinterpret_cast<uint64_t*>(s_aff + a.slices * N);
  uint64_t* empty = full + a.stages;
  uint64_t* cfull = empty + a.stages;                    // chunk accumulator b is complete
  uint64_t* cempty = cfull + 2;                          // ... has been drained
  uint64_t* dempty = cempty + 2;                         // the small products' accumulators have been read
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(dempty + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int s = 0; s < a.stages; ++s) {
      mbar_init(smem_u32(&full[s]), kF32Rows + 1);
      mbar_init(smem_u32(&empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&cfull[b]), 1);
      mbar_init(smem_u32(&cempty[b]), kF32Rows);
    }
    mbar_init(smem_u32(dempty), kF32Rows);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 8) tmem_alloc(tmem_holder, a.tmem_cols);
  grid_dependency_wait();
  for (int n = tid; n < a.slices * N; n += kF32Threads)
    s_aff[n] = n < a.cout ? channel_affine(a.aff, n) : make_float2(1.f, 0.f);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_holder;

  // item -> (tile, slice, split): the slices and splits of a tile are neighbours in time and reuse
  // its gathered rows in L2
  const int per_tile = a.slices * a.splits;
  const int items = a.tiles * per_tile;
  auto item_split = [&](int item) { return item % a.splits; };
  auto item_slice = [&](int item) { return (item / a.splits) % a.slices; };
  auto item_nkb = [&](int item) { return min(a.kb_per_split, a.nkb - item_split(item) * a.kb_per_split); };

  if (warp < 4) {
    // ---------------- neighbour table + A gather ----------------
    // lane = (row of eight, 16-byte chunk of the K-block's 64 bytes), part by part.  (All 192 bytes
    // of a row in a row of lanes touches fewer lines, but a returning line's two parts then meet in
    // the same shared-memory banks: 213 us against 194 for 32 -> 64 at 217 k nodes.)
    const int c = lane & 3, rr = lane >> 2;
    const int cpt = a.cp >> 3;
    const uint32_t row_bytes = (uint32_t)a.cp * 6u;
    const int* my_idx = nbr + warp * 32 + rr * 4;
    // rows r, r + 8, r + 16, r + 24 of a warp sit side by side in the table; a warp reads only the 32
    // rows it has written
    const int slot = (tid & ~31) + ((tid & 7) << 2) + ((tid >> 3) & 3);
    bool alive = true;
    int s = 0, filled = -1;
    uint32_t pe = 1;
    ZeroRows<4> zeros;
    long long gk = 0;
    for (int item = blockIdx.x; item < items; item += gridDim.x) {
      const int tile = item / per_tile;
      if (tile != filled) {
        filled = tile;
        const int h = tile * kF32Rows + tid;
        const bool live = h < a.h_out;
        __syncwarp();
        const int hn = (a.ichild != nullptr && live) ? a.ichild[h] : h;
        if (a.identity) {
          nbr[slot] = live ? h : -1;
        } else if (a.up) {
#pragma unroll 1
          for (int t = 0; t < a.T; ++t) {
            const int code = a.tap[t];
            nbr[t * kF32TableStride + slot] =
                live ? up_source_group(a.neigh, hn, (code >> 4) * 9 + ((code >> 2) & 3) * 3 + (code & 3)) : -1;
          }
        } else {
          const int oct_code = ((hn & 4) << 2) | ((hn & 2) << 1) | (hn & 1);
          // nine table reads in flight (all 27 unrolled are several KB of code that runs once per
          // tile: its instruction fetches took longer than the reads, 7 k cycles)
#pragma unroll 1
          for (int t0 = 0; t0 < a.T; t0 += 9) {
            int pv[9];
#pragma unroll
            for (int j = 0; j < 9; ++j) {
              const int t = t0 + j;
              pv[j] = -1;
              if (t < a.T && live) {
                const int code = a.tap[t];
                pv[j] = a.neigh[a.stride == 2 ? ((long long)hn << 6) + code
                                              : ((long long)(hn >> 3) << 6) + code + oct_code];
              }
            }
            if (a.child != nullptr) {
#pragma unroll
              for (int j = 0; j < 9; ++j)
                if (pv[j] >= 0) pv[j] = a.child[pv[j]];
            }
#pragma unroll
            for (int j = 0; j < 9; ++j)
              if (t0 + j < a.T) nbr[(t0 + j) * kF32TableStride + slot] = pv[j];
          }
        }
        __syncwarp();
      }
      const int kb0 = item_split(item) * a.kb_per_split, nkb = item_nkb(item);
      int t = (kb0 * 4 + c) / cpt, cc = (kb0 * 4 + c) - t * cpt;
      for (int kb = 0; kb < nkb; ++kb, ++gk) {
        int4 p4 = make_int4(-1, -1, -1, -1);
        if (t < a.T) p4 = *reinterpret_cast<const int4*>(my_idx + t * kF32TableStride);
        if (alive && gk >= a.stages)
          alive = mbar_wait(smem_u32(&empty[s]), pe, abort_flag, a.status, kErrEmptyWait);
        if (alive) {
          const uint32_t stage = smem_u32(sA + s * (3 * kF32PartA));
          uint32_t off, width;
          chunk_place(cc, cpt, off, width);
          const int p[4] = {p4.x, p4.y, p4.z, p4.w};
          const uint32_t copies = zeros.copies(s, live_rows<4>(p));
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int row = warp * 32 + 8 * i + rr;
            const uint32_t dst = stage + (uint32_t)row * 64u + (((uint32_t)c ^ (uint32_t)((row >> 1) & 3)) << 4);
            const bool have = p[i] >= 0;
            const uint8_t* src = have ? a.xs + (size_t)p[i] * row_bytes + off : a.xs;
            const uint32_t step = have ? width : 0u, n = have ? 16u : 0u;
            if ((copies >> i) & 1u) {
#pragma unroll
              for (int q = 0; q < 3; ++q) cp_async16(dst + q * kF32PartA, src + q * step, n);
            }
          }
        }
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&full[s]))
                     : "memory");
        if (++s == a.stages) { s = 0; pe ^= 1u; }
        cc += 4;
        while (cc >= cpt) { cc -= cpt; ++t; }
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (warp < 8) {
    // ---------------- drain, epilogue ----------------
    const int q4 = warp & 3;                 // TMEM lane quarter of this warp
    const uint32_t lane_base = tmem_base + ((uint32_t)(q4 * 32) << 16);
    bool alive = true;
    int buf = 0;
    uint32_t ph = 0;
    for (int item = blockIdx.x; item < items && alive; item += gridDim.x) {
      const int nkb = item_nkb(item);
      float acc[N];
#pragma unroll
      for (int j = 0; j < N; ++j) acc[j] = 0.f;
      for (int kb = 0; kb < nkb; kb += kChunk) {
        alive = mbar_wait(smem_u32(&cfull[buf]), ph, abort_flag, a.status, kErrAccumWait);
        alive = __all_sync(0xffffffffu, alive);
        if (!alive) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int g = 0; g < 2 * NG; ++g) {      // eight columns at a time: the sums fill the registers
          uint32_t v[8];
          tmem_ld8(lane_base + (uint32_t)(buf * 3 * N + 8 * g), v);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 8; ++j) acc[8 * g + j] += __uint_as_float(v[j]);
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        mbar_arrive(smem_u32(&cempty[buf]));
        buf ^= 1;
        if (buf == 0) ph ^= 1u;
      }
      if (!alive) break;
#pragma unroll
      for (int g = 0; g < 2 * NG; ++g) {
        uint32_t v1[8], v2[8];
        tmem_ld8(lane_base + (uint32_t)(N + 8 * g), v1);
        tmem_ld8(lane_base + (uint32_t)(2 * N + 8 * g), v2);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[8 * g + j] = join_products(acc[8 * g + j], __uint_as_float(v1[j]), __uint_as_float(v2[j]));
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      mbar_arrive(smem_u32(dempty));

      const int h = (item / per_tile) * kF32Rows + q4 * 32 + lane;
      if (h >= a.h_out) continue;
      const int co_base = item_slice(item) * N;
      float* out = a.partial ? a.partial + item_split(item) * a.y_elems : a.y;
      const bool finish = a.partial == nullptr;
      if (a.vec4) {
        const long long at0 = (long long)h * a.cout + co_base;
#pragma unroll
        for (int j = 0; j < N; j += 4) {
          if (co_base + j >= a.cout) break;
          float4 v = make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
          if (finish) {
            const float2* af = s_aff + co_base + j;
            v.x = fmaf(v.x, af[0].x, af[0].y); v.y = fmaf(v.y, af[1].x, af[1].y);
            v.z = fmaf(v.z, af[2].x, af[2].y); v.w = fmaf(v.w, af[3].x, af[3].y);
            if (a.residual) {
              const float* r = a.residual + at0 + j;
              v.x += r[0]; v.y += r[1]; v.z += r[2]; v.w += r[3];
            }
            if (a.relu) { v.x = fmaxf(v.x, 0.f); v.y = fmaxf(v.y, 0.f); v.z = fmaxf(v.z, 0.f); v.w = fmaxf(v.w, 0.f); }
          }
          *reinterpret_cast<float4*>(out + at0 + j) = v;
        }
      } else {
        // channel-major: a warp's store is 32 consecutive nodes of one channel
        const long long step = a.node_major ? 1 : a.h_out;
        long long at = a.node_major ? (long long)h * a.cout + co_base : (long long)co_base * a.h_out + h;
#pragma unroll
        for (int j = 0; j < N; ++j) {
          if (co_base + j >= a.cout) break;
          float v = acc[j];
          if (finish) {
            v = fmaf(v, s_aff[co_base + j].x, s_aff[co_base + j].y);
            if (a.residual) v += a.residual[at];
            if (a.relu) v = fmaxf(v, 0.f);
          }
          out[at] = v;
          at += step;
        }
      }
    }
  } else if (warp == 8) {
    // ---------------- MMA issue: one thread ----------------
    if (lane == 0) {
      const uint32_t idesc0 = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kF32Rows >> 4) << 24);
      constexpr uint32_t n1 = (uint32_t)(N >> 3) << 17, n2 = (uint32_t)(2 * N >> 3) << 17,
                         n3 = (uint32_t)(3 * N >> 3) << 17;
      bool alive = true;
      int s = 0, buf = 0, it = 0;
      uint32_t pf = 0, pc = 1;
      for (int item = blockIdx.x; item < items && alive; item += gridDim.x, ++it) {
        const int nkb = item_nkb(item);
        if (it > 0) alive = mbar_wait(smem_u32(dempty), (uint32_t)(it - 1) & 1u, abort_flag, a.status, kErrAccumWait);
        for (int kb = 0; kb < nkb && alive; ++kb) {
          if (kb % kChunk == 0) {
            alive = mbar_wait(smem_u32(&cempty[buf]), pc, abort_flag, a.status, kErrAccumWait);
            if (!alive) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          }
          alive = mbar_wait(smem_u32(&full[s]), pf, abort_flag, a.status, kErrFullWait);
          if (!alive) break;
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t aa = smem_u32(sA + s * (3 * kF32PartA)), bb = smem_u32(sB + s * kBytesB);
          const uint32_t d1 = tmem_base + N, d2 = tmem_base + 2 * N, d0 = tmem_base + (uint32_t)(buf * 3 * N);
#pragma unroll
          for (int k2 = 0; k2 < 2; ++k2) {
            const uint64_t ah = smem_desc_sw64(aa + k2 * 32), am = smem_desc_sw64(aa + kF32PartA + k2 * 32),
                           al = smem_desc_sw64(aa + 2 * kF32PartA + k2 * 32);
            const uint64_t bh = smem_desc_sw64(bb + k2 * 32), bm = smem_desc_sw64(bb + N * 64 + k2 * 32);
            const bool first_of_chunk = kb % kChunk == 0 && k2 == 0, first = kb == 0 && k2 == 0;
            if (kOne && !(first_of_chunk && !first)) {
              // buffer 0: [Bh | Bm | Bl] -> [D0 | D1 | D2]; buffer 1: [Bm | Bl | Bh] -> [D1 | D2 | D0]
              umma_bf16(buf == 0 ? d0 : d1, ah, buf == 0 ? bh : bm, idesc0 | n3, first ? 0u : 1u);
            } else {
              // (a chunk's first instruction clears D0 but not the running sums beside it)
              umma_bf16(d0, ah, bh, idesc0 | n1, first_of_chunk ? 0u : 1u);
              umma_bf16(d1, ah, bm, idesc0 | n2, first ? 0u : 1u);
            }
            umma_bf16(d1, am, bh, idesc0 | n2, 1u);
            umma_bf16(d2, al, bh, idesc0 | n1, 1u);
          }
          umma_commit(smem_u32(&empty[s]));
          if (++s == a.stages) { s = 0; pf ^= 1u; }
          if (kb % kChunk == kChunk - 1 || kb == nkb - 1) {
            umma_commit(smem_u32(&cfull[buf]));
            buf ^= 1;
            if (buf == 0) pc ^= 1u;
          }
        }
      }
      if (!alive) {
        // gave up: leave the MMAs already issued time to retire before TMEM is freed
        for (int w = 0; w < 64; ++w) __nanosleep(1000);
      }
    }
  } else if (lane == 0) {
    // ---------------- weight images ----------------
    bool alive = true;
    int s = 0;
    uint32_t pe = 1;
    long long gk = 0;
    for (int item = blockIdx.x; item < items && alive; item += gridDim.x) {
      const int nkb = item_nkb(item);
      const uint8_t* wp = a.wp + ((long long)item_slice(item) * a.nkb + item_split(item) * a.kb_per_split) * kBytesB;
      for (int kb = 0; kb < nkb && alive; ++kb, ++gk) {
        if (gk >= a.stages)
          alive = mbar_wait(smem_u32(&empty[s]), pe, abort_flag, a.status, kErrWeightWait);
        if (!alive) break;
        const uint32_t bar = smem_u32(&full[s]);
        mbar_arrive_expect_tx(bar, (uint32_t)kBytesB);
        bulk_copy(smem_u32(sB + s * kBytesB), wp + (size_t)kb * kBytesB, (uint32_t)kBytesB, bar);
        if (++s == a.stages) { s = 0; pe ^= 1u; }
      }
    }
    if (!alive) {
      for (int it = 0; it < 64; ++it) __nanosleep(1000);   // copies in flight land before the CTA exits
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 8) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"((uint32_t)a.tmem_cols)
                 : "memory");
  }
}

// Sum of the K splits' partial outputs, then the epilogue.
__global__ void __launch_bounds__(256) conv_f32_reduce_kernel(const float* __restrict__ partial, float* __restrict__ y,
                                                              long long elems, int splits, int cout, int h_out,
                                                              int node_major, const ChannelAffine aff,
                                                              const float* __restrict__ residual, int relu) {
  grid_dependency_trigger();
  grid_dependency_wait();
  for (long long i = blockIdx.x * 256LL + threadIdx.x; i < elems; i += gridDim.x * 256LL) {
    float v = 0.f;
    for (int s = 0; s < splits; ++s) v += partial[s * elems + i];
    const float2 sb = channel_affine(aff, node_major ? (int)(i % cout) : (int)(i / h_out));
    v = fmaf(v, sb.x, sb.y);
    if (residual) v += residual[i];
    if (relu) v = fmaxf(v, 0.f);
    y[i] = v;
  }
}

struct F32Shape {
  int cp, npad, slices, T, nkb, tiles, splits, kb_per_split, stages, tmem_cols, ctas;
  size_t smem, xs_bytes, wp_bytes, partial_bytes;
};

// Launch shape and workspace of a layer; false where the kernel does not serve it.
bool f32_shape(const ocnn_conv_geometry* g, int cin, int cout, const TapList& tl, F32Shape* s) {
  s->T = tl.count;
  s->cp = (cin + 7) / 8 * 8;
  s->nkb = ceil_div((long long)s->T * s->cp, kF32K);
  // output channels in slices of at most 128 (four accumulators of N columns each in TMEM's 512)
  s->slices = ceil_div(cout, 128);
  s->npad = (ceil_div(cout, s->slices) + 15) / 16 * 16;
  s->tiles = ceil_div(g->h_out, kF32Rows);
  // two CTAs share an SM as long as their accumulators fit, i.e. up to 64 columns
  const bool pair = s->npad <= 64;
  const int sms = sm_count();
  const long long ctas = (long long)s->tiles * s->slices;
  const long long room = (long long)sms * (pair ? 2 : 1);
  // A level too small to give every SM its CTAs is also split along K, a chunk or more per split:
  // the sum is finished by a reduction pass.
  s->splits = 1;
  if (2 * ctas <= room) {
    const long long want = room / ctas, most = s->nkb / kChunk;
    s->splits = (int)(want < most ? want : most);
    if (s->splits < 1) s->splits = 1;
  }
  s->kb_per_split = (ceil_div(s->nkb, s->splits) + kChunk - 1) / kChunk * kChunk;
  s->splits = ceil_div(s->nkb, s->kb_per_split);
  s->tmem_cols = 64;
  while (s->tmem_cols < 4 * s->npad) s->tmem_cols *= 2;
  const size_t fixed = 1024 + (size_t)s->T * kF32TableStride * 4 + (size_t)s->slices * s->npad * 8 + 256;
  const size_t stage = 3 * kF32PartA + (size_t)s->npad * 64 * f32_stacks(s->npad);
  const long long items = ctas * s->splits;
  const bool share = pair && items > sms;
  const size_t budget = (share ? 112 : 220) * 1024;
  // (scale and bias of all slices take 8 bytes a channel: beyond about 13 k output channels no ring is left)
  if (fixed + 2 * stage > budget) return false;
  int st = (int)((budget - fixed) / stage);
  if (st > 6) st = 6;
  s->stages = st;
  s->smem = fixed + st * stage;
  // the same number of items (within one) for every CTA
  const long long slots = share ? 2LL * sms : sms;
  s->ctas = ceil_div(items, ceil_div(items, slots));
  auto up = [](size_t v) { return (v + 255) / 256 * 256; };
  s->xs_bytes = up((size_t)g->h_in * s->cp * 6);
  s->wp_bytes = up((size_t)s->slices * s->nkb * s->npad * 64 * f32_stacks(s->npad));
  s->partial_bytes = s->splits > 1 ? up((size_t)s->splits * g->h_out * cout * 4) : 0;
  return true;
}

}  // namespace
}  // namespace ocnn

extern "C" size_t ocnn_octree_conv_f32_workspace_bytes(const ocnn_conv_geometry* g, int cin, int cout,
                                                       const int kernel_size[3]) {
  using namespace ocnn;
  if (g == nullptr || kernel_size == nullptr || cin <= 0 || cout <= 0 || g->h_out <= 0 || g->h_in <= 0) return 0;
  const TapList tl = taps_for_kernel(kernel_size);
  F32Shape s;
  if (tl.count < 0 || !f32_shape(g, cin, cout, tl, &s)) return 0;
  return s.xs_bytes + s.wp_bytes + s.partial_bytes;
}

extern "C" int ocnn_octree_conv_f32(const float* x, const float* w, float* y, const ocnn_conv_geometry* g,
                                    int cin, int cout, const int kernel_size[3], int layout,
                                    const ocnn_conv_epilogue* ep, void* workspace, size_t workspace_bytes,
                                    int32_t* status, void* stream) {
  using namespace ocnn;
  const char* who = "ocnn_octree_conv_f32";
  OCNN_REQUIRE(kernel_size != nullptr && g != nullptr, "%s: null argument", who);
  const TapList tl = taps_for_kernel(kernel_size);
  if (tl.count < 0)
    return fail(OCNN_ERR_UNSUPPORTED, "%s: unsupported kernel size %dx%dx%d", who, kernel_size[0], kernel_size[1],
                kernel_size[2]);
  OCNN_REQUIRE(cin > 0 && cout > 0, "%s: channel counts must be positive", who);
  OCNN_REQUIRE(layout == OCNN_CHANNEL_MAJOR || layout == OCNN_NODE_MAJOR, "%s: unknown layout %d", who, layout);
  if (int rc = check_conv_geometry(g, tl, who)) return rc;
  if (g->h_out == 0) return OCNN_OK;
  OCNN_REQUIRE(x && w && y && workspace && status, "%s: null pointer", who);
  OCNN_REQUIRE((uintptr_t)workspace % 256 == 0, "%s: the workspace must be 256-byte aligned", who);
  F32Shape s;
  if (g->h_in <= 0 || !f32_shape(g, cin, cout, tl, &s))
    return fail(OCNN_ERR_UNSUPPORTED, "%s: layer not served", who);
  if (workspace_bytes < s.xs_bytes + s.wp_bytes + s.partial_bytes)
    return fail(OCNN_ERR_CAPACITY, "%s: workspace of %zu bytes, need %zu", who, workspace_bytes,
                s.xs_bytes + s.wp_bytes + s.partial_bytes);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  const bool transposed = g->transposed != 0, identity = tl.count == 1 && g->stride == 1;

  PrepareArgs p;
  p.x = x; p.xs = ws; p.w = w; p.wp = ws + s.xs_bytes;
  p.h_in = g->h_in; p.cin = cin; p.cp = s.cp; p.node_major = layout == OCNN_NODE_MAJOR;
  p.cout = cout; p.npad = s.npad; p.T = s.T; p.nkb = s.nkb; p.transposed = transposed;
  p.x_items = (long long)g->h_in * (s.cp / 8);
  p.w_items = (long long)s.slices * s.nkb * s.npad * 4;
  p.x_blocks = ceil_div(p.x_items, 256);
  OCNN_CUDA_OK(launch_chained(conv_f32_prepare_kernel, dim3(p.x_blocks + ceil_div(p.w_items, 256)), dim3(256), 0,
                              st, p));
  OCNN_LAUNCH_OK("conv_f32_prepare_kernel");

  F32Args a;
  a.xs = ws; a.wp = ws + s.xs_bytes; a.y = y;
  a.partial = s.splits > 1 ? reinterpret_cast<float*>(ws + s.xs_bytes + s.wp_bytes) : nullptr;
  a.neigh = identity ? nullptr : g->neigh_dev;
  a.child = (g->nempty && !identity && !(transposed && g->stride == 2)) ? g->child_dev : nullptr;
  a.ichild = (g->nempty && !identity && !(g->stride == 2 && !transposed)) ? g->ichild_dev : nullptr;
  a.h_in = g->h_in; a.h_out = g->h_out; a.cp = s.cp; a.cout = cout; a.npad = s.npad; a.T = s.T;
  a.stride = g->stride; a.identity = identity; a.up = transposed && g->stride == 2;
  a.tiles = s.tiles; a.slices = s.slices; a.splits = s.splits;
  a.nkb = s.nkb; a.kb_per_split = s.kb_per_split; a.stages = s.stages;
  a.tmem_cols = s.tmem_cols; a.node_major = layout == OCNN_NODE_MAJOR;
  a.vec4 = a.node_major && cout % 4 == 0 && (uintptr_t)y % 16 == 0;
  a.y_elems = (long long)g->h_out * cout;
  a.aff = channel_affine_of(ep);
  a.residual = ep ? static_cast<const float*>(ep->residual_dev) : nullptr;
  a.relu = epilogue_relu(ep);
  a.status = status;
  for (int i = 0; i < 27; ++i) {
    int tap = i < tl.count ? tl.tap[i] : 0;
    if (transposed && g->stride == 1) tap = 26 - tap;    // gathers from the mirrored offsets
    a.tap[i] = (signed char)(((tap / 9) << 4) | (((tap / 3) % 3) << 2) | (tap % 3));
  }
  typedef void (*KernelFn)(const F32Args);
  static const KernelFn table[8] = {conv_f32_kernel<1>, conv_f32_kernel<2>, conv_f32_kernel<3>, conv_f32_kernel<4>,
                                    conv_f32_kernel<5>, conv_f32_kernel<6>, conv_f32_kernel<7>, conv_f32_kernel<8>};
  static PerDeviceOnce attr_once;
  const int limits = attr_once.run([&]() -> int {
    for (int k = 0; k < 8; ++k)
      OCNN_CUDA_OK(cudaFuncSetAttribute(table[k], cudaFuncAttributeMaxDynamicSharedMemorySize, 222 * 1024));
    return OCNN_OK;
  });
  if (limits != OCNN_OK) return limits;
  OCNN_CUDA_OK(launch_chained(table[s.npad / 16 - 1], dim3(s.ctas), dim3(kF32Threads), s.smem, st, a));
  OCNN_LAUNCH_OK("conv_f32_kernel");
  if (s.splits > 1) {
    OCNN_CUDA_OK(launch_chained(conv_f32_reduce_kernel, dim3(grid_for(a.y_elems, 256)), dim3(256), 0, st,
                                (const float*)a.partial, y, a.y_elems, s.splits, cout, g->h_out, a.node_major, a.aff,
                                a.residual, a.relu));
    OCNN_LAUNCH_OK("conv_f32_reduce_kernel");
  }
  return OCNN_OK;
}
