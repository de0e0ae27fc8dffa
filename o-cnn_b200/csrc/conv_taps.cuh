// The 3x3x3 convolution of conv_tc.cu on a tap plan (taps.cu): a tile is 128 nodes that share few of the 27
// taps, and only K-blocks (64 channels) that hold a present tap are gathered, fetched and multiplied.
//
// What bounds it: latency.  With 5 to 16 taps a tile's loop is 8 to 50 K-blocks, and setting a tile up is a chain of
// its mask, its table of rows and its first copies, a microsecond each, with the epilogue behind it; two or three
// CTAs with a short ring share an SM to cover one another.  The gathered rows' indices come from the plan's table
// in one bulk copy instead of 27 look-ups through neighbour and child arrays.  96 -> 96 at 192 k nodes of depth 9
// (7 of 27 taps a tile): 146 us over all taps, 52 us so.  Slower, when this form took 58: indices read from the plan
// by the gathering threads (they queue behind their copies, 80 us), one persistent CTA per SM with a ring of six
// stages, tables a tile ahead and its own epilogue warps (91 us at best: a K-block is a chain of barriers, and one
// such chain per SM is too few), and a warp that waits as a whole for the issuing lane (73 us).  With K split over
// CTAs as an option the same layers took 58 us in place of 52.
//
// K-blocks keep the packed weights' layout, in which a tap need not start on a block: of a block that is
// shared by taps only the 16-channel steps of present ones are multiplied, and only their chunks gathered.
// Results are those of the walk over all taps bit for bit, where that walk does not split K: what is left out are
// additions of zero.  Weights
// that are not finite are the exception (zero times infinity); the packed image says so, and then every tap
// is walked.
#pragma once

#include "taps.cuh"
#include "tc.cuh"

namespace ocnn {
namespace {

constexpr int kTapThreads = 192;
constexpr int kTapMaxBlocks = 256;       // K-blocks a layer may have

struct TapConvArgs {
  const uint8_t* x;
  const uint8_t* wpacked;
  const int* nonfinite;
  uint8_t* y;
  TapPlanView plan;
  int cin, npad, nkb, stages, tmem_cols;
  int row_elems;                         // output columns of a slice
  int y_stride;                          // elements between output rows
  int wide;                              // output and residual rows lie on 32-byte boundaries
  int relu;
  ChannelAffine aff;
  const uint8_t* residual;
  int* status;
  uint32_t tap_magic;                    // ceil(2^32 / (cin / 8)): a chunk's tap without a division
  __device__ __forceinline__ uint32_t tap_of(uint32_t chunk) const { return __umulhi(chunk, tap_magic); }
};

// grid: x = tiles, y = 256-column slices
template <bool HALF>
__global__ void __launch_bounds__(kTapThreads, 3) conv_taps_kernel(const TapConvArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  constexpr int kA = kTapTile * 128;     // bytes of an A stage
  const int stage_b = a.npad * 128;
  uint8_t* sA = smem;
  uint8_t* sB = sA + a.stages * kA;
  int* s_table = reinterpret_cast<int*>(sB + a.stages * stage_b);      // [present taps][128]
  float* s_scale = reinterpret_cast<float*>(s_table + 27 * kTapTile);
  float* s_bias = s_scale + a.npad;
  uint64_t* full = reinterpret_cast<uint64_t*>(s_bias + a.npad);
  uint64_t* empty = full + a.stages;
  uint64_t* accum = empty + a.stages;
  uint64_t* table_in = accum + 1;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(table_in + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);
  int* s_blocks = reinterpret_cast<int*>(tmem_holder + 2);           // number of K-blocks to walk
  // and which: the block in the low byte (kTapMaxBlocks = 256), a bit per walked 16-channel step above it
  uint16_t* s_list = reinterpret_cast<uint16_t*>(s_blocks + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // (tiles of many taps come last in the plan's order: they start first)
  const int tile = a.plan.tiles - 1 - (int)blockIdx.x;
  const int co_base = blockIdx.y * a.row_elems;
  const uint8_t* wpacked = a.wpacked + (size_t)blockIdx.y * a.nkb * stage_b;
  if (tid == 0) {
    for (int s = 0; s < a.stages; ++s) {
      mbar_init(smem_u32(&full[s]), kTapTile + 1);
      mbar_init(smem_u32(&empty[s]), 1);
    }
    mbar_init(smem_u32(accum), 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // (by the thread that uses it first, ahead of the CTA's first barrier)
  if (tid == 160) {
    mbar_init(smem_u32(table_in), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 4) tmem_alloc(tmem_holder, a.tmem_cols);
  grid_dependency_wait();
  const uint32_t present = a.plan.mask[tile];
  if (warp == 5) {
    const uint32_t walked = *a.nonfinite != 0 ? 0x7ffffffu : present;
    if (lane == 0) {
      const uint32_t bytes = (uint32_t)__popc(present) * (kTapTile * 4u);
      mbar_arrive_expect_tx(smem_u32(table_in), bytes);
      bulk_copy(smem_u32(s_table), a.plan.table + (long long)tile * (27 * kTapTile), bytes, smem_u32(table_in));
    }
    int count = 0;
    for (int k0 = 0; k0 < a.nkb; k0 += 32) {
      const int kb = k0 + lane;
      uint32_t steps = 0;
#pragma unroll
      for (int k4 = 0; k4 < 4; ++k4) {               // (cin % 16 == 0: a step lies inside one tap)
        const uint32_t t = a.tap_of(kb * 8 + 2 * k4);
        if (t < 27 && ((walked >> t) & 1u)) steps |= 1u << k4;
      }
      if (kb >= a.nkb) steps = 0;
      const uint32_t which = __ballot_sync(0xffffffffu, steps != 0);
      if (steps != 0) s_list[count + __popc(which & ((1u << lane) - 1u))] = (uint16_t)(kb | (steps << 8));
      count += __popc(which);
    }
    if (lane == 0) *s_blocks = count;
  } else {
    for (int n = tid; n < a.npad; n += kTapThreads - 32) {
      const float2 sb = n < a.row_elems ? channel_affine(a.aff, co_base + n) : make_float2(1.f, 0.f);
      s_scale[n] = sb.x;
      s_bias[n] = sb.y;
    }
  }
  const int row = tid < kTapTile ? a.plan.order[tile * kTapTile + tid] : -1;
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_holder;
  const int blocks = *s_blocks;
  bool alive = true;

  if (warp < 4) {
    // ---------------- A gather ----------------
    const int sub = lane >> 3, chunk = lane & 7;
    const int rbase = warp * 32 + sub;             // rows rbase + 4i
    const uint32_t row_bytes = (uint32_t)a.cin * 2u, cpt = (uint32_t)a.cin >> 3;     // cpt: 16-byte chunks per tap
    const int* my_idx = s_table + warp * 32 + sub * 8;
    int s = 0;
    uint32_t pe = 1;
    ZeroRows<8> zeros;
    alive = mbar_wait(smem_u32(table_in), 0, abort_flag, a.status, kErrFullWait);
    for (int b = 0; b < blocks; ++b) {
      const uint32_t entry = s_list[b];
      // (a chunk whose tap is not walked stays as it is: nobody multiplies it)
      const bool has = (entry >> (8 + (chunk >> 1))) & 1u;
      const uint32_t g = (entry & 255u) * 8u + (uint32_t)chunk, t = a.tap_of(g), off = (g - t * cpt) * 16u;
      int p[8] = {-1, -1, -1, -1, -1, -1, -1, -1};
      if (has && ((present >> t) & 1u)) {
        const int* at = my_idx + __popc(present & ((1u << t) - 1u)) * kTapTile;
        const int4 lo = reinterpret_cast<const int4*>(at)[0], hi = reinterpret_cast<const int4*>(at)[1];
        p[0] = lo.x; p[1] = lo.y; p[2] = lo.z; p[3] = lo.w;
        p[4] = hi.x; p[5] = hi.y; p[6] = hi.z; p[7] = hi.w;
      }
      if (alive && b >= a.stages)
        alive = mbar_wait(smem_u32(&empty[s]), pe, abort_flag, a.status, kErrEmptyWait);
      if (alive && has) {
        const uint32_t stage_base = smem_u32(sA + s * kA);
        const uint32_t copies = zeros.copies(s, live_rows<8>(p));
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int r = rbase + 4 * i;
          const uint32_t dst = stage_base + (uint32_t)r * 128u + (((uint32_t)chunk ^ (uint32_t)(r & 7)) << 4);
          const uint8_t* src = p[i] >= 0 ? a.x + (size_t)((uint32_t)p[i] * row_bytes) + off : a.x;
          if ((copies >> i) & 1u) cp_async16(dst, src, p[i] >= 0 ? 16u : 0u);
        }
      }
      asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&full[s])) : "memory");
      if (++s == a.stages) { s = 0; pe ^= 1u; }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");

    // ---------------- epilogue: TMEM -> registers -> global ----------------
    const bool row_ok = row >= 0;
    const uint16_t* res_row = (a.residual != nullptr && row_ok)
        ? reinterpret_cast<const uint16_t*>(a.residual) + (long long)row * a.y_stride + co_base : nullptr;
    uint16_t* y_row = reinterpret_cast<uint16_t*>(a.y) + (long long)row * a.y_stride + co_base;
    uint4 res_nxt[4];
    auto load_line = [&](int c0) {
#pragma unroll
      for (int k = 0; k < 4; ++k) res_nxt[k] = make_uint4(0, 0, 0, 0);
      if (res_row == nullptr) return;
      if (a.wide) {
#pragma unroll
        for (int k = 0; k < 4; k += 2)
          if (c0 + 8 * k < a.row_elems) ld_global_32B(res_row + c0 + 8 * k, res_nxt[k], res_nxt[k + 1]);
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (c0 + 8 * k < a.row_elems) res_nxt[k] = *reinterpret_cast<const uint4*>(res_row + c0 + 8 * k);
      }
    };
    load_line(0);
    if (alive) alive = mbar_wait(smem_u32(accum), 0, abort_flag, a.status, kErrAccumWait);
    alive = __all_sync(0xffffffffu, alive);        // tcgen05.ld is warp-collective: decide per warp
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t lane_base = tmem_base + ((uint32_t)(warp * 32) << 16);
    const bool has_sb = a.aff.any();
    for (int c0 = 0; alive && c0 < a.npad; c0 += 32) {
      uint4 res_cur[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) res_cur[k] = res_nxt[k];
      if (c0 + 32 < a.npad) load_line(c0 + 32);
      uint32_t v2[2][16];
      __syncwarp();
      tmem_ld16(lane_base + (uint32_t)c0, v2[0]);
      if (c0 + 16 < a.npad) tmem_ld16(lane_base + (uint32_t)(c0 + 16), v2[1]);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int part = 0; part < 2; ++part) {
        const int n0 = c0 + 16 * part;
        if (n0 >= a.npad || !row_ok || n0 >= a.row_elems) break;
        const uint32_t (&v)[16] = v2[part];
        uint4 ov[2];
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const int n = n0 + 8 * half;
          if (n >= a.row_elems) break;
          float f[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) f[j] = __uint_as_float(v[8 * half + j]);
          if (has_sb) {
#pragma unroll
            for (int j = 0; j < 8; j += 4) {
              const float4 sc = *reinterpret_cast<const float4*>(s_scale + n + j);
              const float4 bi = *reinterpret_cast<const float4*>(s_bias + n + j);
              f[j] = fmaf(f[j], sc.x, bi.x);
              f[j + 1] = fmaf(f[j + 1], sc.y, bi.y);
              f[j + 2] = fmaf(f[j + 2], sc.z, bi.z);
              f[j + 3] = fmaf(f[j + 3], sc.w, bi.w);
            }
          }
          if (res_row != nullptr) {
            const uint32_t* rp = reinterpret_cast<const uint32_t*>(&res_cur[2 * part + half]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float2 rf = unpack2(rp[j], HALF);
              f[2 * j] += rf.x;
              f[2 * j + 1] += rf.y;
            }
          }
          if (a.relu) {
#pragma unroll
            for (int j = 0; j < 8; ++j) f[j] = fmaxf(f[j], 0.f);
          }
          uint32_t* op = reinterpret_cast<uint32_t*>(&ov[half]);
#pragma unroll
          for (int j = 0; j < 4; ++j) op[j] = pack2(f[2 * j], f[2 * j + 1], HALF);
          if (!a.wide) *reinterpret_cast<uint4*>(y_row + n) = ov[half];
        }
        if (a.wide) st_global_32B(y_row + n0, ov[0], ov[1]);
      }
    }
  } else if (warp == 4) {
    // ---------------- MMA issue: one thread ----------------
    if (lane == 0) {
      const uint32_t ab = HALF ? 0u : 1u;
      const uint32_t idesc = (1u << 4) | (ab << 7) | (ab << 10) | ((uint32_t)(a.npad >> 3) << 17) |
                             ((uint32_t)(kTapTile >> 4) << 24);
      int s = 0;
      uint32_t pf = 0, sum = 0;
      for (int b = 0; b < blocks; ++b) {
        const uint32_t steps = (uint32_t)s_list[b] >> 8;
        alive = mbar_wait(smem_u32(&full[s]), pf, abort_flag, a.status, kErrFullWait);
        if (!alive) break;
        // the rows were written through the generic proxy (cp.async), the tensor core reads through the async one
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t a_desc = smem_desc_sw128(smem_u32(sA) + s * kA), b_desc = smem_desc_sw128(smem_u32(sB) + s * stage_b);
#pragma unroll
        for (int k4 = 0; k4 < 4; ++k4) {
          if ((steps >> k4) & 1u) {
            umma_bf16(tmem_base, a_desc + 2 * k4, b_desc + 2 * k4, idesc, sum);      // (16 channels on: 32 bytes)
            sum = 1;
          }
        }
        umma_commit(smem_u32(&empty[s]));
        if (++s == a.stages) { s = 0; pf ^= 1u; }
      }
      umma_commit(smem_u32(accum));
      if (!alive) {
        // gave up: the MMAs already issued retire (bounded) before TMEM is freed
        for (unsigned it = 0; it < kSpinLimit; ++it)
          if (mbar_try_wait(smem_u32(accum), 0)) break;
      }
    }
  } else if (lane == 0) {
    // ---------------- weight tiles: one bulk copy per K-block ----------------
    int s = 0;
    uint32_t pe = 1;
    for (int b = 0; b < blocks; ++b) {
      if (b >= a.stages) alive = mbar_wait(smem_u32(&empty[s]), pe, abort_flag, a.status, kErrWeightWait);
      if (!alive) break;
      const uint32_t bar = smem_u32(&full[s]);
      mbar_arrive_expect_tx(bar, (uint32_t)stage_b);
      bulk_copy(smem_u32(sB + s * stage_b), wpacked + (size_t)(s_list[b] & 255u) * stage_b, (uint32_t)stage_b, bar);
      if (++s == a.stages) { s = 0; pe ^= 1u; }
    }
    if (!alive) {
      // gave up with copies in flight into this CTA's shared memory: leave them time (bounded) to land
      for (int it = 0; it < 64; ++it) __nanosleep(1000);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 4)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)a.tmem_cols)
                 : "memory");
}

}  // namespace
}  // namespace ocnn
