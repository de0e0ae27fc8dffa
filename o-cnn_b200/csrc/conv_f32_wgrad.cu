// Weight gradient of the octree (de)convolution in fp32 on the tensor cores:
//     dW[m, c*K + t] = sum_h A[m, h] * X[c, nbr(h, t)]
// (A: the output gradient and X the layer's input for a convolution, the other way round for a
// deconvolution; nbr: the convolution's gather.)  The reduction runs over the nodes, so this is a
// matrix product whose K dimension is h:
//     D[(t, c), m] = G^T S,   G[h, (t, c)] = X[c, nbr(h, t)] gathered,   S[h, m] = A[m, h]
// with every fp32 value as three bf16 parts and six products, as in conv_f32.cu (same rows, same
// order of the (t, c) pairs in chunks of eight channels, same accumulators and drains).  Both operands
// arrive with the non-reduced index contiguous (a neighbour's channels; a node's gradients), which
// is the MN-major operand layout of the tensor core: a 64-byte piece of a gathered row is one K row
// of a 32-wide block.
//
// An item is (128 (t, c) pairs, up to 128 columns m, a range of nodes); the ranges are chosen so that
// the items fill the SMs, and a reduction adds their partial results in a fixed order (the CUDA-core
// kernel added partial tiles with atomics: 2.41 ms for 32 -> 64 channels at 217 k nodes).
// Bound: as conv_f32.cu, the gather (each node's row once per tap) and the MMAs' operand reads.
#include "f32.cuh"

namespace ocnn {
namespace {

constexpr int kWgStep = 32;                      // nodes per stage: two K = 16 steps
constexpr int kWgChunk = 2;                      // stages per drained chunk: 4 accumulations
constexpr int kWgBlock = kWgStep * 64;           // bytes of one 32-wide block of a part (LBO)

struct WgF32Args {
  const uint8_t* xs;        // split rows of X
  const uint8_t* as;        // A as operand images: per slice and 32 nodes [stacks][N / 32][32 rows x 64 bytes]
  float* partial;           // [split][group][slice][N][128]
  const int* neigh;
  const int* child;
  const int* ichild;
  int h_a, cp, T, stride, identity;
  int groups, slices, splits, steps, steps_per_split, stages, tmem_cols;
  int* status;
  signed char tap[27];
};

// MN-major, 64-byte swizzle: 32 contiguous values per K row, eight K rows per 512-byte atom (the
// stride between atoms along K), blocks of 32 values kWgBlock apart (the leading stride).
__device__ __forceinline__ uint64_t smem_desc_mn64(uint32_t addr) {
  return (uint64_t)((addr & 0x3ffffu) >> 4) | ((uint64_t)(kWgBlock >> 4) << 16) | ((uint64_t)(512 >> 4) << 32) |
         (1ull << 46) | (4ull << 61);
}

struct WgPrepareArgs {
  const float* x;
  uint8_t* xs;
  const float* a;
  uint8_t* as;
  int h_x, channels, cp, node_major;
  int h_a, m, npad, slices, steps;
  long long x_items, a_items;
  int x_blocks;
};

// X as split rows, A as operand images (rows past the last node and columns past M are zero).
__global__ void __launch_bounds__(256) conv_f32_wgrad_prepare_kernel(const WgPrepareArgs a) {
  grid_dependency_trigger();
  grid_dependency_wait();
  if ((int)blockIdx.x < a.x_blocks) {
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i < a.x_items) split_rows(a.x, a.xs, i, a.h_x, a.channels, a.cp, a.node_major);
    return;
  }
  const long long i = (long long)(blockIdx.x - a.x_blocks) * 256 + threadIdx.x;
  if (i >= a.a_items) return;
  const long long rows = (long long)a.steps * kWgStep;
  int c8;
  long long h;
  chunk_of_block(i, rows, a.slices * a.npad / 8, c8, h);     // (a row of an image is four chunks)
  uint4 part[3];
  split_chunk(a.a, h, c8, a.h_a, a.m, a.node_major, part);
  const int slice = c8 / (a.npad / 8), n8 = c8 - slice * (a.npad / 8);
  const int stacks = f32_stacks(a.npad), row = (int)(h % kWgStep);
  uint8_t* dst = a.as + ((long long)slice * a.steps + h / kWgStep) * (stacks * a.npad * 64) +
                 (n8 >> 2) * kWgBlock + row * 64 + (((n8 & 3) ^ ((row >> 1) & 3)) << 4);
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    if (b >= stacks) break;
    *reinterpret_cast<uint4*>(dst + b * a.npad * 64) = part[b == 3 ? 0 : b];
  }
}

// Warps 0-3 gather (warp j: 32-wide block j of the item's 128 (t, c) pairs), 4-7 drain and store, 8
// issues the MMAs, 9 streams A's images; persistent over the items, two CTAs per SM up to 64 columns.
template <int NB>                          // N / 32
__global__ void __launch_bounds__(kF32Threads, NB <= 2 ? 2 : 1) conv_f32_wgrad_kernel(const WgF32Args a) {
  constexpr int N = 32 * NB;
  constexpr bool kOne = f32_stacks(N) == 4;
  constexpr int kBytesB = N * 64 * f32_stacks(N);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* sA = smem;
  uint8_t* sB = sA + a.stages * (3 * kF32PartA);
  uint64_t* full = reinterpret_cast<uint64_t*>(sB + a.stages * kBytesB);
  uint64_t* empty = full + a.stages;
  uint64_t* cfull = empty + a.stages;
  uint64_t* cempty = cfull + 2;
  uint64_t* dempty = cempty + 2;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(dempty + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int s = 0; s < a.stages; ++s) {
      mbar_init(smem_u32(&full[s]), 128 + 1);
      mbar_init(smem_u32(&empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&cfull[b]), 1);
      mbar_init(smem_u32(&cempty[b]), 128);
    }
    mbar_init(smem_u32(dempty), 128);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 8) tmem_alloc(tmem_holder, a.tmem_cols);
  grid_dependency_wait();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_holder;

  // item -> (split, group, slice), the groups of a node range side by side in time
  const int per_split = a.groups * a.slices;
  const int items = per_split * a.splits;
  auto first_step = [&](int item) { return item / per_split * a.steps_per_split; };
  auto item_steps = [&](int item) { return min(a.steps_per_split, a.steps - first_step(item)); };

  if (warp < 4) {
    // ---------------- gather: lane = (node of eight, 16-byte chunk of the block's 64 bytes) ----------------
    const int c = lane & 3, rr = lane >> 2;
    const int cpt = a.cp >> 3;
    const uint32_t row_bytes = (uint32_t)a.cp * 6u;
    bool alive = true;
    int s = 0;
    uint32_t pe = 1;
    long long gk = 0;
    ZeroRows<4> zeros;
    for (int item = blockIdx.x; item < items; item += gridDim.x) {
      const int group = item % per_split / a.slices;
      const int g = (group * 4 + warp) * 4 + c;              // chunk of eight (t, c) pairs
      const int t = g / cpt, cc = g - t * cpt;
      uint32_t off, width;
      chunk_place(cc, cpt, off, width);
      const bool have_tap = t < a.T;
      const int code = have_tap ? a.tap[t] : 0;
      auto look = [&](int step, int (&p)[4]) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int h = step * kWgStep + 8 * i + rr;
          p[i] = -1;
          if (!have_tap || h >= a.h_a) continue;
          if (a.identity) { p[i] = h; continue; }
          const int hn = a.ichild != nullptr ? a.ichild[h] : h;
          p[i] = a.neigh[a.stride == 2 ? ((long long)hn << 6) + code
                                       : ((long long)(hn >> 3) << 6) + code +
                                             (((hn & 4) << 2) | ((hn & 2) << 1) | (hn & 1))];
        }
        if (a.child != nullptr) {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (p[i] >= 0) p[i] = a.child[p[i]];
        }
      };
      const int step0 = first_step(item), steps = item_steps(item);
      int p[4];
      look(step0, p);
      for (int k = 0; k < steps; ++k, ++gk) {
        int nxt[4] = {-1, -1, -1, -1};                       // the next step's neighbours, ahead of the copies
        if (k + 1 < steps) look(step0 + k + 1, nxt);
        if (alive && gk >= a.stages)
          alive = mbar_wait(smem_u32(&empty[s]), pe, abort_flag, a.status, kErrEmptyWait);
        if (alive) {
          const uint32_t block = smem_u32(sA + s * (3 * kF32PartA)) + (uint32_t)warp * kWgBlock;
          const uint32_t copies = zeros.copies(s, live_rows<4>(p));
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int row = 8 * i + rr;
            const uint32_t dst = block + (uint32_t)row * 64u + (((uint32_t)c ^ (uint32_t)((row >> 1) & 3)) << 4);
            const bool have = p[i] >= 0;
            const uint8_t* src = have ? a.xs + (size_t)p[i] * row_bytes + off : a.xs;
            const uint32_t stride = have ? width : 0u, n = have ? 16u : 0u;
            if ((copies >> i) & 1u) {
#pragma unroll
              for (int q = 0; q < 3; ++q) cp_async16(dst + q * kF32PartA, src + q * stride, n);
            }
          }
        }
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&full[s]))
                     : "memory");
        if (++s == a.stages) { s = 0; pe ^= 1u; }
#pragma unroll
        for (int i = 0; i < 4; ++i) p[i] = nxt[i];
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (warp < 8) {
    // ---------------- drain, store the partial result ----------------
    const int q4 = warp & 3;
    const uint32_t lane_base = tmem_base + ((uint32_t)(q4 * 32) << 16);
    bool alive = true;
    int buf = 0;
    uint32_t ph = 0;
    for (int item = blockIdx.x; item < items && alive; item += gridDim.x) {
      const int steps = item_steps(item);
      float acc[N];
#pragma unroll
      for (int j = 0; j < N; ++j) acc[j] = 0.f;
      for (int k = 0; k < steps; k += kWgChunk) {
        alive = mbar_wait(smem_u32(&cfull[buf]), ph, abort_flag, a.status, kErrAccumWait);
        alive = __all_sync(0xffffffffu, alive);
        if (!alive) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int g = 0; g < N / 8; ++g) {
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
      for (int g = 0; g < N / 8; ++g) {
        uint32_t v1[8], v2[8];
        tmem_ld8(lane_base + (uint32_t)(N + 8 * g), v1);
        tmem_ld8(lane_base + (uint32_t)(2 * N + 8 * g), v2);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[8 * g + j] = join_products(acc[8 * g + j], __uint_as_float(v1[j]), __uint_as_float(v2[j]));
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      mbar_arrive(smem_u32(dempty));
      // item order is the partial array's order
      float* out = a.partial + (long long)item * (N * 128) + q4 * 32 + lane;
#pragma unroll
      for (int j = 0; j < N; ++j) out[j * 128] = acc[j];
    }
  } else if (warp == 8) {
    // ---------------- MMA issue: one thread ----------------
    if (lane == 0) {
      // both operands MN-major (bits 15, 16)
      const uint32_t idesc0 = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((uint32_t)(128 >> 4) << 24);
      constexpr uint32_t n1 = (uint32_t)(N >> 3) << 17, n2 = (uint32_t)(2 * N >> 3) << 17,
                         n3 = (uint32_t)(3 * N >> 3) << 17;
      bool alive = true;
      int s = 0, buf = 0, it = 0;
      uint32_t pf = 0, pc = 1;
      for (int item = blockIdx.x; item < items && alive; item += gridDim.x, ++it) {
        const int steps = item_steps(item);
        if (it > 0) alive = mbar_wait(smem_u32(dempty), (uint32_t)(it - 1) & 1u, abort_flag, a.status, kErrAccumWait);
        for (int k = 0; k < steps && alive; ++k) {
          if (k % kWgChunk == 0) {
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
          for (int k2 = 0; k2 < 2; ++k2) {                    // 16 nodes: two 512-byte atoms
            const uint64_t ah = smem_desc_mn64(aa + k2 * 1024), am = smem_desc_mn64(aa + kF32PartA + k2 * 1024),
                           al = smem_desc_mn64(aa + 2 * kF32PartA + k2 * 1024);
            const uint64_t bh = smem_desc_mn64(bb + k2 * 1024), bm = smem_desc_mn64(bb + N * 64 + k2 * 1024);
            const bool first_of_chunk = k % kWgChunk == 0 && k2 == 0, first = k == 0 && k2 == 0;
            if (kOne && !(first_of_chunk && !first)) {
              umma_bf16(buf == 0 ? d0 : d1, ah, buf == 0 ? bh : bm, idesc0 | n3, first ? 0u : 1u);
            } else {
              umma_bf16(d0, ah, bh, idesc0 | n1, first_of_chunk ? 0u : 1u);
              umma_bf16(d1, ah, bm, idesc0 | n2, first ? 0u : 1u);
            }
            umma_bf16(d1, am, bh, idesc0 | n2, 1u);
            umma_bf16(d2, al, bh, idesc0 | n1, 1u);
          }
          umma_commit(smem_u32(&empty[s]));
          if (++s == a.stages) { s = 0; pf ^= 1u; }
          if (k % kWgChunk == kWgChunk - 1 || k == steps - 1) {
            umma_commit(smem_u32(&cfull[buf]));
            buf ^= 1;
            if (buf == 0) pc ^= 1u;
          }
        }
      }
      if (!alive) {
        for (int w = 0; w < 64; ++w) __nanosleep(1000);      // issued MMAs retire before TMEM is freed
      }
    }
  } else if (lane == 0) {
    // ---------------- A's operand images ----------------
    bool alive = true;
    int s = 0;
    uint32_t pe = 1;
    long long gk = 0;
    for (int item = blockIdx.x; item < items && alive; item += gridDim.x) {
      const int steps = item_steps(item), slice = item % a.slices;
      const uint8_t* src = a.as + ((long long)slice * a.steps + first_step(item)) * kBytesB;
      for (int k = 0; k < steps && alive; ++k, ++gk) {
        if (gk >= a.stages)
          alive = mbar_wait(smem_u32(&empty[s]), pe, abort_flag, a.status, kErrWeightWait);
        if (!alive) break;
        const uint32_t bar = smem_u32(&full[s]);
        mbar_arrive_expect_tx(bar, (uint32_t)kBytesB);
        bulk_copy(smem_u32(sB + s * kBytesB), src + (size_t)k * kBytesB, (uint32_t)kBytesB, bar);
        if (++s == a.stages) { s = 0; pe ^= 1u; }
      }
    }
    if (!alive) {
      for (int it = 0; it < 64; ++it) __nanosleep(1000);
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

// dW = sum of the node ranges' partial results, in their order.  Threads walk the (t, c) pairs, which
// are contiguous in the partial array.
__global__ void __launch_bounds__(256) conv_f32_wgrad_reduce_kernel(const float* __restrict__ partial,
                                                                    float* __restrict__ dw, int splits, int groups,
                                                                    int slices, int npad, int M, int channels, int cp,
                                                                    int T) {
  grid_dependency_trigger();
  grid_dependency_wait();
  // 32 outputs per block, the splits of each dealt to eight warps: with few output tiles there are up to
  // some 290 splits, and one thread adding them was a chain of that many loads
  __shared__ float part[8][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long width = (long long)groups * 128;
  const long long stride = width * slices * npad;
  for (long long base = blockIdx.x * 32LL; base < width * M; base += gridDim.x * 32LL) {
    const long long i = base + lane;                       // (width is a multiple of 128: no tail)
    const int m = (int)(i / width), lin = (int)(i - m * width);
    const int t = lin / cp, c = lin - t * cp;
    const int slice = m / npad, n = m - slice * npad, group = lin >> 7;
    const bool on = t < T && c < channels;
    float v = 0.f;
    if (on) {
      const float* p = partial + (((long long)group * slices + slice) * npad + n) * 128 + (lin & 127);
#pragma unroll 4
      for (int s = warp; s < splits; s += 8) v += p[s * stride];
    }
    part[warp][lane] = v;
    __syncthreads();
    if (warp == 0 && on) {
      for (int w = 1; w < 8; ++w) v += part[w][lane];
      dw[((long long)m * channels + c) * T + t] = v;
    }
    __syncthreads();
  }
}

struct WgF32Shape {
  int cp, npad, slices, groups, steps, splits, steps_per_split, stages, tmem_cols, ctas;
  size_t smem, xs_bytes, as_bytes, partial_bytes;
};

void wgrad_f32_shape(const ocnn_conv_geometry* g, int m, int channels, int taps, WgF32Shape* s) {
  s->cp = (channels + 7) / 8 * 8;
  s->slices = ceil_div(m, 128);
  s->npad = (ceil_div(m, s->slices) + 31) / 32 * 32;
  s->groups = ceil_div((long long)taps * s->cp, 128);
  s->steps = ceil_div(g->h_out, kWgStep);
  const int sms = sm_count();
  const bool pair = s->npad <= 64;
  // as many node ranges as fill the SMs' CTA slots once, none shorter than a drained chunk
  const long long per = (long long)s->groups * s->slices, room = (long long)sms * (pair ? 2 : 1);
  long long splits = room / per;
  const long long most = ceil_div(s->steps, kWgChunk);
  if (splits > most) splits = most;
  if (splits < 1) splits = 1;
  s->steps_per_split = (ceil_div(s->steps, splits) + kWgChunk - 1) / kWgChunk * kWgChunk;
  s->splits = ceil_div(s->steps, s->steps_per_split);
  s->tmem_cols = 4 * s->npad <= 128 ? 128 : (4 * s->npad <= 256 ? 256 : 512);
  const long long items = per * s->splits;
  const bool share = pair && items > sms;
  const size_t stage = 3 * kF32PartA + (size_t)s->npad * 64 * f32_stacks(s->npad), fixed = 1024 + 512;
  int st = (int)(((share ? 112 : 220) * 1024 - fixed) / stage);
  if (st > 6) st = 6;
  s->stages = st;
  s->smem = fixed + st * stage;
  const long long slots = share ? 2LL * sms : sms;
  s->ctas = ceil_div(items, ceil_div(items, slots));
  auto up = [](size_t v) { return (v + 255) / 256 * 256; };
  s->xs_bytes = up((size_t)g->h_in * s->cp * 6);
  s->as_bytes = up((size_t)s->slices * s->steps * s->npad * 64 * f32_stacks(s->npad));
  s->partial_bytes = (size_t)items * s->npad * 128 * 4;
}

}  // namespace
}  // namespace ocnn

extern "C" size_t ocnn_octree_conv_weight_grad_f32_workspace_bytes(const ocnn_conv_geometry* g, int m_channels,
                                                                   int x_channels, const int kernel_size[3]) {
  using namespace ocnn;
  if (g == nullptr || kernel_size == nullptr || m_channels <= 0 || x_channels <= 0 || g->h_out <= 0 || g->h_in <= 0)
    return 0;
  const TapList tl = taps_for_kernel(kernel_size);
  if (tl.count < 0 || g->transposed) return 0;
  WgF32Shape s;
  wgrad_f32_shape(g, m_channels, x_channels, tl.count, &s);
  return s.xs_bytes + s.as_bytes + s.partial_bytes;
}

extern "C" int ocnn_octree_conv_weight_grad_f32(const float* a, const float* x, float* dw,
                                                const ocnn_conv_geometry* g, int m_channels, int x_channels,
                                                const int kernel_size[3], int layout, void* workspace,
                                                size_t workspace_bytes, int32_t* status, void* stream) {
  using namespace ocnn;
  const char* who = "ocnn_octree_conv_weight_grad_f32";
  OCNN_REQUIRE(kernel_size != nullptr && g != nullptr, "%s: null argument", who);
  const TapList tl = taps_for_kernel(kernel_size);
  if (tl.count < 0)
    return fail(OCNN_ERR_UNSUPPORTED, "%s: unsupported kernel size %dx%dx%d", who, kernel_size[0], kernel_size[1],
                kernel_size[2]);
  OCNN_REQUIRE(!g->transposed, "%s: pass the convolution-type geometry of the column matrix", who);
  OCNN_REQUIRE(m_channels > 0 && x_channels > 0, "%s: channel counts must be positive", who);
  OCNN_REQUIRE(layout == OCNN_CHANNEL_MAJOR || layout == OCNN_NODE_MAJOR, "%s: unknown layout %d", who, layout);
  if (int rc = check_conv_geometry(g, tl, who)) return rc;
  OCNN_REQUIRE(g->h_out > 0 && g->h_in > 0, "%s: empty data", who);
  OCNN_REQUIRE(a && x && dw && workspace && status, "%s: null pointer", who);
  OCNN_REQUIRE((uintptr_t)workspace % 256 == 0, "%s: the workspace must be 256-byte aligned", who);
  WgF32Shape s;
  wgrad_f32_shape(g, m_channels, x_channels, tl.count, &s);
  if (workspace_bytes < s.xs_bytes + s.as_bytes + s.partial_bytes)
    return fail(OCNN_ERR_CAPACITY, "%s: workspace of %zu bytes, need %zu", who, workspace_bytes,
                s.xs_bytes + s.as_bytes + s.partial_bytes);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  const bool identity = tl.count == 1 && g->stride == 1;

  WgPrepareArgs p;
  p.x = x; p.xs = ws; p.a = a; p.as = ws + s.xs_bytes;
  p.h_x = g->h_in; p.channels = x_channels; p.cp = s.cp; p.node_major = layout == OCNN_NODE_MAJOR;
  p.h_a = g->h_out; p.m = m_channels; p.npad = s.npad; p.slices = s.slices; p.steps = s.steps;
  p.x_items = (long long)g->h_in * (s.cp / 8);
  p.a_items = (long long)s.slices * (s.npad / 8) * s.steps * kWgStep;
  p.x_blocks = ceil_div(p.x_items, 256);
  OCNN_CUDA_OK(launch_chained(conv_f32_wgrad_prepare_kernel, dim3(p.x_blocks + ceil_div(p.a_items, 256)), dim3(256),
                              0, st, p));
  OCNN_LAUNCH_OK("conv_f32_wgrad_prepare_kernel");

  WgF32Args w;
  w.xs = ws; w.as = ws + s.xs_bytes; w.partial = reinterpret_cast<float*>(ws + s.xs_bytes + s.as_bytes);
  w.neigh = identity ? nullptr : g->neigh_dev;
  w.child = (g->nempty && !identity) ? g->child_dev : nullptr;
  w.ichild = (g->nempty && !identity && g->stride == 1) ? g->ichild_dev : nullptr;
  w.h_a = g->h_out; w.cp = s.cp; w.T = tl.count; w.stride = g->stride; w.identity = identity;
  w.groups = s.groups; w.slices = s.slices; w.splits = s.splits; w.steps = s.steps;
  w.steps_per_split = s.steps_per_split; w.stages = s.stages; w.tmem_cols = s.tmem_cols;
  w.status = status;
  for (int i = 0; i < 27; ++i) {
    const int tap = i < tl.count ? tl.tap[i] : 0;
    w.tap[i] = (signed char)(((tap / 9) << 4) | (((tap / 3) % 3) << 2) | (tap % 3));
  }
  typedef void (*KernelFn)(const WgF32Args);
  static const KernelFn table[4] = {conv_f32_wgrad_kernel<1>, conv_f32_wgrad_kernel<2>, conv_f32_wgrad_kernel<3>,
                                    conv_f32_wgrad_kernel<4>};
  static PerDeviceOnce attr_once;
  const int limits = attr_once.run([&]() -> int {
    for (int k = 0; k < 4; ++k)
      OCNN_CUDA_OK(cudaFuncSetAttribute(table[k], cudaFuncAttributeMaxDynamicSharedMemorySize, 222 * 1024));
    return OCNN_OK;
  });
  if (limits != OCNN_OK) return limits;
  OCNN_CUDA_OK(launch_chained(table[s.npad / 32 - 1], dim3(s.ctas), dim3(kF32Threads), s.smem, st, w));
  OCNN_LAUNCH_OK("conv_f32_wgrad_kernel");
  OCNN_CUDA_OK(launch_chained(conv_f32_wgrad_reduce_kernel, dim3(grid_for((long long)s.groups * 4 * m_channels, 1)),
                              dim3(256), 0, st, (const float*)w.partial, dw, s.splits, s.groups, s.slices, s.npad,
                              m_channels, x_channels, s.cp, tl.count));
  OCNN_LAUNCH_OK("conv_f32_wgrad_reduce_kernel");
  return OCNN_OK;
}
