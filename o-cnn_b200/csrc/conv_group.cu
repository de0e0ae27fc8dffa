// fp32 3x3x3 stride-1 octree convolution (and its data gradient) of whole sibling groups on the CUDA
// cores.
//
// The eight nodes of a sibling group share one 4x4x4 block of neighbours, so per input channel the
// group needs 64 values for its 8 x 27 products per output channel.  A warp takes GPW groups and a lane
// holds J output channels: per input channel the 64 values pass through shared memory once (two
// gathered reads per lane and group), are read back as sixteen 16-byte broadcasts into registers, and
// feed 216 J multiply-adds per group; the 27 J weights of a lane come from shared memory, shared by the
// CTA's warps and used for all of the warp's groups.  Nothing is gathered twice and there is no index
// arithmetic in the loop: per 864 multiply-adds (J = GPW = 2) a lane issues about 100 other
// instructions, where the general kernel (conv_simt.cu) spent one on every second.
//
// Every output is one chain of rounded multiply-adds over (channel, tap) in the weights' own order,
// the same as in conv_simt.cu: results are bit-identical to that kernel's.  Bound: the FMA pipes.
#include "common.cuh"

namespace ocnn {
namespace {

struct GroupArgs {
  const float* x;         // [cin, h]
  const float* w;         // [cout, cin * 27]
  float* y;               // [cout, h]
  const int* neigh;
  int h, cin, cout;
  ChannelAffine aff;
  const float* residual;
  int relu;
};

constexpr int kGroupCi = 2;              // input channels per weight stage

// Four bytes global -> shared (zeros unless `live`), asynchronously.
__device__ __forceinline__ void copy4(float* dst, const float* src, bool live) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(live ? 4u : 0u)
               : "memory");
}

// CO output channels per CTA slice: 64 (two per lane), 32, or 16 (half a warp per group).
// TRANS: the data gradient (stride-1 deconvolution): weights [cin, cout * 27], tap t read from the
// mirrored position.
template <int CO, int WARPS, int GPW, bool TRANS>
__global__ void __launch_bounds__(32 * WARPS) conv_group_kernel(const GroupArgs a) {
  constexpr int J = CO == 64 ? 2 : 1;
  constexpr int kHalves = CO == 16 ? 2 : 1;              // lane sets that work on groups of their own
  constexpr int kWarpGroups = GPW * kHalves;
  constexpr int kStride = CO + 2;                        // words between taps: spreads the transposing stores
                                                         // (channel c's tap t is row 27 c + t)
  __shared__ __align__(16) float sw[2][kGroupCi][27 * kStride];
  __shared__ __align__(16) float sx[WARPS][kWarpGroups][64];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int co0 = blockIdx.y * CO;
  const int groups = a.h >> 3;
  const int g0 = (blockIdx.x * WARPS + warp) * kWarpGroups;
  const int half = kHalves == 2 ? lane >> 4 : 0, cl = kHalves == 2 ? lane & 15 : lane;
  grid_dependency_trigger();
  grid_dependency_wait();

  // the groups' neighbour blocks: two positions per lane and group
  int p[kWarpGroups][2];
#pragma unroll
  for (int g = 0; g < kWarpGroups; ++g)
#pragma unroll
    for (int u = 0; u < 2; ++u)
      p[g][u] = g0 + g < groups ? a.neigh[((long long)(g0 + g) << 6) + 32 * u + lane] : -1;
  float v[kWarpGroups][2];
  auto fetch = [&](int ci) {
#pragma unroll
    for (int g = 0; g < kWarpGroups; ++g)
#pragma unroll
      for (int u = 0; u < 2; ++u) v[g][u] = p[g][u] >= 0 ? a.x[(long long)ci * a.h + p[g][u]] : 0.f;
  };

  // weights of channels [ci0, ci0 + kGroupCi) into buffer `buf`, tap-major
  const int KD = a.cin * 27;
  auto stage_weights = [&](int buf, int ci0) {
    // (a channel's weights are contiguous, two channels' only without TRANS; a warp copies whole rows)
    const int n = min(kGroupCi, a.cin - ci0) * 27;
    static_assert(kGroupCi == 2, "54 weights are two reads per lane");
    float* to = &sw[buf][0][0];
#pragma unroll
    for (int i = 0; i < CO / WARPS; ++i) {
      const int co = warp + WARPS * i;
      const bool live = co0 + co < a.cout;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int k = lane + 32 * u;
        const float* from = TRANS ? a.w + ((long long)(ci0 + k / 27) * a.cout + co0 + co) * 27 + k % 27
                                  : a.w + (long long)(co0 + co) * KD + ci0 * 27 + k;
        if (k < n) copy4(to + k * kStride + co, live ? from : a.w, live);
      }
    }
  };

  float acc[GPW][8][J];
#pragma unroll
  for (int g = 0; g < GPW; ++g)
#pragma unroll
    for (int o = 0; o < 8; ++o)
#pragma unroll
      for (int j = 0; j < J; ++j) acc[g][o][j] = 0.f;

  stage_weights(0, 0);
  fetch(0);
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  int buf = 0;
#pragma unroll 1
  for (int ci0 = 0; ci0 < a.cin; ci0 += kGroupCi) {
    if (ci0 + kGroupCi < a.cin) stage_weights(buf ^ 1, ci0 + kGroupCi);
#pragma unroll 1
    for (int c = 0; c < kGroupCi && ci0 + c < a.cin; ++c) {
      __syncwarp();                                      // everyone has read the previous channel
#pragma unroll
      for (int g = 0; g < kWarpGroups; ++g) {
        sx[warp][g][lane] = v[g][0];
        sx[warp][g][32 + lane] = v[g][1];
      }
      __syncwarp();
      if (ci0 + c + 1 < a.cin) fetch(ci0 + c + 1);       // in flight during the products
      float wv[27][J];
#pragma unroll
      for (int t = 0; t < 27; ++t) {
        if constexpr (J == 2) {
          const float2 w2 = *reinterpret_cast<const float2*>(&sw[buf][c][t * kStride + 2 * cl]);
          wv[t][0] = w2.x;
          wv[t][1] = w2.y;
        } else {
          wv[t][0] = sw[buf][c][t * kStride + cl];
        }
      }
#pragma unroll
      for (int g = 0; g < GPW; ++g) {
        const float4* in = reinterpret_cast<const float4*>(sx[warp][g * kHalves + half]);
        // x planes of the block two at a time would not help: an octant needs three of the four
        float b[4][4][4];
#pragma unroll
        for (int r = 0; r < 16; ++r) {
          const float4 q = in[r];
          b[r >> 2][r & 3][0] = q.x; b[r >> 2][r & 3][1] = q.y;
          b[r >> 2][r & 3][2] = q.z; b[r >> 2][r & 3][3] = q.w;
        }
#pragma unroll
        for (int t = 0; t < 27; ++t) {
          const int at = TRANS ? 26 - t : t;
          const int tx = at / 9, ty = at / 3 % 3, tz = at % 3;
#pragma unroll
          for (int o = 0; o < 8; ++o) {
            const float in_v = b[tx + (o >> 2)][ty + ((o >> 1) & 1)][tz + (o & 1)];
#pragma unroll
            for (int j = 0; j < J; ++j) acc[g][o][j] = fmaf(in_v, wv[t][j], acc[g][o][j]);
          }
        }
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    buf ^= 1;
  }

  // a lane's eight nodes are one 32-byte sector of its channel's row
#pragma unroll
  for (int j = 0; j < J; ++j) {
    const int co = co0 + (J == 2 ? 2 * cl + j : cl);
    if (co >= a.cout) continue;
    const float2 sb = channel_affine(a.aff, co);
#pragma unroll
    for (int g = 0; g < GPW; ++g) {
      const int group = g0 + g * kHalves + half;
      if (group >= groups) continue;
      const long long at = (long long)co * a.h + 8LL * group;
      float f[8];
#pragma unroll
      for (int o = 0; o < 8; ++o) f[o] = fmaf(acc[g][o][j], sb.x, sb.y);
      if (a.residual) {
#pragma unroll
        for (int o = 0; o < 8; ++o) f[o] += a.residual[at + o];
      }
      if (a.relu) {
#pragma unroll
        for (int o = 0; o < 8; ++o) f[o] = fmaxf(f[o], 0.f);
      }
      float4* out = reinterpret_cast<float4*>(a.y + at);
      out[0] = make_float4(f[0], f[1], f[2], f[3]);
      out[1] = make_float4(f[4], f[5], f[6], f[7]);
    }
  }
}

template <int CO, bool TRANS>
cudaError_t launch_group(const GroupArgs& a, cudaStream_t st) {
  const int groups = a.h >> 3, slices = ceil_div(a.cout, CO), halves = CO == 16 ? 2 : 1;
  // two groups per warp and eight warps per CTA share the weights best; a level too small to give
  // every SM a few warps that way is cut finer
  if ((long long)ceil_div(groups, 16 * halves) * slices >= 2LL * sm_count())
    return launch_chained(conv_group_kernel<CO, 8, 2, TRANS>, dim3(ceil_div(groups, 16 * halves), slices), dim3(256), 0, st, a);
  return launch_chained(conv_group_kernel<CO, 4, 1, TRANS>, dim3(ceil_div(groups, 4 * halves), slices), dim3(128), 0, st, a);
}

template <bool TRANS>
cudaError_t launch_for(const GroupArgs& a, cudaStream_t st) {
  if (a.cout > 32) return launch_group<64, TRANS>(a, st);
  return a.cout > 16 ? launch_group<32, TRANS>(a, st) : launch_group<16, TRANS>(a, st);
}

}  // namespace

// Serves fp32 channel-major data on all nodes, kernel 3, stride 1; -1 otherwise.
int conv_group_f32(const float* x, const float* w, float* y, const ocnn_conv_geometry* g, int cin, int cout,
                   const TapList& tl, int layout, const ocnn_conv_epilogue* ep, cudaStream_t st) {
  if (layout != OCNN_CHANNEL_MAJOR || tl.count != 27 || g->stride != 1 || g->nempty ||
      g->h_out % 8 != 0 || g->h_out != g->h_in || (uintptr_t)y % 16 != 0)
    return -1;
  GroupArgs a;
  a.x = x; a.w = w; a.y = y; a.neigh = g->neigh_dev;
  a.h = g->h_out; a.cin = cin; a.cout = cout;
  a.aff = channel_affine_of(ep);
  a.residual = ep ? static_cast<const float*>(ep->residual_dev) : nullptr;
  a.relu = epilogue_relu(ep);
  OCNN_CUDA_OK((g->transposed ? launch_for<true>(a, st) : launch_for<false>(a, st)));
  OCNN_LAUNCH_OK("conv_group_kernel");
  return OCNN_OK;
}

}  // namespace ocnn
