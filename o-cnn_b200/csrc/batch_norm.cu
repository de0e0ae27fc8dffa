// What surrounds torch's BatchNorm in a training block, on fp32 channel-major data [C][H]: the residual, the ReLU
// and the count of batches behind it (one launch), and its gradient with the ReLU's mask where that gradient goes no
// further than to parameters (a network's first layer).  Elsewhere statistics and gradient stay torch's: a
// network's gradient is not a smooth function of last bits (1x1 layers in TF32, maxima, ReLUs).  With this gradient
// everywhere the training step of 16 x 10k points was 300 us shorter and its gradients 5e-7 off with TF32 off,
// but 3e-4 with it on, where any other last bit moves roundings to TF32.
//
// What bounds the gradient: memory.  It reads x, gy and the output's sign and writes gx: four passes.  A channel's
// H values are split over a cluster of up to eight CTAs; each CTA keeps x and g of its slice in shared memory
// between the two sums and the result (of a slice that does not fit the rest is read again, from L2 mostly), the
// sums travel through distributed shared memory, and so one launch reads every value once.  Sums are formed in 64
// bits: their conversions and multiply-adds hide under the loads, and the result is exact to fp32's rounding of its
// last few operations.
// 64 channels on depth 5 of 16 x 10k points: cuDNN 142 us and the mask 8, 51 us so.
#include <cooperative_groups.h>

#include "common.cuh"

namespace ocnn {
namespace {
namespace cg = cooperative_groups;

constexpr int kBnThreads = 512;
constexpr int kMaxCluster = 8;               // the portable cluster size
constexpr size_t kBnSmem = 200 * 1024;

struct BnArgs {
  const float* x;
  const float* gy;
  const float* out;          // the block's output where a ReLU ended it (its sign), else NULL
  const float* weight;
  const float* mean;
  const float* invstd;
  float* gx;
  float* g_weight;
  float* g_bias;
  int channels, rows, cluster;
  int per, keep;             // rows of a CTA's slice, and how many of them shared memory holds
};

// Sum of a pair over the cluster, in every thread; the same order on every CTA.
__device__ __forceinline__ double2 cluster_sum(double a, double b, double2* warps, double2* total) {
  cg::cluster_group cluster = cg::this_cluster();
  const int tid = threadIdx.x;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
  if ((tid & 31) == 0) warps[tid >> 5] = make_double2(a, b);
  __syncthreads();
  if (tid == 0) {
    double2 s = warps[0];
    for (int w = 1; w < kBnThreads / 32; ++w) {
      s.x += warps[w].x;
      s.y += warps[w].y;
    }
    *total = s;
  }
  cluster.sync();
  double2 all = make_double2(0., 0.);
  for (unsigned r = 0; r < cluster.num_blocks(); ++r) {
    const double2 v = *cluster.map_shared_rank(total, r);
    all.x += v.x;
    all.y += v.y;
  }
  cluster.sync();            // nobody leaves while its sum is still to be read
  return all;
}

// Values come in pieces of V floats: four where rows and pointers allow 16-byte accesses.
template <int V>
struct Piece {
  float v[V];
};
template <int V>
__device__ __forceinline__ Piece<V> load_piece(const float* p) {
  Piece<V> r;
  if constexpr (V == 4) {
    const float4 f = *reinterpret_cast<const float4*>(p);
    r.v[0] = f.x; r.v[1] = f.y; r.v[2] = f.z; r.v[3] = f.w;
  } else {
    r.v[0] = *p;
  }
  return r;
}
template <int V>
__device__ __forceinline__ void store_piece(float* p, const Piece<V>& r) {
  if constexpr (V == 4) *reinterpret_cast<float4*>(p) = make_float4(r.v[0], r.v[1], r.v[2], r.v[3]);
  else *p = r.v[0];
}

// y = relu?(y + residual), in place; num_batches += 1 (BatchNorm's count of what it has seen).
template <int V>
__global__ void __launch_bounds__(256) bn_finish_kernel(float* __restrict__ y, const float* __restrict__ residual,
                                                        long long pieces, int relu, long long* num_batches) {
  grid_dependency_trigger();
  grid_dependency_wait();
  if (num_batches != nullptr && blockIdx.x == 0 && threadIdx.x == 0) *num_batches += 1;
  for (long long i = blockIdx.x * 256LL + threadIdx.x; i < pieces; i += gridDim.x * 256LL) {
    Piece<V> p = load_piece<V>(y + i * V);
    if (residual != nullptr) {
      const Piece<V> r = load_piece<V>(residual + i * V);
#pragma unroll
      for (int j = 0; j < V; ++j) p.v[j] += r.v[j];
    }
    if (relu) {
#pragma unroll
      for (int j = 0; j < V; ++j) p.v[j] = p.v[j] != p.v[j] ? p.v[j] : fmaxf(p.v[j], 0.f);     // (a NaN stays, as in torch)
    }
    store_piece<V>(y + i * V, p);
  }
}

// gx = weight * invstd * (g - mean(g) - xhat * mean(g * xhat)),  g = gy where the output is above zero.
template <int V>
__global__ void __launch_bounds__(kBnThreads) bn_backward_kernel(const BnArgs a) {
  extern __shared__ __align__(16) float kept[];      // x, then g, `keep` values each
  __shared__ double2 warps[kBnThreads / 32], total;
  constexpr int kUnroll = V == 4 ? 2 : 4;
  const unsigned part = cg::this_cluster().block_rank();
  const int c = blockIdx.x / a.cluster, first = part * a.per, tid = threadIdx.x;
  const int n = max(0, min(a.per, a.rows - first)) / V;
  const int keep = min(n, a.keep / V);
  float* kept_g = kept + a.keep;
  const long long base = (long long)c * a.rows + first;
  grid_dependency_trigger();
  grid_dependency_wait();
  auto load_g = [&](long long at) {
    Piece<V> g = load_piece<V>(a.gy + at);
    if (a.out != nullptr) {
      const Piece<V> o = load_piece<V>(a.out + at);
#pragma unroll
      for (int j = 0; j < V; ++j) g.v[j] = o.v[j] <= 0.f ? 0.f : g.v[j];
    }
    return g;
  };
  double sg = 0., sx = 0.;
  for (int i0 = tid; i0 < n; i0 += kUnroll * kBnThreads) {
    Piece<V> p[kUnroll], g[kUnroll];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const int i = i0 + u * kBnThreads;
      if (i < n) {
        p[u] = load_piece<V>(a.x + base + (long long)i * V);
        g[u] = load_g(base + (long long)i * V);
      }
    }
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const int i = i0 + u * kBnThreads;
      if (i >= n) break;
#pragma unroll
      for (int j = 0; j < V; ++j) {
        const double d = (double)g[u].v[j];
        sg += d;
        sx = fma(d, (double)p[u].v[j], sx);
      }
      if (i < keep) {
        store_piece<V>(kept + i * V, p[u]);
        store_piece<V>(kept_g + i * V, g[u]);
      }
    }
  }
  const double2 sum = cluster_sum(sg, sx, warps, &total);
  const float mean = a.mean[c], invstd = a.invstd[c];
  const double dot = sum.y - (double)mean * sum.x;            // sum of g * (x - mean)
  if (part == 0 && tid == 0) {
    a.g_weight[c] = (float)(dot * (double)invstd);
    a.g_bias[c] = (float)sum.x;
  }
  const float gmean = (float)(sum.x / a.rows), slope = (float)(dot / a.rows * (double)invstd * (double)invstd);
  const float scale = invstd * a.weight[c];
  for (int i0 = tid; i0 < n; i0 += kUnroll * kBnThreads) {
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const int i = i0 + u * kBnThreads;
      if (i >= n) break;
      Piece<V> p, g;
      if (i < keep) {
        p = load_piece<V>(kept + i * V);
        g = load_piece<V>(kept_g + i * V);
      } else {
        p = load_piece<V>(a.x + base + (long long)i * V);
        g = load_g(base + (long long)i * V);
      }
#pragma unroll
      for (int j = 0; j < V; ++j) p.v[j] = (g.v[j] - gmean - (p.v[j] - mean) * slope) * scale;
      store_piece<V>(a.gx + base + (long long)i * V, p);
    }
  }
}

// Cluster size: doubled while a CTA still has 4096 rows or more (eight a thread: less does not pay for the
// exchange) and the GPU is not full (four CTAs an SM), or the slice does not fit into shared memory.  In us with data
// in L2, 1 / 2 / 4 / 8 CTAs a channel: 16 channels x 40 k rows 14.0 / 10.8 / 8.9 / 8.7 (the rule takes 8), 64 x 107 k
// 65 / 33 / 35 / 34 (8), 256 x 107 k 169 / 137 / 136 / 123 (8), 256 x 16 k 14.5 / 13.5 / 14.2 / 22.8 (4), 256 x 4 k
// 8.8 / 8.8 / 9.4 / 19.7 (2); it is off the best at 128 x 16 k, 8.7 / 8.9 / 8.8 / 12.5 (8).
int bn_backward(BnArgs a, bool vec, cudaStream_t st) {
  constexpr size_t kRowBytes = 8;              // x and g
  int cluster = 1;
  while (cluster < kMaxCluster &&
         (((size_t)a.rows * kRowBytes > cluster * kBnSmem) ||
          (a.rows >= 4096 * cluster && (long long)a.channels * cluster < 4LL * sm_count())))
    cluster *= 2;
  a.cluster = cluster;
  a.per = ((a.rows + cluster - 1) / cluster + 3) / 4 * 4;
  const int most = (int)(kBnSmem / kRowBytes);
  a.keep = a.per < most ? a.per : most;
  typedef void (*Fn)(const BnArgs);
  static const Fn table[2] = {bn_backward_kernel<1>, bn_backward_kernel<4>};
  static PerDeviceOnce attr_once;
  const int limits = attr_once.run([&]() -> int {
    for (Fn f : table)
      OCNN_CUDA_OK(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBnSmem));
    return OCNN_OK;
  });
  if (limits != OCNN_OK) return limits;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)cluster * a.channels);
  cfg.blockDim = dim3(kBnThreads);
  cfg.dynamicSmemBytes = (size_t)a.keep * kRowBytes;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  OCNN_CUDA_OK(cudaLaunchKernelEx(&cfg, table[vec ? 1 : 0], a));
  OCNN_LAUNCH_OK("bn_backward_kernel");
  return OCNN_OK;
}

bool aligned16(const void* p) { return (uintptr_t)p % 16 == 0; }      // (true for NULL)

}  // namespace
}  // namespace ocnn

extern "C" {

int ocnn_batch_norm_finish(float* y, const float* residual, int64_t count, int relu, int64_t* num_batches,
                           void* stream) {
  using namespace ocnn;
  OCNN_REQUIRE(count >= 0 && (count == 0 || y), "ocnn_batch_norm_finish: null pointer");
  if (count == 0 && num_batches == nullptr) return OCNN_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  long long* seen = reinterpret_cast<long long*>(num_batches);
  if (residual == nullptr && !relu) count = 0;               // only the counter
  if (count % 4 == 0 && aligned16(y) && aligned16(residual))
    OCNN_CUDA_OK(launch_chained(bn_finish_kernel<4>, dim3(grid_for(count / 4, 256)), dim3(256), 0, st, y, residual,
                                (long long)(count / 4), relu, seen));
  else
    OCNN_CUDA_OK(launch_chained(bn_finish_kernel<1>, dim3(grid_for(count, 256)), dim3(256), 0, st, y, residual,
                                (long long)count, relu, seen));
  OCNN_LAUNCH_OK("bn_finish_kernel");
  return OCNN_OK;
}

int ocnn_batch_norm_backward(const float* x, const float* gy, const float* out, float* gx, int channels, int rows,
                             const float* weight, const float* save_mean, const float* save_invstd, float* g_weight,
                             float* g_bias, void* stream) {
  using namespace ocnn;
  OCNN_REQUIRE(channels > 0 && channels < (1 << 28) && rows > 1,
               "ocnn_batch_norm_backward: channels (%d) and more than one row (%d)", channels, rows);
  OCNN_REQUIRE(x && gy && gx && weight && save_mean && save_invstd && g_weight && g_bias,
               "ocnn_batch_norm_backward: null pointer");
  BnArgs a = {};
  a.x = x; a.gy = gy; a.out = out; a.gx = gx; a.weight = weight;
  a.mean = save_mean; a.invstd = save_invstd; a.g_weight = g_weight; a.g_bias = g_bias;
  a.channels = channels; a.rows = rows;
  const bool vec = rows % 4 == 0 && aligned16(x) && aligned16(gy) && aligned16(out) && aligned16(gx);
  return bn_backward(a, vec, static_cast<cudaStream_t>(stream));
}

}  // extern "C"
