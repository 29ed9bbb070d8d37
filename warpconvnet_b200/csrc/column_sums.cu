// Column sums of a matrix of contiguous rows: a layer's bias gradient.
//
// Bound by reading the matrix once.  Two launches: blocks of rows, a thread 16 bytes of eight rows at a time, leave partial sums; a
// block per 32 columns adds them in order.  Eight numbers are added in a tree in fp32, everything else in double: a thread of a
// large matrix has hundreds to thousands of rows (300 000 x 1024 fp32 one after the other in fp32: 5.8e-7 of the sums' 2-norm, torch
// 2.2e-7, here 5.4e-8).  No atomics: the same bits on every run.  us, torch's reduction / a row at a time / eight, L2 flushed:
// fp32 60 000 x 64 31 / 17 / 19, 800 000 x 128 303 / 119 / 91, 800 000 x 256 254 / 214 / 149, 300 000 x 1024 227 / 308 / 206, bf16 154 / 223 / 134.
#include "wcn_common.cuh"

namespace {

constexpr int THREADS = 256, SLICES = 8, ROWS = 8;   // ROWS: of a thread at a time

template <typename T>
__global__ void __launch_bounds__(THREADS) column_partials_kernel(const T* __restrict__ x, int64_t n, int c, double* __restrict__ partial) {
  constexpr int V = 16 / (int)sizeof(T);
  __shared__ double part[THREADS * V];
  const int across = c / V, lanes = THREADS / across;          // threads of a row, rows at a time
  const int col = (int)threadIdx.x % across * V, lane = (int)threadIdx.x / across;
  if (lane < lanes) {
    double sum[V];
#pragma unroll
    for (int u = 0; u < V; ++u) sum[u] = 0.;
    const int64_t step = (int64_t)gridDim.x * lanes;
    for (int64_t r = (int64_t)blockIdx.x * lanes + lane; r < n; r += ROWS * step) {
      uint4 q[ROWS];
#pragma unroll
      for (int i = 0; i < ROWS; ++i)
        q[i] = r + i * step < n ? __ldg(reinterpret_cast<const uint4*>(x + (r + i * step) * c + col)) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int u = 0; u < V; ++u) {
        float v[ROWS];
#pragma unroll
        for (int i = 0; i < ROWS; ++i) v[i] = wcn_to_float<T>(reinterpret_cast<const T*>(&q[i])[u]);
#pragma unroll
        for (int w = ROWS / 2; w > 0; w /= 2)
#pragma unroll
          for (int i = 0; i < w; ++i) v[i] += v[i + w];
        sum[u] += v[0];
      }
    }
#pragma unroll
    for (int u = 0; u < V; ++u) part[lane * c + col + u] = sum[u];
  }
  __syncthreads();
  for (int j = threadIdx.x; j < c; j += THREADS) {
    double s = 0.;
    for (int l = 0; l < lanes; ++l) s += part[l * c + j];
    partial[(int64_t)blockIdx.x * c + j] = s;
  }
}

__global__ void __launch_bounds__(32 * SLICES) column_totals_kernel(const double* __restrict__ partial, int blocks, int c, float* __restrict__ out) {
  __shared__ double part[SLICES][32];
  const int j = blockIdx.x * 32 + (threadIdx.x & 31), slice = threadIdx.x >> 5;
  double s = 0.;
  if (j < c)
#pragma unroll 8
    for (int b = slice; b < blocks; b += SLICES) s += __ldcg(&partial[(int64_t)b * c + j]);
  part[slice][threadIdx.x & 31] = s;
  __syncthreads();
  if (slice == 0 && j < c) {
    for (int q = 1; q < SLICES; ++q) s += part[q][threadIdx.x];
    out[j] = (float)s;
  }
}

int partial_blocks(int64_t n, int c, int width) {
  const int lanes = THREADS / (c / width);
  const int64_t want = (n + 4 * lanes - 1) / (4 * lanes), most = 2 * (int64_t)wcn_num_sms();   // four rows a thread at least
  return (int)(want < most ? want : most);
}

bool sums_supported(int64_t n, int c, int dtype) {
  const int width = dtype == WCN_F32 ? 4 : 8;
  return n > 0 && c > 0 && dtype >= WCN_F32 && dtype <= WCN_BF16 && c % width == 0 && c / width <= THREADS;
}

}  // namespace

extern "C" int wcn_column_sums_workspace_bytes(int64_t n, int32_t channels, int dtype, int64_t* bytes) {
  if (!bytes || n < 0 || channels <= 0) return WCN_ERR_INVALID_PARAMETERS;
  *bytes = sums_supported(n, channels, dtype) ? (int64_t)partial_blocks(n, channels, dtype == WCN_F32 ? 4 : 8) * channels * (int64_t)sizeof(double) : 0;
  return WCN_OK;
}

extern "C" int wcn_column_sums(const void* x, int64_t n, int32_t channels, int dtype, float* sums, void* workspace, void* stream) {
  if (!sums_supported(n, channels, dtype)) return WCN_ERR_UNSUPPORTED_CONFIG;
  if (!x || !sums || !workspace || (reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(workspace) & 7)) return WCN_ERR_INVALID_PARAMETERS;
  cudaStream_t st = wcn_stream(stream);
  double* partial = reinterpret_cast<double*>(workspace);
  const int blocks = partial_blocks(n, channels, dtype == WCN_F32 ? 4 : 8);
  if (dtype == WCN_F32) column_partials_kernel<float><<<blocks, THREADS, 0, st>>>((const float*)x, n, channels, partial);
  else if (dtype == WCN_F16) column_partials_kernel<__half><<<blocks, THREADS, 0, st>>>((const __half*)x, n, channels, partial);
  else column_partials_kernel<__nv_bfloat16><<<blocks, THREADS, 0, st>>>((const __nv_bfloat16*)x, n, channels, partial);
  column_totals_kernel<<<(channels + 31) / 32, 32 * SLICES, 0, st>>>(partial, blocks, channels, sums);
  WCN_CHECK_LAUNCH();
  return WCN_OK;
}
