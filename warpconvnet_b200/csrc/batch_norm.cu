// Batch normalisation of [N, C] rows in training, with the ReLU and the residual addition behind it.
//
// Bound by HBM / L2: forward reads the rows twice (statistics, then normalise) and writes them once, backward reads rows
// and gradient twice and writes one (two with a residual).  As separate torch kernels a conv block's tail also wrote and
// re-read the normalised rows for the ReLU and the sum, and its statistics kernels ran far below the memory rate
// (240 000 x 64 bf16: statistics 36 us, normalise 21, backward reductions 41, input gradient 16, ReLU 7 + 7).
// A thread owns 16 bytes of channels and walks rows; the last block to finish adds the blocks' partial sums in order (the
// same bits on every run) and leaves mean, 1 / std and the running statistics, so each direction is two launches.
// Sums are of differences from a typical value of the channel, which keeps the variance where the mean is large against
// the spread: the median of five rows spread over the matrix.  (The first row alone put (first row - mean)^2 / variance
// roundings on the variance: a first row of 1 000 before values of unit spread, fp32: 5e-4 of it for 50 001 rows, 3e-3 for
// 200 000.  A mean and deviations of every thread's own, put together in fp64, need no such value but took 27 us instead of
// 19 for 60 000 x 64 fp32, 40 instead of 31 for 240 000 x 64 fp16.)
#include <string.h>

#include "wcn_common.cuh"

namespace {

constexpr int THREADS = 512;
constexpr int MAX_C = 1024;

template <typename T> struct Piece {
  static constexpr int N = 16 / (int)sizeof(T);
  T v[N];
};
template <typename T> __device__ __forceinline__ Piece<T> load_piece(const T* p) {
  Piece<T> q;
  *reinterpret_cast<uint4*>(q.v) = __ldg(reinterpret_cast<const uint4*>(p));
  return q;
}

struct NormParams {
  const void* x;
  const void* dy;          // backward
  const void* res;         // forward: residual (or null)
  const void* y;           // backward with a residual: the output, whose sign is the ReLU's mask
  void* out;               // forward: y, backward: dx
  void* dres;              // backward: gradient of the residual (or null)
  const float* gamma;      // null: 1
  const float* beta;       // null: 0
  float* mean;             // [C] saved
  float* rstd;             // [C] saved
  float* sums;             // [2][C]: backward: d beta, d gamma
  float* running_mean;     // may be null
  float* running_var;
  int64_t* batches;        // num_batches_tracked, may be null
  float* partial;          // [blocks][2][C]
  unsigned* counter;       // zero before, zero after
  int64_t N;
  int C;
  float eps, momentum;
  int relu;
};

constexpr int TOTALS_AT = THREADS * 4 * sizeof(double);  // bytes of the groups' sums below

// Leaves this block's 2C sums (in smem[0..2C) as floats) in the workspace; true in the last block to do so, which adds the
// blocks' sums in order - four values a thread, the blocks dealt to groups of threads, the groups' sums added in order -
// and has the totals at smem + TOTALS_AT.
__device__ bool last_block_totals(const NormParams& p, uint8_t* smem) {
  __shared__ bool last;
  const float* mine = reinterpret_cast<const float*>(smem);
  const int n = 2 * p.C, quads = n / 4, groups = THREADS / quads;
  for (int i = threadIdx.x; i < n; i += THREADS) p.partial[(int64_t)blockIdx.x * n + i] = mine[i];
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(p.counter, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return false;
  __threadfence();
  double* sums = reinterpret_cast<double*>(smem);
  const int g = threadIdx.x / quads, q = threadIdx.x % quads;
  if (g < groups) {
    double t[4] = {0, 0, 0, 0};
    for (int b0 = g; b0 < (int)gridDim.x; b0 += 8 * groups) {
      float4 v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int b = b0 + u * groups;
        v[u] = b < (int)gridDim.x ? __ldcg(reinterpret_cast<const float4*>(p.partial + (int64_t)b * n) + q) : make_float4(0, 0, 0, 0);
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) { t[0] += v[u].x; t[1] += v[u].y; t[2] += v[u].z; t[3] += v[u].w; }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) sums[g * n + q * 4 + j] = t[j];
  }
  __syncthreads();
  double* tot = reinterpret_cast<double*>(smem + TOTALS_AT);
  for (int i = threadIdx.x; i < n; i += THREADS) {
    double v = sums[i];
    for (int r = 1; r < groups; ++r) v += sums[r * n + i];
    tot[i] = v;
  }
  if (threadIdx.x == 0) *p.counter = 0;
  __syncthreads();
  return true;
}

constexpr int SAMPLES = 5;
__device__ __forceinline__ int64_t sample_row(int64_t N, int j) { return j < 2 ? j * (N / 4) : j == 2 ? N / 2 : N - 1 - (4 - j) * (N / 4); }
__device__ __forceinline__ float median(const float (&v)[SAMPLES]) {
  const float lo = fmaxf(fminf(v[0], v[1]), fminf(v[2], v[3])), hi = fminf(fmaxf(v[0], v[1]), fmaxf(v[2], v[3]));
  return fmaxf(fminf(v[4], lo), fminf(fmaxf(v[4], lo), hi));
}

template <typename T>
__global__ void __launch_bounds__(THREADS) norm_stats_kernel(const NormParams p) {
  constexpr int V = Piece<T>::N;
  extern __shared__ __align__(16) uint8_t smem_raw[];
  float* s = reinterpret_cast<float*>(smem_raw);                       // [tys][2][C]
  const int txs = p.C / V, tys = THREADS / txs, tx = threadIdx.x % txs, ty = threadIdx.x / txs;
  const T* x = reinterpret_cast<const T*>(p.x);
  const int c0 = tx * V;
  float a[V], b[V], k[V];
#pragma unroll
  for (int i = 0; i < V; ++i) a[i] = b[i] = k[i] = 0.f;
  if (ty < tys) {
    Piece<T> of[SAMPLES];
#pragma unroll
    for (int j = 0; j < SAMPLES; ++j) of[j] = load_piece(x + sample_row(p.N, j) * p.C + c0);
#pragma unroll
    for (int i = 0; i < V; ++i) {
      float v[SAMPLES];
#pragma unroll
      for (int j = 0; j < SAMPLES; ++j) v[j] = wcn_to_float<T>(of[j].v[i]);
      k[i] = median(v);
    }
    const int64_t step = (int64_t)gridDim.x * tys;
    for (int64_t r = (int64_t)blockIdx.x * tys + ty; r < p.N; r += 4 * step) {
      Piece<T> q[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) q[u] = load_piece(x + (r + u * step < p.N ? r + u * step : 0) * p.C + c0);
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int i = 0; i < V; ++i) {
          const float d = r + u * step < p.N ? wcn_to_float<T>(q[u].v[i]) - k[i] : 0.f;
          a[i] += d;
          b[i] = fmaf(d, d, b[i]);
        }
    }
  }
  if (ty < tys) {
#pragma unroll
    for (int i = 0; i < V; ++i) { s[(ty * 2) * p.C + c0 + i] = a[i]; s[(ty * 2 + 1) * p.C + c0 + i] = b[i]; }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * p.C; i += THREADS) {
    float v = s[i];
    for (int r = 1; r < tys; ++r) v += s[r * 2 * p.C + i];
    s[i] = v;
  }
  __syncthreads();
  if (!last_block_totals(p, smem_raw)) return;
  const double* tot = reinterpret_cast<const double*>(smem_raw + TOTALS_AT);
  for (int c = threadIdx.x; c < p.C; c += THREADS) {
    float v[SAMPLES];
#pragma unroll
    for (int j = 0; j < SAMPLES; ++j) v[j] = wcn_to_float<T>(x[sample_row(p.N, j) * p.C + c]);
    const double n = (double)p.N, shift = (double)median(v);
    const double d = tot[c] / n;
    double var = tot[p.C + c] / n - d * d;
    if (var < 0) var = 0;
    const double mean = shift + d;
    p.mean[c] = (float)mean;
    p.rstd[c] = (float)(1.0 / sqrt(var + (double)p.eps));
    if (p.running_mean) {
      p.running_mean[c] = (1.f - p.momentum) * p.running_mean[c] + p.momentum * (float)mean;
      p.running_var[c] = (1.f - p.momentum) * p.running_var[c] + p.momentum * (float)(var * n / (n - 1.0));
    }
  }
  if (threadIdx.x == 0 && p.batches) *p.batches += 1;
}

template <typename T>
__global__ void __launch_bounds__(THREADS) norm_apply_kernel(const NormParams p) {
  constexpr int V = Piece<T>::N;
  const int txs = p.C / V, tys = THREADS / txs, tx = threadIdx.x % txs, ty = threadIdx.x / txs;
  if (ty >= tys) return;
  const int c0 = tx * V;
  float mean[V], scale[V], beta[V];
#pragma unroll
  for (int i = 0; i < V; ++i) {
    mean[i] = p.mean[c0 + i];
    scale[i] = p.rstd[c0 + i] * (p.gamma ? __ldg(&p.gamma[c0 + i]) : 1.f);
    beta[i] = p.beta ? __ldg(&p.beta[c0 + i]) : 0.f;
  }
  const T* x = reinterpret_cast<const T*>(p.x);
  const T* res = reinterpret_cast<const T*>(p.res);
  const int64_t step = (int64_t)gridDim.x * tys;
  for (int64_t r0 = (int64_t)blockIdx.x * tys + ty; r0 < p.N; r0 += 2 * step) {
    Piece<T> q[2], e[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int64_t r = r0 + u * step;
      if (r < p.N) {
        q[u] = load_piece(x + r * p.C + c0);
        if (res) e[u] = load_piece(res + r * p.C + c0);
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int64_t r = r0 + u * step;
      if (r >= p.N) break;
      Piece<T> o;
#pragma unroll
      for (int i = 0; i < V; ++i) {
        // rounded where the separate layers round: after the normalisation and after the addition
        T z = wcn_from_float<T>(fmaf(wcn_to_float<T>(q[u].v[i]) - mean[i], scale[i], beta[i]));
        if (res) z = wcn_from_float<T>(wcn_to_float<T>(z) + wcn_to_float<T>(e[u].v[i]));
        const float f = wcn_to_float<T>(z);
        o.v[i] = p.relu && !(f > 0.f) && f == f ? wcn_from_float<T>(0.f) : z;
      }
      *reinterpret_cast<uint4*>(reinterpret_cast<T*>(p.out) + r * p.C + c0) = *reinterpret_cast<const uint4*>(o.v);
    }
  }
}

// dz = dy where the ReLU let the value through.  Without a residual the sign is recomputed from x.
template <typename T>
__device__ __forceinline__ float masked(const NormParams& p, float g, float x, float mean, float scale, float beta, bool has_y, T y) {
  if (!p.relu) return g;
  const float z = has_y ? wcn_to_float<T>(y) : wcn_to_float<T>(wcn_from_float<T>(fmaf(x - mean, scale, beta)));
  return z > 0.f || z != z ? g : 0.f;
}

template <typename T>
__global__ void __launch_bounds__(THREADS) norm_backward_sums_kernel(const NormParams p) {
  constexpr int V = Piece<T>::N;
  extern __shared__ __align__(16) uint8_t smem_raw[];
  float* s = reinterpret_cast<float*>(smem_raw);
  const int txs = p.C / V, tys = THREADS / txs, tx = threadIdx.x % txs, ty = threadIdx.x / txs;
  const int c0 = tx * V;
  const T *x = reinterpret_cast<const T*>(p.x), *dy = reinterpret_cast<const T*>(p.dy), *y = reinterpret_cast<const T*>(p.y);
  float a[V], b[V], mean[V], scale[V], beta[V];
#pragma unroll
  for (int i = 0; i < V; ++i) a[i] = b[i] = 0.f;
  if (ty < tys) {
#pragma unroll
    for (int i = 0; i < V; ++i) {
      mean[i] = p.mean[c0 + i];
      scale[i] = p.rstd[c0 + i] * (p.gamma ? __ldg(&p.gamma[c0 + i]) : 1.f);
      beta[i] = p.beta ? __ldg(&p.beta[c0 + i]) : 0.f;
    }
    const int64_t step = (int64_t)gridDim.x * tys;
    for (int64_t r0 = (int64_t)blockIdx.x * tys + ty; r0 < p.N; r0 += 2 * step) {
      Piece<T> q[2], g[2], o[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int64_t r = r0 + u * step;
        if (r < p.N) {
          q[u] = load_piece(x + r * p.C + c0);
          g[u] = load_piece(dy + r * p.C + c0);
          if (y) o[u] = load_piece(y + r * p.C + c0);
        }
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        if (r0 + u * step >= p.N) break;
#pragma unroll
        for (int i = 0; i < V; ++i) {
          const float xv = wcn_to_float<T>(q[u].v[i]);
          const float dz = masked<T>(p, wcn_to_float<T>(g[u].v[i]), xv, mean[i], scale[i], beta[i], y != nullptr, o[u].v[i]);
          a[i] += dz;
          b[i] = fmaf(dz, xv - mean[i], b[i]);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < V; ++i) { s[(ty * 2) * p.C + c0 + i] = a[i]; s[(ty * 2 + 1) * p.C + c0 + i] = b[i]; }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * p.C; i += THREADS) {
    float v = s[i];
    for (int r = 1; r < tys; ++r) v += s[r * 2 * p.C + i];
    s[i] = v;
  }
  __syncthreads();
  if (!last_block_totals(p, smem_raw)) return;
  const double* tot = reinterpret_cast<const double*>(smem_raw + TOTALS_AT);
  for (int c = threadIdx.x; c < p.C; c += THREADS) {
    p.sums[c] = (float)tot[c];
    p.sums[p.C + c] = (float)(tot[p.C + c] * (double)p.rstd[c]);
  }
}

template <typename T>
__global__ void __launch_bounds__(THREADS) norm_backward_apply_kernel(const NormParams p) {
  constexpr int V = Piece<T>::N;
  const int txs = p.C / V, tys = THREADS / txs, tx = threadIdx.x % txs, ty = threadIdx.x / txs;
  if (ty >= tys) return;
  const int c0 = tx * V;
  const T *x = reinterpret_cast<const T*>(p.x), *dy = reinterpret_cast<const T*>(p.dy), *y = reinterpret_cast<const T*>(p.y);
  float mean[V], scale[V], beta[V], k0[V], k1[V];
  const float inv_n = (float)(1.0 / (double)p.N);
#pragma unroll
  for (int i = 0; i < V; ++i) {
    const float rstd = p.rstd[c0 + i];
    mean[i] = p.mean[c0 + i];
    scale[i] = rstd * (p.gamma ? __ldg(&p.gamma[c0 + i]) : 1.f);
    beta[i] = p.beta ? __ldg(&p.beta[c0 + i]) : 0.f;
    k0[i] = p.sums[c0 + i] * inv_n;                      // mean of dz
    k1[i] = p.sums[p.C + c0 + i] * rstd * inv_n;         // mean of dz * xhat, over std
  }
  const int64_t step = (int64_t)gridDim.x * tys;
  for (int64_t r0 = (int64_t)blockIdx.x * tys + ty; r0 < p.N; r0 += 2 * step) {
    Piece<T> q[2], g[2], o[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int64_t r = r0 + u * step;
      if (r < p.N) {
        q[u] = load_piece(x + r * p.C + c0);
        g[u] = load_piece(dy + r * p.C + c0);
        if (y) o[u] = load_piece(y + r * p.C + c0);
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int64_t r = r0 + u * step;
      if (r >= p.N) break;
      Piece<T> dx, dz_out;
#pragma unroll
      for (int i = 0; i < V; ++i) {
        const float xv = wcn_to_float<T>(q[u].v[i]);
        const float dz = masked<T>(p, wcn_to_float<T>(g[u].v[i]), xv, mean[i], scale[i], beta[i], y != nullptr, o[u].v[i]);
        dx.v[i] = wcn_from_float<T>((dz - k0[i] - (xv - mean[i]) * k1[i]) * scale[i]);
        dz_out.v[i] = wcn_from_float<T>(dz);
      }
      *reinterpret_cast<uint4*>(reinterpret_cast<T*>(p.out) + r * p.C + c0) = *reinterpret_cast<const uint4*>(dx.v);
      if (p.dres) *reinterpret_cast<uint4*>(reinterpret_cast<T*>(p.dres) + r * p.C + c0) = *reinterpret_cast<const uint4*>(dz_out.v);
    }
  }
}

inline int norm_blocks(int64_t N, int C, int elem) {
  const int tys = THREADS / (C / (16 / elem));
  const int64_t want = (N + 4 * tys - 1) / (4 * tys);  // at least four rows a thread
  const int64_t most = 2 * (int64_t)wcn_num_sms();
  return (int)(want < most ? want : most);
}

inline size_t norm_smem(int C, int elem) {
  const size_t rows = (size_t)(THREADS / (C / (16 / elem))) * 2 * C * sizeof(float), totals = TOTALS_AT + (size_t)2 * C * sizeof(double);
  return rows > totals ? rows : totals;
}

bool norm_ok(int64_t N, int C, int dtype) {
  if (dtype < WCN_F32 || dtype > WCN_BF16) return false;
  const int v = 16 / wcn_dtype_size(dtype);
  return N > 1 && C > 0 && C <= MAX_C && C % v == 0 && C / v <= THREADS;
}

bool on16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

template <typename T> int forward(const NormParams& p, cudaStream_t st) {
  const unsigned blocks = (unsigned)norm_blocks(p.N, p.C, sizeof(T));
  norm_stats_kernel<T><<<blocks, THREADS, norm_smem(p.C, sizeof(T)), st>>>(p);
  norm_apply_kernel<T><<<blocks, THREADS, 0, st>>>(p);
  return cudaGetLastError() == cudaSuccess ? WCN_OK : WCN_ERR_EXECUTION;
}

template <typename T> int backward(const NormParams& p, cudaStream_t st) {
  const unsigned blocks = (unsigned)norm_blocks(p.N, p.C, sizeof(T));
  norm_backward_sums_kernel<T><<<blocks, THREADS, norm_smem(p.C, sizeof(T)), st>>>(p);
  if (p.out) norm_backward_apply_kernel<T><<<blocks, THREADS, 0, st>>>(p);
  return cudaGetLastError() == cudaSuccess ? WCN_OK : WCN_ERR_EXECUTION;
}

}  // namespace

extern "C" int wcn_batch_norm_workspace_bytes(int64_t n, int32_t channels, int dtype, int64_t* bytes) {
  if (!bytes || n < 0 || channels <= 0) return WCN_ERR_INVALID_PARAMETERS;
  *bytes = norm_ok(n, channels, dtype) ? (int64_t)norm_blocks(n, channels, wcn_dtype_size(dtype)) * 2 * channels * 4 : 0;
  return WCN_OK;
}

static float from_bits(uint32_t b) {
  float f;
  memcpy(&f, &b, sizeof f);
  return f;
}

extern "C" int wcn_batch_norm_train(const void* x, int64_t n, int32_t channels, int dtype, const float* gamma, const float* beta,
                                    uint32_t eps_bits, uint32_t momentum_bits, float* running_mean, float* running_var,
                                    int64_t* num_batches, const void* residual, int relu, void* y, float* mean, float* rstd,
                                    void* workspace, uint32_t* counter, void* stream) {
  if (!norm_ok(n, channels, dtype)) return WCN_ERR_UNSUPPORTED_CONFIG;
  if (!x || !y || !mean || !rstd || !workspace || !counter || !on16(x) || !on16(y) || !on16(residual) || (running_mean && !running_var))
    return WCN_ERR_INVALID_PARAMETERS;
  NormParams p = {};
  p.x = x; p.res = residual; p.out = y; p.gamma = gamma; p.beta = beta; p.mean = mean; p.rstd = rstd;
  p.running_mean = running_mean; p.running_var = running_var; p.batches = num_batches;
  p.partial = (float*)workspace; p.counter = counter; p.N = n; p.C = channels; p.eps = from_bits(eps_bits); p.momentum = from_bits(momentum_bits); p.relu = relu;
  cudaStream_t st = wcn_stream(stream);
  if (dtype == WCN_F32) return forward<float>(p, st);
  if (dtype == WCN_F16) return forward<__half>(p, st);
  return forward<__nv_bfloat16>(p, st);
}

extern "C" int wcn_batch_norm_backward(const void* x, const void* dy, const void* y, int64_t n, int32_t channels, int dtype,
                                       const float* gamma, const float* beta, const float* mean, const float* rstd, int relu,
                                       void* dx, void* dresidual, float* sums, void* workspace, uint32_t* counter,
                                       void* stream) {
  if (!norm_ok(n, channels, dtype)) return WCN_ERR_UNSUPPORTED_CONFIG;
  if (!x || !dy || !mean || !rstd || !sums || !workspace || !counter || !on16(x) || !on16(dy) || !on16(y) || !on16(dx) ||
      !on16(dresidual) || (dresidual && !dx))
    return WCN_ERR_INVALID_PARAMETERS;
  NormParams p = {};
  p.x = x; p.dy = dy; p.y = y; p.out = dx; p.dres = dresidual; p.gamma = gamma; p.beta = beta;
  p.mean = const_cast<float*>(mean); p.rstd = const_cast<float*>(rstd); p.sums = sums;
  p.partial = (float*)workspace; p.counter = counter; p.N = n; p.C = channels; p.relu = relu;
  cudaStream_t st = wcn_stream(stream);
  if (dtype == WCN_F32) return backward<float>(p, st);
  if (dtype == WCN_F16) return backward<__half>(p, st);
  return backward<__nv_bfloat16>(p, st);
}
