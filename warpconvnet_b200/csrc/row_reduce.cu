// Pooling over a kernel map: output row m reduces the feature rows nbr[k][m] >= 0, forward and backward.
//
// Bound by latency first and HBM second: a row is a table entry per offset and, behind it, one feature row.
// A thread owns 16 bytes of channels of one row and requests kAhead table entries together, then the rows
// they name together, so two memory latencies cover kAhead offsets (a 2x2x2 window is one such round).
#include "wcn_common.cuh"

namespace {

constexpr int kAhead = 8;

template <typename T, int VEC>
__device__ __forceinline__ void load_piece(const T* __restrict__ src, T (&v)[VEC]) {
  if constexpr (VEC > 1) {
    static_assert(VEC * sizeof(T) == 16, "one 16-byte piece");
    *reinterpret_cast<uint4*>(v) = __ldg(reinterpret_cast<const uint4*>(src));
  } else {
    v[0] = __ldg(src);
  }
}

template <typename T, int VEC>
__device__ __forceinline__ void store_piece(T* dst, const T (&v)[VEC]) {
  if constexpr (VEC > 1) *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(v);
  else dst[0] = v[0];
}

// Row and first channel of thread t.  32-bit division where the problem allows: the 64-bit one is a long
// instruction sequence in front of the first load.
__device__ __forceinline__ void split_thread(int64_t t, int per_row, bool narrow, int64_t* row, int* piece) {
  if (narrow) {
    const uint32_t q = (uint32_t)t / (uint32_t)per_row;
    *row = q;
    *piece = (int)((uint32_t)t - q * (uint32_t)per_row);
  } else {
    *row = t / per_row;
    *piece = (int)(t - *row * per_row);
  }
}

// out[m, :] = reduce over the offsets k that have a neighbour (nbr[k*M + m] >= 0) of
// feats[nbr[k*M + m], :] in order of k, in fp32; rows without any neighbour become 0.
// arg (min, max; may be null): per element the first offset that attained the result, kNoArg where there is none.
// count (mean; may be null): neighbours of every row, at least 1.
// (The reduction is a template argument: decided per element, an un-pooling to 250 000 rows of 64 channels executed 1 200
// instructions a warp and took 65 us; 36 us now, with the single row of such a map taken by itself.)
enum RowOp { ROW_SUM = 0, ROW_EXTREMUM = 1, ROW_MUL = 2 };   // ROW_SUM: sum and mean, ROW_EXTREMUM: min and max
template <typename T, int VEC, typename TA, int OP>
__global__ void row_reduce_kernel(const T* __restrict__ feats, int num_in, const int32_t* __restrict__ nbr, int64_t M,
                                  int K, int channels, int op, bool narrow, T* __restrict__ out, TA* __restrict__ arg,
                                  float* __restrict__ count_out, int32_t* dev_status) {
  int64_t m;
  int piece;
  split_thread((int64_t)blockIdx.x * blockDim.x + threadIdx.x, channels / VEC, narrow, &m, &piece);
  if (m >= M) return;
  const int c0 = piece * VEC;
  float acc[VEC];
  TA at[VEC];
#pragma unroll
  for (int i = 0; i < VEC; ++i) { acc[i] = 0.f; at[i] = (TA)~(TA)0; }
  int count = 0;
  bool bad = false;
  auto take = [&](const T (&x_of)[VEC], int k) {   // row of offset k
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
      const float x = wcn_to_float<T>(x_of[i]);
      if constexpr (OP == ROW_SUM) {
        acc[i] = count == 0 ? x : __fadd_rn(acc[i], x);
        continue;
      }
      if (OP == ROW_EXTREMUM) {
        // a later value takes the place only if it is strictly beyond (or follows a NaN): the first one that
        // attains the result keeps it
        const bool beyond = op == WCN_REDUCE_MAX ? x > acc[i] : x < acc[i];
        if (count == 0 ? x == x : (beyond || (acc[i] != acc[i] && x == x))) at[i] = (TA)k;
      }
      if (count == 0) acc[i] = x;
      else if (OP == ROW_EXTREMUM) acc[i] = op == WCN_REDUCE_MAX ? fmaxf(acc[i], x) : fminf(acc[i], x);
      else acc[i] = __fmul_rn(acc[i], x);
    }
    ++count;
  };
  for (int k0 = 0; k0 < K; k0 += kAhead) {
    int src[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) src[u] = k0 + u < K ? __ldg(&nbr[(int64_t)(k0 + u) * M + m]) : -1;
    int present = 0, one = 0, at_one = 0;
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      if (src[u] >= num_in) { bad = true; src[u] = -1; }  // not a feature row: counts as absent, reported once below
      if (src[u] >= 0) { ++present; one = src[u]; at_one = k0 + u; }
    }
    __align__(16) T v[kAhead][VEC];
    if (present <= 1) {  // the finer side of a strided map: a single row instead of eight conditional ones
      if (present) {
        load_piece<T, VEC>(feats + (int64_t)one * channels + c0, v[0]);
        take(v[0], at_one);
      }
      continue;
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u)
      if (src[u] >= 0) load_piece<T, VEC>(feats + (int64_t)src[u] * channels + c0, v[u]);
#pragma unroll
    for (int u = 0; u < kAhead; ++u)
      if (src[u] >= 0) take(v[u], k0 + u);
  }
  __align__(16) T o[VEC];
#pragma unroll
  for (int i = 0; i < VEC; ++i) {
    float y = acc[i];
    if (OP == ROW_SUM && op == WCN_REDUCE_MEAN && count) y = __fdiv_rn(y, (float)count);
    o[i] = wcn_from_float<T>(y);
  }
  store_piece<T, VEC>(out + m * channels + c0, o);
  if (arg) {
#pragma unroll
    for (int i = 0; i < VEC; ++i) arg[m * channels + c0 + i] = at[i];
  }
  if (count_out && piece == 0) count_out[m] = count > 1 ? (float)count : 1.f;
  if (bad) wcn_report_bounds(dev_status);
}

// Gradient of the above: grad_in[i, :] = sum over the offsets k with m = nbr_t[k*N + i] >= 0 of
//   sum         grad_out[m]
//   mean        grad_out[m] / count[m]
//   min, max    grad_out[m] where arg[m] == k
// Every input row gathers what it is due: no atomics, summed in order of k in fp32, rounded once.
template <typename T, int VEC, typename TA, bool ARG>
__global__ void row_reduce_backward_kernel(const T* __restrict__ gout, int num_out, const int32_t* __restrict__ nbr_t,
                                           int64_t N, int K, int channels, bool narrow, const TA* __restrict__ arg,
                                           const float* __restrict__ count, T* __restrict__ gin, int32_t* dev_status) {
  int64_t n;
  int piece;
  split_thread((int64_t)blockIdx.x * blockDim.x + threadIdx.x, channels / VEC, narrow, &n, &piece);
  if (n >= N) return;
  const int c0 = piece * VEC;
  float acc[VEC];
#pragma unroll
  for (int i = 0; i < VEC; ++i) acc[i] = 0.f;
  bool bad = false;
  for (int k0 = 0; k0 < K; k0 += kAhead) {
    int src[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) src[u] = k0 + u < K ? __ldg(&nbr_t[(int64_t)(k0 + u) * N + n]) : -1;
    int present = 0, one = 0, at_one = 0;
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      if (src[u] >= num_out) { bad = true; src[u] = -1; }
      if (src[u] >= 0) { ++present; one = src[u]; at_one = k0 + u; }
    }
    __align__(16) T v[kAhead][VEC];
    __align__(16) TA a[kAhead][VEC];
    float c[kAhead];
    auto fetch = [&](int row, T (&g_of)[VEC], TA (&a_of)[VEC], float& c_of) {
      const int64_t at = (int64_t)row * channels + c0;
      load_piece<T, VEC>(gout + at, g_of);
      if constexpr (ARG) {
        if constexpr (VEC == 8 && sizeof(TA) == 1) *reinterpret_cast<uint2*>(a_of) = __ldg(reinterpret_cast<const uint2*>(arg + at));
        else if constexpr (VEC == 4 && sizeof(TA) == 1) *reinterpret_cast<uint32_t*>(a_of) = __ldg(reinterpret_cast<const uint32_t*>(arg + at));
        else {
#pragma unroll
          for (int i = 0; i < VEC; ++i) a_of[i] = __ldg(arg + at + i);
        }
      } else {
        c_of = count ? __ldg(&count[row]) : 1.f;
      }
    };
    auto take = [&](const T (&g_of)[VEC], const TA (&a_of)[VEC], int k) {
#pragma unroll
      for (int i = 0; i < VEC; ++i) {
        const float g = wcn_to_float<T>(g_of[i]);
        if constexpr (ARG) {
          if (a_of[i] == (TA)k) acc[i] = __fadd_rn(acc[i], g);
        } else {
          acc[i] = __fadd_rn(acc[i], g);
        }
      }
    };
    auto take_mean = [&](const T (&g_of)[VEC], float c_of) {
#pragma unroll
      for (int i = 0; i < VEC; ++i) acc[i] = __fadd_rn(acc[i], __fdiv_rn(wcn_to_float<T>(g_of[i]), c_of));
    };
    const bool mean = !ARG && count;
    if (present <= 1) {
      if (present) {
        fetch(one, v[0], a[0], c[0]);
        if (mean) take_mean(v[0], c[0]);
        else take(v[0], a[0], at_one);
      }
      continue;
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u)
      if (src[u] >= 0) fetch(src[u], v[u], a[u], c[u]);
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      if (src[u] < 0) continue;
      if (mean) take_mean(v[u], c[u]);
      else take(v[u], a[u], k0 + u);
    }
  }
  __align__(16) T o[VEC];
#pragma unroll
  for (int i = 0; i < VEC; ++i) o[i] = wcn_from_float<T>(acc[i]);
  store_piece<T, VEC>(gin + n * channels + c0, o);
  if (bad) wcn_report_bounds(dev_status);
}

constexpr int kThreads = 256;

// 16-byte pieces when a row is a whole number of them and the matrices are aligned to them, else single elements.
template <typename T>
bool in_pieces(int channels, const void* a, const void* b) {
  return channels % (int)(16 / sizeof(T)) == 0 && !(reinterpret_cast<uintptr_t>(a) & 15) && !(reinterpret_cast<uintptr_t>(b) & 15);
}

template <typename T, typename TA>
int launch_row_reduce(const void* feats, int num_in, const int32_t* nbr, int64_t M, int K, int channels, int op,
                      void* out, void* arg, float* count, int32_t* dev_status, cudaStream_t st) {
  constexpr int V = (int)(16 / sizeof(T));
  const bool vec = in_pieces<T>(channels, feats, out);
  const int64_t total = M * (channels / (vec ? V : 1));
  const unsigned grid = (unsigned)((total + kThreads - 1) / kThreads);
  const bool narrow = total + kThreads < 0xFFFFFFFFll;
#define WCN_ROW_LAUNCH(VEC, OP)                                                                                          \
  row_reduce_kernel<T, VEC, TA, OP><<<grid, kThreads, 0, st>>>((const T*)feats, num_in, nbr, M, K, channels, op, narrow, \
                                                              (T*)out, (TA*)arg, count, dev_status)
  if (op == WCN_REDUCE_MIN || op == WCN_REDUCE_MAX) {
    if (vec) WCN_ROW_LAUNCH(V, ROW_EXTREMUM);
    else WCN_ROW_LAUNCH(1, ROW_EXTREMUM);
  } else if (op == WCN_REDUCE_MUL) {
    if (vec) WCN_ROW_LAUNCH(V, ROW_MUL);
    else WCN_ROW_LAUNCH(1, ROW_MUL);
  } else {
    if (vec) WCN_ROW_LAUNCH(V, ROW_SUM);
    else WCN_ROW_LAUNCH(1, ROW_SUM);
  }
#undef WCN_ROW_LAUNCH
  return cudaGetLastError() == cudaSuccess ? WCN_OK : WCN_ERR_EXECUTION;
}

template <typename T, typename TA>
int launch_row_reduce_backward(const void* gout, int num_out, const int32_t* nbr_t, int64_t N, int K, int channels,
                               const void* arg, const float* count, void* gin, int32_t* dev_status, cudaStream_t st) {
  constexpr int V = (int)(16 / sizeof(T));
  const bool vec = in_pieces<T>(channels, gout, gin) && !(reinterpret_cast<uintptr_t>(arg) & 7);
  const int64_t total = N * (channels / (vec ? V : 1));
  const unsigned grid = (unsigned)((total + kThreads - 1) / kThreads);
  const bool narrow = total + kThreads < 0xFFFFFFFFll;
#define WCN_ROW_LAUNCH(VEC, ARG)                                                                                         \
  row_reduce_backward_kernel<T, VEC, TA, ARG><<<grid, kThreads, 0, st>>>((const T*)gout, num_out, nbr_t, N, K, channels, \
                                                                        narrow, (const TA*)arg, count, (T*)gin, dev_status)
  if (arg) {
    if (vec) WCN_ROW_LAUNCH(V, true);
    else WCN_ROW_LAUNCH(1, true);
  } else {
    if (vec) WCN_ROW_LAUNCH(V, false);
    else WCN_ROW_LAUNCH(1, false);
  }
#undef WCN_ROW_LAUNCH
  return cudaGetLastError() == cudaSuccess ? WCN_OK : WCN_ERR_EXECUTION;
}

}  // namespace

extern "C" int wcn_row_reduce_train(const void* feats, int64_t num_in, const int32_t* nbr, int64_t num_out,
                              int32_t num_offsets, int32_t channels, int dtype, int op, void* out, void* arg,
                              int32_t arg_bytes, float* count, int32_t* dev_status, void* stream) {
  if (num_out < 0 || num_in < 0 || num_offsets <= 0 || channels <= 0 || op < WCN_REDUCE_MIN || op > WCN_REDUCE_MUL)
    return WCN_ERR_INVALID_PARAMETERS;
  const int nin = (int)(num_in < 0x7FFFFFFFll ? num_in : 0x7FFFFFFFll);
  if (num_out == 0) return WCN_OK;
  if (!nbr || !out) return WCN_ERR_INVALID_PARAMETERS;
  // an offset and the "none" mark must fit an argument
  if (arg && !((arg_bytes == 1 && num_offsets <= 255) || (arg_bytes == 2 && num_offsets <= 65535))) return WCN_ERR_INVALID_PARAMETERS;
  if ((int64_t)num_out * channels >= (int64_t)0x7FFFFFFF * 256) return WCN_ERR_INVALID_PARAMETERS;
  cudaStream_t st = wcn_stream(stream);
#define WCN_REDUCE_CASE(T)                                                                                            \
  return arg_bytes == 2                                                                                               \
             ? launch_row_reduce<T, uint16_t>(feats, nin, nbr, num_out, num_offsets, channels, op, out, arg, count, dev_status, st) \
             : launch_row_reduce<T, uint8_t>(feats, nin, nbr, num_out, num_offsets, channels, op, out, arg, count, dev_status, st)
  switch (dtype) {
    case WCN_F32: WCN_REDUCE_CASE(float);
    case WCN_F16: WCN_REDUCE_CASE(__half);
    case WCN_BF16: WCN_REDUCE_CASE(__nv_bfloat16);
    default: return WCN_ERR_INVALID_PARAMETERS;
  }
#undef WCN_REDUCE_CASE
}

extern "C" int wcn_row_reduce(const void* feats, int64_t num_in, const int32_t* nbr, int64_t num_out,
                              int32_t num_offsets, int32_t channels, int dtype, int op, void* out,
                              int32_t* dev_status, void* stream) {
  return wcn_row_reduce_train(feats, num_in, nbr, num_out, num_offsets, channels, dtype, op, out, nullptr, 0, nullptr,
                              dev_status, stream);
}

extern "C" int wcn_row_reduce_backward(const void* grad_out, int64_t num_out, const int32_t* nbr_t, int64_t num_in,
                                       int32_t num_offsets, int32_t channels, int dtype, const void* arg,
                                       int32_t arg_bytes, const float* count, void* grad_in, int32_t* dev_status,
                                       void* stream) {
  if (num_out < 0 || num_in < 0 || num_offsets <= 0 || channels <= 0) return WCN_ERR_INVALID_PARAMETERS;
  if (num_in == 0) return WCN_OK;
  if (!nbr_t || !grad_in || (num_out > 0 && !grad_out)) return WCN_ERR_INVALID_PARAMETERS;
  if (arg && arg_bytes != 1 && arg_bytes != 2) return WCN_ERR_INVALID_PARAMETERS;
  if ((int64_t)num_in * channels >= (int64_t)0x7FFFFFFF * 256) return WCN_ERR_INVALID_PARAMETERS;
  const int nout = (int)(num_out < 0x7FFFFFFFll ? num_out : 0x7FFFFFFFll);
  cudaStream_t st = wcn_stream(stream);
#define WCN_REDUCE_CASE(T)                                                                                            \
  return arg_bytes == 2                                                                                               \
             ? launch_row_reduce_backward<T, uint16_t>(grad_out, nout, nbr_t, num_in, num_offsets, channels, arg, count, grad_in, dev_status, st) \
             : launch_row_reduce_backward<T, uint8_t>(grad_out, nout, nbr_t, num_in, num_offsets, channels, arg, count, grad_in, dev_status, st)
  switch (dtype) {
    case WCN_F32: WCN_REDUCE_CASE(float);
    case WCN_F16: WCN_REDUCE_CASE(__half);
    case WCN_BF16: WCN_REDUCE_CASE(__nv_bfloat16);
    default: return WCN_ERR_INVALID_PARAMETERS;
  }
#undef WCN_REDUCE_CASE
}
