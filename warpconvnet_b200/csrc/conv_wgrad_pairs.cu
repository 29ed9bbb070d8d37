// Weight gradient of the sparse convolution on the FP32 pipes, for fp32 tensors that conv_wgrad_split_tcgen05.cu does not take
// (few offsets, narrow layers) and for widths the tensor-core kernels do not take (a 3-channel stem, odd widths):
//     dW[k][ci][co] = sum over rows m with a neighbour at offset k of X[nbr[k][m]][ci] * dY[m][co].
//
// Bound by FMA issue.  A block owns one offset, a TI x TJ tile of its matrix and a range of rows.  It lists the rows
// of the range that have a neighbour (ballots), stages P listed (X row, dY row) pieces at a time in shared memory
// (the next P in registers meanwhile) and accumulates the outer products in registers: a thread owns RI x 4
// elements, and where a tile has fewer threads than the block the remaining ones take other pairs of the stage and
// are added in at the end.  The ranges leave partial sums in a workspace and a second kernel adds them in order: no
// atomics, the same bits on every run.
// Before, these layers ran a row gather and a cuBLAS GEMM per offset over compacted pair lists: 60 000 room voxels,
// C = 64 fp32, 27 offsets: 2.0 ms (the GEMMs 1.7 ms: 64 x 64 outputs, a reduction 20 000 long, on a few SMs).
#include "wcn_common.cuh"

namespace {

constexpr int THREADS = 128;
constexpr int P = 32;            // pairs per stage
constexpr int LIST = 1024;       // rows listed at a time

struct PairsParams {
  const void* feats;
  const void* gout;
  const int32_t* nbr;
  const int32_t* out_rows;
  float* dst;                    // [ranges][K][c_in][c_out]
  int64_t M, rows_per_range;
  int K, c_in, c_out, num_in, tiles_j;
  int32_t* dev_status;
};

// Four consecutive elements of a row as fp32, zero beyond `limit`; VEC: the four are one aligned request.
template <typename T, bool VEC>
__device__ __forceinline__ float4 load4(const T* row, int c, int limit) {
  float4 v = make_float4(0, 0, 0, 0);
  if constexpr (VEC) {
    if (c >= limit) return v;
    if constexpr (sizeof(T) == 4) {
      v = __ldg(reinterpret_cast<const float4*>(row + c));
    } else {
      const uint2 q = __ldg(reinterpret_cast<const uint2*>(row + c));
      const T* t = reinterpret_cast<const T*>(&q);
      v = make_float4(wcn_to_float<T>(t[0]), wcn_to_float<T>(t[1]), wcn_to_float<T>(t[2]), wcn_to_float<T>(t[3]));
    }
  } else {
    if (c < limit) v.x = wcn_to_float<T>(row[c]);
    if (c + 1 < limit) v.y = wcn_to_float<T>(row[c + 1]);
    if (c + 2 < limit) v.z = wcn_to_float<T>(row[c + 2]);
    if (c + 3 < limit) v.w = wcn_to_float<T>(row[c + 3]);
  }
  return v;
}

template <typename T, int TI, int TJ, bool VEC>
__global__ void __launch_bounds__(THREADS)
conv_wgrad_pairs_kernel(const PairsParams p) {
  constexpr int RI = 8;
  constexpr int TY = TI / RI, TX = TJ / 4, G = THREADS / (TX * TY);
  constexpr int XQ = P * TI / 4, YQ = P * TJ / 4;              // four-element pieces of a stage
  constexpr int XN = (XQ + THREADS - 1) / THREADS, YN = (YQ + THREADS - 1) / THREADS;
  __shared__ __align__(16) float x_s[2][P][TI];
  __shared__ __align__(16) float y_s[2][P][TJ];
  __shared__ int32_t src_s[LIST], row_s[LIST];
  __shared__ int warp_n[THREADS / 32];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tx = tid % TX, ty = (tid / TX) % TY, g = tid / (TX * TY);
  const int k = blockIdx.y, i0 = (blockIdx.z / p.tiles_j) * TI, j0 = (blockIdx.z % p.tiles_j) * TJ;
  const T* feats = reinterpret_cast<const T*>(p.feats) + i0;
  const T* gout = reinterpret_cast<const T*>(p.gout) + j0;
  const int ci = p.c_in - i0, co = p.c_out - j0;                // columns that exist in this tile
  const int64_t begin = (int64_t)blockIdx.x * p.rows_per_range;
  const int64_t end = min(p.M, begin + p.rows_per_range);
  float acc[RI][4];
#pragma unroll
  for (int r = 0; r < RI; ++r) acc[r][0] = acc[r][1] = acc[r][2] = acc[r][3] = 0.f;
  bool bad = false;

  for (int64_t base = begin; base < end; base += LIST) {
    // ---- list this block of rows: each warp LIST / 4 consecutive ones, in order
    constexpr int PER_WARP = LIST / (THREADS / 32);
    int32_t src[PER_WARP / 32];
    int mine = 0;
#pragma unroll
    for (int b = 0; b < PER_WARP / 32; ++b) {
      const int64_t m = base + warp * PER_WARP + b * 32 + lane;
      src[b] = m < end ? __ldg(&p.nbr[(int64_t)k * p.M + m]) : -1;
      if (src[b] >= p.num_in) { src[b] = -1; bad = true; }
    }
#pragma unroll
    for (int b = 0; b < PER_WARP / 32; ++b) mine += __popc(__ballot_sync(0xFFFFFFFFu, src[b] >= 0));
    __syncthreads();  // the previous list has been read
    if (lane == 0) warp_n[warp] = mine;
    __syncthreads();
    int at = 0, n = 0;
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w) { if (w < warp) at += warp_n[w]; n += warp_n[w]; }
#pragma unroll
    for (int b = 0; b < PER_WARP / 32; ++b) {
      const uint32_t have = __ballot_sync(0xFFFFFFFFu, src[b] >= 0);
      if (src[b] >= 0) {
        const int to = at + __popc(have & ((1u << lane) - 1u));
        const int64_t m = base + warp * PER_WARP + b * 32 + lane;
        src_s[to] = src[b];
        row_s[to] = p.out_rows ? __ldg(&p.out_rows[m]) : (int32_t)m;
      }
      at += __popc(have);
    }
    __syncthreads();
    if (n == 0) continue;

    // ---- stages of P pairs
    float4 xr[XN], yr[YN];
    auto fetch = [&](int p0) {
#pragma unroll
      for (int u = 0; u < XN; ++u) {
        const int q = tid + u * THREADS, pair = p0 + q / (TI / 4), c = (q % (TI / 4)) * 4;
        xr[u] = (q < XQ && pair < n) ? load4<T, VEC>(feats + (int64_t)src_s[pair] * p.c_in, c, ci) : make_float4(0, 0, 0, 0);
      }
#pragma unroll
      for (int u = 0; u < YN; ++u) {
        const int q = tid + u * THREADS, pair = p0 + q / (TJ / 4), c = (q % (TJ / 4)) * 4;
        yr[u] = (q < YQ && pair < n) ? load4<T, VEC>(gout + (int64_t)row_s[pair] * p.c_out, c, co) : make_float4(0, 0, 0, 0);
      }
    };
    fetch(0);
    int buf = 0;
    for (int p0 = 0; p0 < n; p0 += P) {
#pragma unroll
      for (int u = 0; u < XN; ++u) {
        const int q = tid + u * THREADS;
        if (q < XQ) *reinterpret_cast<float4*>(&x_s[buf][q / (TI / 4)][(q % (TI / 4)) * 4]) = xr[u];
      }
#pragma unroll
      for (int u = 0; u < YN; ++u) {
        const int q = tid + u * THREADS;
        if (q < YQ) *reinterpret_cast<float4*>(&y_s[buf][q / (TJ / 4)][(q % (TJ / 4)) * 4]) = yr[u];
      }
      __syncthreads();  // (two buffers: the one written next was last read before this barrier)
      if (p0 + P < n) fetch(p0 + P);
#pragma unroll 4
      for (int q = g; q < P; q += G) {
        float x[RI];
        *reinterpret_cast<float4*>(x) = *reinterpret_cast<const float4*>(&x_s[buf][q][ty * 4]);
        *reinterpret_cast<float4*>(x + 4) = *reinterpret_cast<const float4*>(&x_s[buf][q][TI / 2 + ty * 4]);
        const float4 y = *reinterpret_cast<const float4*>(&y_s[buf][q][tx * 4]);
#pragma unroll
        for (int r = 0; r < RI; ++r) {
          acc[r][0] = fmaf(x[r], y.x, acc[r][0]);
          acc[r][1] = fmaf(x[r], y.y, acc[r][1]);
          acc[r][2] = fmaf(x[r], y.z, acc[r][2]);
          acc[r][3] = fmaf(x[r], y.w, acc[r][3]);
        }
      }
      buf ^= 1;
    }
  }

  // ---- add the pair groups in order, then leave the tile
  static_assert(TJ <= 2 * P, "a tile fits the X stages");
  float* sum_s = &x_s[0][0][0];
  auto row_of = [&](int r) { return r < 4 ? ty * 4 + r : TI / 2 + ty * 4 + r - 4; };
  if constexpr (G > 1) {
    for (int from = 1; from < G; ++from) {  // one group at a time through one tile of shared memory
      __syncthreads();
      if (g == from) {
#pragma unroll
        for (int r = 0; r < RI; ++r)
          *reinterpret_cast<float4*>(sum_s + row_of(r) * TJ + tx * 4) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
      }
      __syncthreads();
      if (g == 0) {
#pragma unroll
        for (int r = 0; r < RI; ++r) {
          const float4 v = *reinterpret_cast<const float4*>(sum_s + row_of(r) * TJ + tx * 4);
          acc[r][0] += v.x; acc[r][1] += v.y; acc[r][2] += v.z; acc[r][3] += v.w;
        }
      }
    }
  }
  if (g == 0) {
    float* dst = p.dst + (((int64_t)blockIdx.x * p.K + k) * p.c_in + i0) * p.c_out + j0;
#pragma unroll
    for (int r = 0; r < RI; ++r) {
      const int i = row_of(r);
      if (i >= ci) continue;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (tx * 4 + j < co) dst[(int64_t)i * p.c_out + tx * 4 + j] = acc[r][j];
    }
  }
  if (bad) wcn_report_bounds(p.dev_status);
}

// Up to CI = 8 input channels (a network's stem).  What counts is how often dY is read and how many instructions a (row,
// offset) takes: a warp holds the dY rows of 32 table rows (lane = output channel) in registers, stages the input rows of
// KG offsets in shared memory and multiplies them from there, one broadcast load and CI multiply-adds per row and offset.
// (240 000 rows, 3 -> 32 channels, 27 offsets: 222 us walking the present pairs of one offset at a time, which reads a dY
// row per pair; 114 us here.)
constexpr int NARROW_THREADS = 256;
__host__ __device__ constexpr int narrow_offsets(int ci) { return 36 / ci; }   // 9 offsets of 4 channels, 4 of 8: 36 and 32 sums a thread

// One element of dW over the rows begin .. end - 1, present pairs only.
template <typename T>
__device__ __noinline__ float present_sum(const PairsParams& p, int k, int c, int n, int64_t begin, int64_t end) {
  float v = 0.f;
  for (int64_t m = begin; m < end; ++m) {
    const int r = __ldg(&p.nbr[(int64_t)k * p.M + m]);
    if (r < 0 || r >= p.num_in) continue;
    const int64_t row = p.out_rows ? (int64_t)__ldg(&p.out_rows[m]) : m;
    v = fmaf(wcn_to_float<T>(reinterpret_cast<const T*>(p.feats)[(int64_t)r * p.c_in + c]),
             wcn_to_float<T>(reinterpret_cast<const T*>(p.gout)[row * p.c_out + n]), v);
  }
  return v;
}

template <typename T, int CI>
__global__ void __launch_bounds__(NARROW_THREADS, 2)
conv_wgrad_narrow_kernel(const PairsParams p) {
  constexpr int KG = narrow_offsets(CI), WARPS = NARROW_THREADS / 32;
  __shared__ __align__(16) float xs[WARPS][KG][32][CI];
  __shared__ int again;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int k0 = blockIdx.y * KG, j = blockIdx.z * 32 + lane;
  const bool col = j < p.c_out;
  const T* feats = reinterpret_cast<const T*>(p.feats);
  const T* gout = reinterpret_cast<const T*>(p.gout) + (col ? j : 0);
  const int64_t begin = (int64_t)blockIdx.x * p.rows_per_range, end = min(p.M, begin + p.rows_per_range);
  float acc[KG][CI];
#pragma unroll
  for (int q = 0; q < KG; ++q)
#pragma unroll
    for (int c = 0; c < CI; ++c) acc[q][c] = 0.f;
  bool bad = false;
  for (int64_t base = begin + warp * 32; base < end; base += NARROW_THREADS) {
    const int64_t m = base + lane;
    int src[KG];
#pragma unroll
    for (int q = 0; q < KG; ++q) src[q] = (k0 + q < p.K && m < end) ? __ldg(&p.nbr[(int64_t)(k0 + q) * p.M + m]) : -1;
    const int row = m < end ? (p.out_rows ? __ldg(&p.out_rows[m]) : (int)m) : -1;
    uint32_t any = 0;
#pragma unroll
    for (int q = 0; q < KG; ++q) {
      if (src[q] >= p.num_in) { src[q] = -1; bad = true; }
      any |= __any_sync(0xFFFFFFFFu, src[q] >= 0) ? 1u << q : 0u;
      float x[CI];
#pragma unroll
      for (int c = 0; c < CI; ++c) x[c] = src[q] >= 0 && c < p.c_in ? wcn_to_float<T>(feats[(int64_t)src[q] * p.c_in + c]) : 0.f;
#pragma unroll
      for (int c = 0; c < CI; c += 4) *reinterpret_cast<float4*>(&xs[warp][q][lane][c]) = make_float4(x[c], x[c + 1], x[c + 2], x[c + 3]);
    }
    if (!any) continue;
    float g[32];
#pragma unroll
    for (int b = 0; b < 32; ++b) {
      const int r = __shfl_sync(0xFFFFFFFFu, row, b);
      g[b] = r >= 0 && col ? wcn_to_float<T>(gout[(int64_t)r * p.c_out]) : 0.f;
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < KG; ++q) {
      if (!((any >> q) & 1u)) continue;
#pragma unroll
      for (int b = 0; b < 32; ++b)
#pragma unroll
        for (int c = 0; c < CI; c += 4) {
          const float4 x = *reinterpret_cast<const float4*>(&xs[warp][q][b][c]);
          acc[q][c] = fmaf(x.x, g[b], acc[q][c]);
          acc[q][c + 1] = fmaf(x.y, g[b], acc[q][c + 1]);
          acc[q][c + 2] = fmaf(x.z, g[b], acc[q][c + 2]);
          acc[q][c + 3] = fmaf(x.w, g[b], acc[q][c + 3]);
        }
    }
    __syncwarp();
  }
  // the block's sums, in warp order
  if (threadIdx.x == 0) again = 0;
  __syncthreads();
  float* part = &xs[0][0][0][0];   // [KG * CI][WARPS][32] would not fit at once: one offset at a time
#pragma unroll
  for (int q = 0; q < KG; ++q) {
#pragma unroll
    for (int c = 0; c < CI; ++c) part[(c * WARPS + warp) * 32 + lane] = acc[q][c];
    __syncthreads();
    for (int i = threadIdx.x; i < CI * 32; i += NARROW_THREADS) {
      const int c = i / 32, n = blockIdx.z * 32 + (i & 31);
      float v = 0.f;
#pragma unroll
      for (int w = 0; w < WARPS; ++w) v += part[(c * WARPS + w) * 32 + (i & 31)];
      if (k0 + q < p.K && c < p.c_in && n < p.c_out) p.dst[(((int64_t)blockIdx.x * p.K + k0 + q) * p.c_in + c) * p.c_out + n] = v;
      if (!isfinite(v)) again = 1;
    }
    __syncthreads();
  }
  // Absent neighbours were multiplied as zeros: an infinity or NaN in dY made sums out of pairs that do not exist.  The sums
  // that are not finite are taken once more, by themselves (kept in registers for a second pass of the warps they cost the
  // finite case its registers: 3 channels bf16, 240 000 rows, 107 -> 120 us).
  if (again)
    for (int q = 0; q < KG; ++q)
      for (int i = threadIdx.x; i < CI * 32; i += NARROW_THREADS) {
        const int c = i / 32, n = blockIdx.z * 32 + (i & 31);
        if (k0 + q >= p.K || c >= p.c_in || n >= p.c_out) continue;
        float* dst = &p.dst[(((int64_t)blockIdx.x * p.K + k0 + q) * p.c_in + c) * p.c_out + n];
        if (!isfinite(*dst)) *dst = present_sum<T>(p, k0 + q, c, n, begin, end);
      }
  if (bad) wcn_report_bounds(p.dev_status);
}

__global__ void sum_ranges_kernel(const float* __restrict__ partial, int ranges, int64_t n, float* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float s = 0.f;
#pragma unroll 8
  for (int r = 0; r < ranges; ++r) s += __ldcg(&partial[r * n + i]);
  out[i] = s;
}

struct PairsPlan {
  int ti, tj, tiles_i, tiles_j, ranges, blocks_k;
  int64_t rows_per_range;
};

// About eight blocks per multiprocessor (two of the narrow kernel), none with fewer than one list of rows.
PairsPlan plan_pairs(int64_t M, int K, int c_in, int c_out) {
  PairsPlan q;
  q.ti = c_in <= 8 ? 8 : c_in <= 32 ? 32 : 64;   // 8: the narrow kernel, 32 columns a block
  q.tj = c_out <= 32 || q.ti == 8 ? 32 : 64;
  q.tiles_i = (c_in + q.ti - 1) / q.ti;
  q.tiles_j = (c_out + q.tj - 1) / q.tj;
  const int ks = narrow_offsets(c_in <= 4 ? 4 : 8);
  q.blocks_k = q.ti == 8 ? (K + ks - 1) / ks : K;
  const int64_t blocks = (int64_t)q.blocks_k * q.tiles_i * q.tiles_j;
  // (the narrow kernel's blocks are resident two at a time)
  int64_t ranges = ((q.ti == 8 ? 2 : 8) * (int64_t)wcn_num_sms() + blocks - 1) / blocks;
  const int64_t most = (M + LIST - 1) / LIST;
  if (ranges > most) ranges = most;
  if (ranges < 1) ranges = 1;
  q.rows_per_range = (M + ranges - 1) / ranges;
  q.ranges = (int)((M + q.rows_per_range - 1) / q.rows_per_range);
  return q;
}

template <typename T, bool VEC>
int launch_pairs(const PairsParams& p, const PairsPlan& q, cudaStream_t st) {
  dim3 grid((unsigned)q.ranges, (unsigned)q.blocks_k, (unsigned)(q.tiles_i * q.tiles_j));
  if (q.ti == 8) {
    if (p.c_in <= 4) conv_wgrad_narrow_kernel<T, 4><<<grid, NARROW_THREADS, 0, st>>>(p);
    else conv_wgrad_narrow_kernel<T, 8><<<grid, NARROW_THREADS, 0, st>>>(p);
    return cudaGetLastError() == cudaSuccess ? WCN_OK : WCN_ERR_EXECUTION;
  }
#define WCN_PAIRS_CASE(TI, TJ)                                                                       \
  if (q.ti == TI && q.tj == TJ) {                                                                    \
    conv_wgrad_pairs_kernel<T, TI, TJ, VEC><<<grid, THREADS, 0, st>>>(p);                            \
    return cudaGetLastError() == cudaSuccess ? WCN_OK : WCN_ERR_EXECUTION;                           \
  }
  WCN_PAIRS_CASE(32, 32) WCN_PAIRS_CASE(32, 64) WCN_PAIRS_CASE(64, 32) WCN_PAIRS_CASE(64, 64)
#undef WCN_PAIRS_CASE
  return WCN_ERR_UNSUPPORTED_CONFIG;
}

}  // namespace

extern "C" int wcn_conv_wgrad_pairs_workspace_bytes(int64_t num_out, int32_t num_offsets, int32_t c_in, int32_t c_out,
                                                    int64_t* bytes) {
  if (!bytes || num_out < 0 || num_offsets <= 0 || num_offsets > 65535 || c_in <= 0 || c_out <= 0) return WCN_ERR_INVALID_PARAMETERS;
  const PairsPlan q = plan_pairs(num_out, num_offsets, c_in, c_out);
  *bytes = q.ranges > 1 ? (int64_t)q.ranges * num_offsets * c_in * c_out * (int64_t)sizeof(float) : 0;
  return WCN_OK;
}

extern "C" int wcn_conv_wgrad_pairs(const void* feats, int64_t num_in, const void* grad_out, const int32_t* nbr,
                                    const int32_t* out_rows, int64_t num_out, int32_t num_offsets, int32_t c_in,
                                    int32_t c_out, int dtype, float* grad_weight, void* workspace,
                                    int64_t workspace_bytes, int32_t* dev_status, void* stream) {
  if (num_in < 0 || num_out < 0 || num_out >= 0x7FFFFFFFll || num_offsets <= 0 || num_offsets > 65535 || c_in <= 0 || c_out <= 0 ||
      dtype < WCN_F32 || dtype > WCN_BF16 || !grad_weight)
    return WCN_ERR_INVALID_PARAMETERS;
  cudaStream_t st = wcn_stream(stream);
  const int64_t n = (int64_t)num_offsets * c_in * c_out;
  if (num_in == 0 || num_out == 0)
    return cudaMemsetAsync(grad_weight, 0, (size_t)n * sizeof(float), st) == cudaSuccess ? WCN_OK : WCN_ERR_EXECUTION;
  if (!feats || !grad_out || !nbr) return WCN_ERR_INVALID_PARAMETERS;
  const PairsPlan q = plan_pairs(num_out, num_offsets, c_in, c_out);
  if ((int64_t)q.tiles_i * q.tiles_j > 65535) return WCN_ERR_UNSUPPORTED_CONFIG;
  if (q.ranges > 1 && (!workspace || workspace_bytes < q.ranges * n * (int64_t)sizeof(float))) return WCN_ERR_INVALID_PARAMETERS;
  PairsParams p;
  p.feats = feats; p.gout = grad_out; p.nbr = nbr; p.out_rows = out_rows;
  p.dst = q.ranges > 1 ? reinterpret_cast<float*>(workspace) : grad_weight;
  p.M = num_out; p.rows_per_range = q.rows_per_range;
  p.K = num_offsets; p.c_in = c_in; p.c_out = c_out; p.tiles_j = q.tiles_j;
  p.num_in = (int)(num_in < 0x7FFFFFFFll ? num_in : 0x7FFFFFFFll);
  p.dev_status = dev_status;
  const int align = 4 * wcn_dtype_size(dtype);
  const bool vec = c_in % 4 == 0 && c_out % 4 == 0 && reinterpret_cast<uintptr_t>(feats) % align == 0 &&
                   reinterpret_cast<uintptr_t>(grad_out) % align == 0;
  int rc = WCN_ERR_UNSUPPORTED_CONFIG;
  if (dtype == WCN_F32) rc = vec ? launch_pairs<float, true>(p, q, st) : launch_pairs<float, false>(p, q, st);
  else if (dtype == WCN_F16) rc = vec ? launch_pairs<__half, true>(p, q, st) : launch_pairs<__half, false>(p, q, st);
  else rc = vec ? launch_pairs<__nv_bfloat16, true>(p, q, st) : launch_pairs<__nv_bfloat16, false>(p, q, st);
  if (rc != WCN_OK || q.ranges == 1) return rc;
  sum_ranges_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(reinterpret_cast<const float*>(workspace), q.ranges, n, grad_weight);
  WCN_CHECK_LAUNCH();
  return WCN_OK;
}
