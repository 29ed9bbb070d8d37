// Output-stationary sparse convolution of fp32 tensors: gathered rows times weights on the FP32 pipes, with the
// absent neighbours left out.  For widths that conv_split_tcgen05.cu does not take, more than 27 offsets, calls without
// workspace, and the problems that are done here before that kernel's two launches are (few rows of narrow layers, one offset).
//
// Bound by FMA issue where neighbours are dense and by latency where they are few.  A block owns TM output rows x TN
// columns.  Per kernel offset the rows of the tile that have a neighbour are listed (ballots over the table column),
// only their input rows are copied (cp.async, 16 bytes a request, two (offset, channel slice) steps ahead of the
// arithmetic) and only they are multiplied: a thread owns four columns of R = ceil(listed / row threads) listed rows,
// R a compile-time constant picked per offset, so an offset with 5 of 64 rows costs an eighth of a full one.  The
// accumulators live in shared memory between offsets (a listed row may be any row of the tile) and in registers
// within one: a load and a store per C_in multiply-adds.  Per output the sum runs over the offsets (of a group, see
// F32Tile) and input channels in ascending order with fused multiply-adds: the same bits on every run and in every
// row order.
//
// Measured (B200): 20 000 random cells, C = 32, 2.9 of 27 neighbours: 30 us, 105 us in conv_simt_kernel (64 x 64
// tiles, every absent row multiplied, two barriers per 16 channels); 60 000 room voxels, C = 64, 9.9 of 27: 193 us
// (25 TFLOP/s, 64 % of the issue slots), before 343 us.
#include "wcn_common.cuh"

namespace {

constexpr int MAX_KB = 32;        // offsets listed at a time

struct F32Params {
  const float* feats;
  const float* weight;
  const int32_t* nbr;
  const int32_t* out_rows;
  int64_t M, in_ld, out_ld, res_ld;
  int K, c_in, c_out, num_in;
  int tiles_per_window;  // row tiles per window of the tile order (0: rows in their own order)
  const float* scale;
  const float* shift;
  const float* residual;
  int relu;
  float* out;
  int32_t* dev_status;
};

__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool have) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(have ? 16u : 0u));
}

// R listed rows x 4 columns over one staged channel slice.
template <int R, class T>
__device__ __forceinline__ void multiply(const float* __restrict__ a, const float* __restrict__ w, float (&acc)[8][4]) {
#pragma unroll
  for (int c = 0; c < T::CK; c += 4) {
    float4 x[R];
#pragma unroll
    for (int r = 0; r < R; ++r) x[r] = *reinterpret_cast<const float4*>(a + r * T::TY * T::A_LD + c);
#pragma unroll
    for (int cc = 0; cc < 4; ++cc) {
      const float4 b = *reinterpret_cast<const float4*>(w + (c + cc) * T::TN);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float v = cc == 0 ? x[r].x : cc == 1 ? x[r].y : cc == 2 ? x[r].z : x[r].w;
        acc[r][0] = fmaf(v, b.x, acc[r][0]);
        acc[r][1] = fmaf(v, b.y, acc[r][1]);
        acc[r][2] = fmaf(v, b.z, acc[r][2]);
        acc[r][3] = fmaf(v, b.w, acc[r][3]);
      }
    }
  }
}

// G: groups of threads that take every G-th offset, each with accumulators of its own (added in group order at the end).
template <int TM_, int TN_, int G_>
struct F32Tile {
  static constexpr int TM = TM_, TN = TN_, G = G_;
  static constexpr int STAGES = G > 1 ? 2 : 3;
  static constexpr int CK = TN == 32 ? 32 : 16;           // input channels per step
  static constexpr int A_LD = CK + 4;                     // floats between staged rows: a warp's row threads read different banks
  static constexpr int TX = TN / 4, TY = 8;               // column threads, row threads
  static constexpr int GROUP = TX * TY, THREADS = G * GROUP;
  static constexpr int RMAX = (TM + TY - 1) / TY;         // listed rows per thread at most
  static constexpr int A_FLOATS = TM * A_LD, W_FLOATS = CK * TN;
  static constexpr size_t SMEM = sizeof(float) * G * (STAGES * (A_FLOATS + W_FLOATS) + TM * TN) + sizeof(int32_t) * MAX_KB * TM +
                                 sizeof(int32_t) * MAX_KB + MAX_KB * TM;
};

// Row tile of block b.  In a table in tile order the rows of a window of `per` tiles are sorted by their neighbour
// pattern, the fullest last: the last tiles of all windows start first and the lightest ones fill the end.
__device__ __forceinline__ int64_t tile_of_block(int b, int tiles, int per) {
  if (per <= 0 || tiles <= per) return tiles - 1 - b;
  const int windows = (tiles + per - 1) / per, last = tiles - (windows - 1) * per;
  const int head = (per - last) * (windows - 1);  // tiles at places the last window does not have
  if (b < head) return (int64_t)(b % (windows - 1)) * per + per - 1 - b / (windows - 1);
  b -= head;
  return (int64_t)(b % windows) * per + last - 1 - b / windows;
}

template <int TM, int TN, int G>
__global__ void __launch_bounds__(F32Tile<TM, TN, G>::THREADS)
conv_fp32_kernel(const F32Params p) {
  using T = F32Tile<TM, TN, G>;
  constexpr int STAGES = T::STAGES;
  extern __shared__ __align__(16) uint8_t smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = tid / T::GROUP, gtid = tid % T::GROUP;
  const int tx = gtid % T::TX, ty = gtid / T::TX;
  float* acc_all = reinterpret_cast<float*>(smem_raw);             // [G][TM][TN]
  float* acc_s = acc_all + g * TM * TN;
  float* a_s = acc_all + G * TM * TN + g * STAGES * T::A_FLOATS;   // [G][STAGES][TM][A_LD]
  float* w_s = acc_all + G * (TM * TN + STAGES * T::A_FLOATS) + g * STAGES * T::W_FLOATS;  // [G][STAGES][CK][TN]
  int32_t* src_s = reinterpret_cast<int32_t*>(acc_all + G * (TM * TN + STAGES * (T::A_FLOATS + T::W_FLOATS)));  // [MAX_KB][TM] input rows of the listed rows
  int32_t* count_s = src_s + MAX_KB * TM;                          // [MAX_KB]
  uint8_t* row_s = reinterpret_cast<uint8_t*>(count_s + MAX_KB);   // [MAX_KB][TM] tile rows of the listed rows

  const int64_t m0 = tile_of_block((int)blockIdx.x, (int)gridDim.x, p.tiles_per_window) * TM;
  const int n0 = blockIdx.y * TN;
  constexpr int CK = T::CK, A_LD = T::A_LD;
  const int slices = (p.c_in + CK - 1) / CK;
  bool bad = false;
  for (int i = tid; i < G * TM * TN / 4; i += T::THREADS) reinterpret_cast<float4*>(acc_all)[i] = make_float4(0, 0, 0, 0);
  auto group_barrier = [&]() {
    if constexpr (G == 1) __syncthreads();
    else asm volatile("bar.sync %0, %1;" ::"r"(1 + g), "n"(T::GROUP) : "memory");
  };

  for (int kb = 0; kb < p.K; kb += MAX_KB) {
    const int nk = min(MAX_KB, p.K - kb);
    // ---- list the rows that have a neighbour, offset by offset (a warp per offset)
    __syncthreads();
    for (int k = warp; k < nk; k += T::THREADS / 32) {
      int n = 0;
      for (int r0 = 0; r0 < TM; r0 += 32) {
        const int r = r0 + lane;
        int src = (r < TM && m0 + r < p.M) ? __ldg(&p.nbr[(int64_t)(kb + k) * p.M + m0 + r]) : -1;
        if (src >= p.num_in) { src = -1; bad = true; }  // not a feature row: absent, reported once below
        const uint32_t have = __ballot_sync(0xFFFFFFFFu, src >= 0);
        if (src >= 0) {
          const int at = n + __popc(have & ((1u << lane) - 1u));
          src_s[k * TM + at] = src;
          row_s[k * TM + at] = (uint8_t)r;
        }
        n += __popc(have);
      }
      if (lane == 0) count_s[k] = n;
    }
    __syncthreads();

    // ---- steps (offset, channel slice); copies run STAGES - 1 steps ahead, one barrier per step
    int k_next = g, s_next = 0, to = 0;
    while (k_next < nk && count_s[k_next] == 0) k_next += G;
    auto copy_step = [&]() {  // enqueue the copies of step (k_next, s_next) as one group, then move on to the next one
      if (k_next < nk) {
        const int c0 = s_next * CK, n = count_s[k_next];
        const float* wk = p.weight + ((int64_t)(kb + k_next) * p.c_in + c0) * p.c_out + n0;
        const uint32_t a_dst = (uint32_t)__cvta_generic_to_shared(a_s + to * T::A_FLOATS);
        const uint32_t w_dst = (uint32_t)__cvta_generic_to_shared(w_s + to * T::W_FLOATS);
        for (int i = gtid; i < n * (CK / 4); i += T::GROUP) {
          const int r = i / (CK / 4), c = (i % (CK / 4)) * 4;
          const bool have = c0 + c < p.c_in;
          cp16(a_dst + (uint32_t)(r * A_LD + c) * 4,
               have ? p.feats + (int64_t)src_s[k_next * TM + r] * p.in_ld + c0 + c : p.feats, have);
        }
#pragma unroll
        for (int i = gtid; i < CK * TN / 4; i += T::GROUP) {
          const int c = i / (TN / 4), n4 = (i % (TN / 4)) * 4;
          const bool have = c0 + c < p.c_in && n0 + n4 < p.c_out;
          cp16(w_dst + (uint32_t)(c * TN + n4) * 4, have ? wk + (int64_t)c * p.c_out + n4 : p.weight, have);
        }
        if (++s_next == slices) {
          s_next = 0;
          do { k_next += G; } while (k_next < nk && count_s[k_next] == 0);
        }
        if (++to == STAGES) to = 0;
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    int k = k_next, s = 0, at_stage = 0;
#pragma unroll
    for (int i = 0; i < STAGES - 1; ++i) copy_step();
    float acc[8][4];
    while (k < nk) {
      asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
      group_barrier();  // this step's tiles are there for everyone, and the previous step's have been read
      copy_step();
      const int n = count_s[k], rows = (n + T::TY - 1) / T::TY;
      const uint8_t* list = row_s + k * TM;
      if (s == 0) {
#pragma unroll
        for (int r = 0; r < T::RMAX; ++r) {
          const int at = ty + r * T::TY;
          if (r < rows && at < n) {
            const float4 v = *reinterpret_cast<const float4*>(acc_s + list[at] * TN + tx * 4);
            acc[r][0] = v.x; acc[r][1] = v.y; acc[r][2] = v.z; acc[r][3] = v.w;
          }
        }
      }
      const float* a = a_s + at_stage * T::A_FLOATS + ty * A_LD;
      const float* w = w_s + at_stage * T::W_FLOATS + tx * 4;
      switch (rows) {  // (uniform in the block; rows beyond the listed ones multiply stale values that are not stored)
        case 1: multiply<1, T>(a, w, acc); break;
        case 2: if constexpr (T::RMAX >= 2) multiply<2, T>(a, w, acc); break;
        case 3: if constexpr (T::RMAX >= 3) multiply<3, T>(a, w, acc); break;
        case 4: if constexpr (T::RMAX >= 4) multiply<4, T>(a, w, acc); break;
        case 5: if constexpr (T::RMAX >= 5) multiply<5, T>(a, w, acc); break;
        case 6: if constexpr (T::RMAX >= 6) multiply<6, T>(a, w, acc); break;
        case 7: if constexpr (T::RMAX >= 7) multiply<7, T>(a, w, acc); break;
        default: if constexpr (T::RMAX >= 8) multiply<8, T>(a, w, acc); break;
      }
      if (++at_stage == STAGES) at_stage = 0;
      if (++s == slices) {
#pragma unroll
        for (int r = 0; r < T::RMAX; ++r) {
          const int at = ty + r * T::TY;
          if (at < n) {  // (the barrier of the next step stands between these and another thread's loads)
            *reinterpret_cast<float4*>(acc_s + list[at] * TN + tx * 4) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
          }
        }
        s = 0;
        do { k += G; } while (k < nk && count_s[k] == 0);
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
  }
  __syncthreads();

  // ---- epilogue: four columns of a row per thread, rows in full lines
  for (int i = tid; i < TM * TN / 4; i += T::THREADS) {
    const int r = i / (TN / 4), n = n0 + (i % (TN / 4)) * 4;
    const int64_t slot = m0 + r;
    if (slot >= p.M || n >= p.c_out) continue;
    const int64_t m = p.out_rows ? (int64_t)__ldg(&p.out_rows[slot]) : slot;
    float4 v = *reinterpret_cast<const float4*>(acc_all + i * 4);
#pragma unroll
    for (int q = 1; q < G; ++q) {
      const float4 u = *reinterpret_cast<const float4*>(acc_all + q * TM * TN + i * 4);
      v.x = __fadd_rn(v.x, u.x); v.y = __fadd_rn(v.y, u.y); v.z = __fadd_rn(v.z, u.z); v.w = __fadd_rn(v.w, u.w);
    }
    float y[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) y[j] = wcn_affine(y[j], p.scale, p.shift, n + j);
    if (p.residual) {
      const float4 q = __ldg(reinterpret_cast<const float4*>(p.residual + m * p.res_ld + n));
      y[0] = __fadd_rn(y[0], q.x); y[1] = __fadd_rn(y[1], q.y); y[2] = __fadd_rn(y[2], q.z); y[3] = __fadd_rn(y[3], q.w);
    }
    if (p.relu) {
#pragma unroll
      for (int j = 0; j < 4; ++j) y[j] = fmaxf(y[j], 0.f);
    }
    *reinterpret_cast<float4*>(p.out + m * p.out_ld + n) = make_float4(y[0], y[1], y[2], y[3]);
  }
  if (bad) wcn_report_bounds(p.dev_status);
}

template <int TM, int TN, int G>
int launch_f32(const F32Params& p, cudaStream_t st) {
  using T = F32Tile<TM, TN, G>;
  static bool configured[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return WCN_ERR_INITIALIZATION;
  if (!configured[dev]) {
    if (cudaFuncSetAttribute(conv_fp32_kernel<TM, TN, G>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T::SMEM) != cudaSuccess) {
      (void)cudaGetLastError();
      return WCN_ERR_INITIALIZATION;
    }
    configured[dev] = true;
  }
  dim3 grid((unsigned)((p.M + TM - 1) / TM), (unsigned)((p.c_out + TN - 1) / TN));
  conv_fp32_kernel<TM, TN, G><<<grid, T::THREADS, T::SMEM, st>>>(p);
  return cudaGetLastError() == cudaSuccess ? WCN_OK : WCN_ERR_EXECUTION;
}

}  // namespace

// 16-byte copies and stores: rows of every matrix and of the weights start on 16-byte boundaries.
bool wcn_conv_fp32_supported(int c_in, int c_out, int dtype, int out_dtype, const void* feats, int64_t feats_ld,
                             const void* weight, const void* out, int64_t out_ld, const void* residual, int64_t residual_ld) {
  auto ok = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  return dtype == WCN_F32 && out_dtype == WCN_F32 && c_in % 4 == 0 && c_out % 4 == 0 && ok(feats) && ok(weight) && ok(out) &&
         ok(residual) && feats_ld % 4 == 0 && out_ld % 4 == 0 && (!residual || residual_ld % 4 == 0);
}

int wcn_conv_fp32_fwd(const void* feats, int64_t num_in, int64_t feats_ld, const void* weight, const int32_t* nbr,
                      const int32_t* out_rows, int64_t M, int K, int c_in, int c_out, const float* scale,
                      const float* shift, const void* residual, int64_t residual_ld, int relu, void* out,
                      int64_t out_ld, int sms, int split_k, int32_t* dev_status, cudaStream_t st) {
  F32Params p;
  p.feats = (const float*)feats; p.weight = (const float*)weight; p.nbr = nbr; p.out_rows = out_rows;
  p.M = M; p.in_ld = feats_ld; p.out_ld = out_ld; p.res_ld = residual_ld;
  p.K = K; p.c_in = c_in; p.c_out = c_out; p.num_in = (int)(num_in < 0x7FFFFFFFll ? num_in : 0x7FFFFFFFll);
  p.scale = scale; p.shift = shift; p.residual = (const float*)residual; p.relu = relu; p.out = (float*)out;
  p.dev_status = dev_status;
  // Column tile: the least arithmetic, counting what a column block costs besides its columns (its rows are gathered
  // again for each block) as 16 columns.
  int tn = 32, best = 0;
  for (int t : {32, 64, 96, 128}) {
    const int blocks = (c_out + t - 1) / t, cost = blocks * (t + 16);
    if (!best || cost < best || (cost == best && t > tn)) { best = cost; tn = t; }
  }
  // Row tile: 64 rows while they give every multiprocessor a block, else 16 (more blocks, each re-reading the weights).
  // With fewer than four blocks per multiprocessor a block's own chain of steps is what takes the time, not the
  // arithmetic: its offsets are dealt to groups of threads (20 000 cells, C = 32: 47 -> 30 us), unless the caller wants sums
  // that do not depend on how many rows a launch has (split_k = 1).
  const int blocks_n = (c_out + tn - 1) / tn;
  const bool small = ((M + 63) / 64) * blocks_n < sms;
  const bool grouped = split_k != 1 && K >= 8 && ((M + 63) / 64) * blocks_n < 4 * (int64_t)sms;
  p.tiles_per_window = out_rows ? (M > 4096 ? 16384 : 4096) / (small ? 16 : 64) : 0;
#define WCN_F32_CASE(TN, GN)                                                               \
  if (tn == TN) {                                                                          \
    if (grouped) return small ? launch_f32<16, TN, GN>(p, st) : launch_f32<64, TN, GN>(p, st); \
    return small ? launch_f32<16, TN, 1>(p, st) : launch_f32<64, TN, 1>(p, st);             \
  }
  WCN_F32_CASE(32, 4)
  WCN_F32_CASE(64, 4)
  WCN_F32_CASE(96, 2)
  WCN_F32_CASE(128, 2)
#undef WCN_F32_CASE
  return WCN_ERR_UNSUPPORTED_CONFIG;
}
