// Entry points that do not belong to one kernel family: version, status text and
// the convolution dispatcher.
#include "wcn_common.cuh"

// conv_simt.cu
int wcn_conv_simt_fwd(const void* feats, int64_t num_in, int64_t feats_ld, const void* weight, const int32_t* nbr,
                      const int32_t* out_rows, int64_t M, int K, int c_in, int c_out, int dtype, const float* scale,
                      const float* shift, const void* residual, int64_t residual_ld, int relu, void* out,
                      int64_t out_ld, int out_dtype, int32_t* dev_status, cudaStream_t st);
bool wcn_conv_narrow_supported(int K, int c_in, int c_out, const void* out, int64_t out_ld, const void* residual,
                               int64_t residual_ld, int out_dtype);
int wcn_conv_narrow_fwd(const void* feats, int64_t num_in, int64_t feats_ld, const void* weight, const int32_t* nbr,
                        const int32_t* out_rows, int64_t M, int K, int c_in, int c_out, int dtype,
                        const float* scale, const float* shift, const void* residual, int64_t residual_ld, int relu,
                        void* out, int64_t out_ld, int out_dtype, int32_t* dev_status, cudaStream_t st);
bool wcn_conv_narrow_out_supported(int K, int c_in, int c_out, int dtype, const void* feats, int64_t feats_ld);
int wcn_conv_narrow_out_fwd(const void* feats, int64_t num_in, int64_t feats_ld, const void* weight,
                            const int32_t* nbr, const int32_t* out_rows, int64_t M, int K, int c_in, int c_out,
                            int dtype, const float* scale, const float* shift, const void* residual,
                            int64_t residual_ld, int relu, void* out, int64_t out_ld, int out_dtype,
                            int32_t* dev_status, cudaStream_t st);
// conv_fp32.cu
bool wcn_conv_fp32_supported(int c_in, int c_out, int dtype, int out_dtype, const void* feats, int64_t feats_ld,
                             const void* weight, const void* out, int64_t out_ld, const void* residual, int64_t residual_ld);
int wcn_conv_fp32_fwd(const void* feats, int64_t num_in, int64_t feats_ld, const void* weight, const int32_t* nbr,
                      const int32_t* out_rows, int64_t M, int K, int c_in, int c_out, const float* scale,
                      const float* shift, const void* residual, int64_t residual_ld, int relu, void* out,
                      int64_t out_ld, int sms, int split_k, int32_t* dev_status, cudaStream_t st);
// conv_split_tcgen05.cu
bool wcn_conv_split_supported(int K, int c_in, int c_out);
thread_local int wcn_f32_launches = 0;   // see wcn_conv_f32_launches
int64_t wcn_conv_split_workspace(int64_t num_in, int K, int c_in, int c_out);
int wcn_conv_split_fwd(const void* feats, int64_t num_in, int64_t feats_ld, const void* weight, const int32_t* nbr,
                       const int32_t* out_rows, int64_t M, int K, int c_in, int c_out, const float* scale, const float* shift,
                       const void* residual, int64_t residual_ld, int relu, void* out, int64_t out_ld, int split_k, void* workspace,
                       int32_t* dev_status, cudaStream_t st);
// conv_tcgen05.cu
bool wcn_conv_tcgen05_supported(int K, int c_in, int c_out, int dtype, int out_dtype);
int64_t wcn_conv_tcgen05_packed_bytes(int K, int c_in, int c_out);
int wcn_conv_tcgen05_pack(const void* weight, int src_dtype, int K, int c_in, int c_out, int dtype, int transposed, int reversed,
                          void* packed, cudaStream_t st);
int wcn_conv_tcgen05_fwd(const void* feats, int64_t num_in, int64_t feats_ld, const void* packed, const int32_t* nbr,
                         const int32_t* out_rows, int64_t M, int K, int c_in, int c_out, int dtype,
                         const float* scale, const float* shift, const void* residual, int64_t residual_ld, int relu,
                         void* out, int64_t out_ld, int out_dtype, int split_k, int32_t* dev_status, cudaStream_t st);
// conv_wgrad_tcgen05.cu
bool wcn_conv_wgrad_tcgen05_supported(int K, int c_in, int c_out, int dtype);
int wcn_conv_wgrad_tcgen05(const void* feats, int64_t num_in, const void* grad_out, const int32_t* nbr,
                           const int32_t* out_rows, const uint32_t* tile_masks, int64_t M, int K, int c_in, int c_out, int dtype,
                           float* grad_weight, int32_t* dev_status, cudaStream_t st);

thread_local bool wcn_overlap_launches = false;

extern "C" int wcn_version(void) { return 100; }

extern "C" const char* wcn_status_string(int status) {
  switch (status) {
    case WCN_OK: return "success";
    case WCN_ERR_PROBLEM_NOT_SUPPORTED: return "problem not supported";
    case WCN_ERR_INITIALIZATION: return "kernel initialization failed";
    case WCN_ERR_EXECUTION: return "kernel launch or execution failed";
    case WCN_ERR_UNSUPPORTED_CONFIG: return "unsupported configuration";
    case WCN_ERR_INVALID_PARAMETERS: return "invalid parameters";
    case WCN_ERR_HASH_OVERFLOW: return "hash table overflow";
    case WCN_ERR_WAIT_EXPIRED: return "a bounded device-side wait expired";
    case WCN_ERR_BOUNDS: return "index out of bounds";
    case WCN_ERR_SCRATCH_TOO_SMALL: return "problem larger than the library's built-in scratch array";
    default: return "unknown status";
  }
}

extern "C" int wcn_conv_packed_weight_bytes(int algo, int32_t num_offsets, int32_t c_in, int32_t c_out,
                                            int dtype, int64_t* bytes) {
  if (!bytes || num_offsets <= 0 || c_in <= 0 || c_out <= 0) return WCN_ERR_INVALID_PARAMETERS;
  *bytes = 0;
  if (algo == WCN_CONV_SIMT) return WCN_OK;
  const bool ok = wcn_conv_tcgen05_supported(num_offsets, c_in, c_out, dtype, dtype);
  if (!ok) return algo == WCN_CONV_TCGEN05 ? WCN_ERR_UNSUPPORTED_CONFIG : WCN_OK;
  *bytes = wcn_conv_tcgen05_packed_bytes(num_offsets, c_in, c_out);
  return WCN_OK;
}

extern "C" int wcn_conv_pack_weight(int algo, const void* weight, int32_t num_offsets, int32_t c_in,
                                    int32_t c_out, int dtype, void* packed, void* stream) {
  if (!weight || !packed) return WCN_ERR_INVALID_PARAMETERS;
  if (algo == WCN_CONV_SIMT || !wcn_conv_tcgen05_supported(num_offsets, c_in, c_out, dtype, dtype))
    return WCN_ERR_UNSUPPORTED_CONFIG;
  return wcn_conv_tcgen05_pack(weight, dtype, num_offsets, c_in, c_out, dtype, 0, 0, packed, wcn_stream(stream));
}

extern "C" int wcn_conv_pack_weight_from(const void* weight, int src_dtype, int32_t num_offsets, int32_t c_in, int32_t c_out,
                                         int dtype, int32_t transposed, int32_t reversed, void* packed, void* stream) {
  if (!weight || !packed || (reinterpret_cast<uintptr_t>(packed) & 15)) return WCN_ERR_INVALID_PARAMETERS;
  if (!wcn_conv_tcgen05_supported(num_offsets, c_in, c_out, dtype, dtype)) return WCN_ERR_UNSUPPORTED_CONFIG;
  return wcn_conv_tcgen05_pack(weight, src_dtype, num_offsets, c_in, c_out, dtype, transposed, reversed, packed, wcn_stream(stream));
}

static bool conv_takes_tcgen05(int algo, bool tc_ok, const void* packed_weight, const int32_t* dev_status,
                               int64_t num_in) {
  return algo == WCN_CONV_TCGEN05 || (algo == WCN_CONV_AUTO && tc_ok && packed_weight && dev_status && num_in > 0);
}

extern "C" int wcn_conv_workspace_bytes(int algo, int64_t num_out, int32_t num_offsets, int32_t c_in, int32_t c_out,
                                        int dtype, int out_dtype, int32_t split_k, int64_t* bytes) {
  if (!bytes || num_out < 0 || num_offsets <= 0 || c_in <= 0 || c_out <= 0) return WCN_ERR_INVALID_PARAMETERS;
  *bytes = 0;  // no kernel of this version keeps partial sums in global memory
  (void)algo; (void)dtype; (void)out_dtype; (void)split_k;
  return WCN_OK;
}

extern "C" int wcn_conv_f32_workspace_bytes(int64_t num_in, int64_t num_out, int32_t num_offsets, int32_t c_in, int32_t c_out,
                                            int64_t* bytes) {
  if (!bytes || num_in < 0 || num_out < 0 || num_offsets <= 0 || c_in <= 0 || c_out <= 0) return WCN_ERR_INVALID_PARAMETERS;
  // Few rows of narrow layers stay on the FP32 pipes, which are done before two launches are (us, FP32 pipes / tensor cores;
  // 32 -> 32: 5 000 room voxels 22 / 20, random cells 17 / 20, outdoor 12 / 17, 10 000: 37 / 28, 25 / 28, 23 / 26, 20 000: 55 / 34,
  // 43 / 30, 33 / 28; 64 -> 64, 2 000: 41 / 21, 33 / 22, 23 / 20).
  // A single offset is one pass over the rows, which the planes double (20 000 rows: 64 -> 64 16 / 22, 128 -> 128 43 / 30); a few
  // offsets of narrow layers run one thread per output row without (8 offsets, 32 -> 32: 59 / 18 for 5 000 rows).
  const int64_t area = (int64_t)c_in * c_out;
  const bool row_per_thread = wcn_conv_narrow_out_supported(num_offsets, c_in, c_out, WCN_F32, nullptr, c_in);
  const bool few = num_offsets == 1 ? area < 12288 || num_out < 12000 : area < 2048 && num_out < 12000 && !row_per_thread;
  // The other way round for the narrowest: rows of 16 channels become planes of 32, written and read, while one thread per row
  // or few offsets are little work (8 offsets, 16 -> 16: 100 000 rows 37 / 42, 1 000 000 150 / 271, 16 -> 32 up to 150 000 rows alike,
  // 250 000 108 / 128; 27 offsets, 16 -> 16: 100 000 100 / 56, 300 000 127 / 132, outdoors 140 / 161).
  const bool narrow = area <= 1024 && (c_in < 32 || c_out < 32) && (row_per_thread || num_offsets <= 8) &&
                      num_out >= (num_offsets <= 8 ? 150000 : 250000);
  // Planes are made of all input rows, so that a launch over a small part of the output rows (a boundary, a crop) may be done
  // sooner without them: 2 ns per 1 000 input numbers against what an output row gains (us, 27 offsets, from 1 000 000 rows: 64 -> 64
  // for 15 625 rows 70 / 148, for 62 500 202 / 173, outdoors 44 / 146 and 123 / 161; 128 -> 128 208 / 288, 650 / 343).
  const double planes = 2e-6 * (double)num_in * ((c_in + 31) / 32 * 32);
  const bool part = num_in > 8 * num_out &&
                    planes > (1e-3 + 2.7e-7 * (double)area) * num_offsets / 27 * (double)num_out + 3.7e-3 * (double)area;
  *bytes = num_in > 0 && num_out > 0 && !few && !narrow && !part && wcn_conv_split_supported(num_offsets, c_in, c_out)
               ? wcn_conv_split_workspace(num_in, num_offsets, c_in, c_out) : 0;
  return WCN_OK;
}

extern "C" int wcn_conv_f32_launches(void) { return wcn_f32_launches; }

extern "C" int wcn_conv_fwd(int algo, const void* feats, int64_t num_in, int64_t feats_ld, const void* weight,
                            const void* packed_weight, const int32_t* nbr, const int32_t* out_rows,
                            int64_t num_out, int32_t num_offsets, int32_t c_in, int32_t c_out, int dtype,
                            const float* scale, const float* shift, const void* residual, int64_t residual_ld,
                            int relu, void* out, int64_t out_ld, int out_dtype, int32_t split_k, void* workspace,
                            int64_t workspace_bytes, int32_t* dev_status, void* stream) {
  if (num_in < 0 || num_out < 0 || num_offsets <= 0 || c_in <= 0 || c_out <= 0) return WCN_ERR_INVALID_PARAMETERS;
  if (num_in >= 0x7FFFFFFFll || num_out >= 0x7FFFFFFFll) return WCN_ERR_INVALID_PARAMETERS;  // row numbers are 32-bit
  if (dtype < WCN_F32 || dtype > WCN_BF16 || out_dtype < WCN_F32 || out_dtype > WCN_BF16)
    return WCN_ERR_INVALID_PARAMETERS;
  if (feats_ld == 0) feats_ld = c_in;  // 0: rows are dense
  if (out_ld == 0) out_ld = c_out;
  if (residual_ld == 0) residual_ld = c_out;
  if (feats_ld < c_in || out_ld < c_out || residual_ld < c_out) return WCN_ERR_INVALID_PARAMETERS;
  if (num_out == 0) return WCN_OK;
  if (!nbr || !out || (num_in > 0 && !feats)) return WCN_ERR_INVALID_PARAMETERS;
  wcn_f32_launches = 1;
  cudaStream_t st = wcn_stream(stream);
  bool tc_ok = wcn_conv_tcgen05_supported(num_offsets, c_in, c_out, dtype, out_dtype);
  if (algo == WCN_CONV_AUTO && weight && tc_ok) {
    // rows that the tensor-core kernel does not read or write (16 bytes at a time): the other kernels take any address
    const int64_t es = wcn_dtype_size(out_dtype);
    auto odd = [](const void* p, int64_t row_bytes) { return ((reinterpret_cast<uintptr_t>(p) | (uintptr_t)row_bytes) & 15) != 0; };
    if (odd(feats, feats_ld * 2) || odd(out, out_ld * es) || (residual && odd(residual, residual_ld * es))) tc_ok = false;
  }
  if (conv_takes_tcgen05(algo, tc_ok, packed_weight, dev_status, num_in)) {
    if (!tc_ok) return WCN_ERR_UNSUPPORTED_CONFIG;
    return wcn_conv_tcgen05_fwd(feats, num_in, feats_ld, packed_weight, nbr, out_rows, num_out, num_offsets, c_in,
                                c_out, dtype, scale, shift, residual, residual_ld, relu, out, out_ld, out_dtype,
                                split_k, dev_status, st);
  }
  if (algo != WCN_CONV_SIMT && algo != WCN_CONV_AUTO) return WCN_ERR_INVALID_PARAMETERS;
  if (!weight) return WCN_ERR_INVALID_PARAMETERS;
  if (algo == WCN_CONV_AUTO && wcn_conv_narrow_supported(num_offsets, c_in, c_out, out, out_ld, residual, residual_ld, out_dtype)) {
    // a few input channels: the streaming kernel (same numbers as the FP32-pipe kernel)
    const int rc = wcn_conv_narrow_fwd(feats, num_in, feats_ld, weight, nbr, out_rows, num_out, num_offsets, c_in,
                                       c_out, dtype, scale, shift, residual, residual_ld, relu, out, out_ld,
                                       out_dtype, dev_status, st);
    if (rc != WCN_ERR_UNSUPPORTED_CONFIG) return rc;
  }
  const bool fp32 = algo == WCN_CONV_AUTO && num_in > 0 &&
                    wcn_conv_fp32_supported(c_in, c_out, dtype, out_dtype, feats, feats_ld, weight, out, out_ld, residual, residual_ld);
  if (fp32 && workspace && dev_status && (reinterpret_cast<uintptr_t>(workspace) & 15) == 0 &&
      wcn_conv_split_supported(num_offsets, c_in, c_out) &&
      workspace_bytes >= wcn_conv_split_workspace(num_in, num_offsets, c_in, c_out)) {
    wcn_f32_launches = 2;
    return wcn_conv_split_fwd(feats, num_in, feats_ld, weight, nbr, out_rows, num_out, num_offsets, c_in, c_out, scale, shift,
                              residual, residual_ld, relu, out, out_ld, split_k, workspace, dev_status, st);
  }
  if (algo == WCN_CONV_AUTO && num_in > 0 && wcn_conv_narrow_out_supported(num_offsets, c_in, c_out, dtype, feats, feats_ld)) {
    // a few output channels (a classification head): one thread per output row
    const int rc = wcn_conv_narrow_out_fwd(feats, num_in, feats_ld, weight, nbr, out_rows, num_out, num_offsets, c_in,
                                           c_out, dtype, scale, shift, residual, residual_ld, relu, out, out_ld,
                                           out_dtype, dev_status, st);
    if (rc != WCN_ERR_UNSUPPORTED_CONFIG) return rc;
  }
  if (fp32) {
    return wcn_conv_fp32_fwd(feats, num_in, feats_ld, weight, nbr, out_rows, num_out, num_offsets, c_in, c_out, scale, shift,
                             residual, residual_ld, relu, out, out_ld, wcn_num_sms(), split_k, dev_status, st);
  }
  return wcn_conv_simt_fwd(feats, num_in, feats_ld, weight, nbr, out_rows, num_out, num_offsets, c_in, c_out, dtype,
                           scale, shift, residual, residual_ld, relu, out, out_ld, out_dtype, dev_status, st);
}

bool wcn_conv_rows_shape_supported(int K, int c_in, int c_out_packed, int dtype, int out_dtype);
int wcn_conv_rows_tcgen05_fwd(const void* feats, int64_t num_in, int64_t feats_ld, const void* packed,
                              const int32_t* dst_rows, int64_t num_out, int K, int c_in, int c_out_packed, int c_out,
                              int dtype, const float* scale, const float* shift, const void* residual,
                              int64_t residual_ld, int relu, void* out, int64_t out_ld, int out_dtype,
                              int32_t* dev_status, cudaStream_t st);

extern "C" int wcn_conv_rows_supported(int32_t num_offsets, int32_t c_in, int32_t c_out_packed, int dtype, int out_dtype,
                                       int32_t* supported) {
  if (!supported) return WCN_ERR_INVALID_PARAMETERS;
  *supported = wcn_conv_rows_shape_supported(num_offsets, c_in, c_out_packed, dtype, out_dtype) ? 1 : 0;
  return WCN_OK;
}

extern "C" int wcn_conv_rows_fwd(const void* feats, int64_t num_in, int64_t feats_ld, const void* packed_weight,
                                 const int32_t* dst_rows, int64_t num_out, int32_t num_offsets, int32_t c_in,
                                 int32_t c_out_packed, int32_t c_out, int dtype, const float* scale, const float* shift,
                                 const void* residual, int64_t residual_ld, int relu, void* out, int64_t out_ld,
                                 int out_dtype, int32_t* dev_status, void* stream) {
  if (num_in < 0 || num_out < 0 || num_offsets <= 0 || c_in <= 0 || c_out <= 0) return WCN_ERR_INVALID_PARAMETERS;
  if (feats_ld == 0) feats_ld = c_in;
  if (out_ld == 0) out_ld = c_out;
  if (residual_ld == 0) residual_ld = c_out;
  if (feats_ld < c_in || out_ld < c_out || residual_ld < c_out) return WCN_ERR_INVALID_PARAMETERS;
  if (num_in == 0 || num_out == 0) return WCN_OK;
  return wcn_conv_rows_tcgen05_fwd(feats, num_in, feats_ld, packed_weight, dst_rows, num_out, num_offsets, c_in,
                                   c_out_packed, c_out, dtype, scale, shift, residual, residual_ld, relu, out, out_ld,
                                   out_dtype, dev_status, wcn_stream(stream));
}

extern "C" int wcn_conv_wgrad(const void* feats, int64_t num_in, const void* grad_out, const int32_t* nbr,
                              const int32_t* out_rows, const uint32_t* tile_masks, int64_t num_out, int32_t num_offsets, int32_t c_in, int32_t c_out, int dtype,
                              float* grad_weight, int32_t* dev_status, void* stream) {
  if (num_in < 0 || num_out < 0 || num_offsets <= 0 || c_in <= 0 || c_out <= 0) return WCN_ERR_INVALID_PARAMETERS;
  if (!wcn_conv_wgrad_tcgen05_supported(num_offsets, c_in, c_out, dtype)) return WCN_ERR_UNSUPPORTED_CONFIG;
  if (num_out == 0 || num_in == 0) return WCN_OK;
  if (!feats || !grad_out || !nbr || !grad_weight || !dev_status) return WCN_ERR_INVALID_PARAMETERS;
  return wcn_conv_wgrad_tcgen05(feats, num_in, grad_out, nbr, out_rows, tile_masks, num_out, num_offsets, c_in, c_out, dtype, grad_weight,
                                dev_status, wcn_stream(stream));
}
