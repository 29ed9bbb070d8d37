/*
 * wcn_b200.h — C ABI of libwcn_b200.so: the sm_100a kernels behind the sparse-convolution
 * hot path (coordinate hash table, kernel-map generation, stride-2 coordinate
 * down-sampling, Morton code, gather-GEMM-scatter convolution with a fused
 * BatchNorm/ReLU/residual epilogue).
 *
 * Conventions
 *  - plain C: device pointers, 64-bit sizes, enum codes; no C++ or torch types.
 *  - every entry point returns an int status (WCN_OK or a negative wcn_status code) and
 *    never throws, exits or allocates device memory: outputs and scratch are passed in,
 *    with a *_bytes query where the size is not obvious.
 *  - `stream` is a cudaStream_t passed as void*; work is enqueued on it and the call
 *    returns without synchronising.
 *  - conditions that can only be detected on the device (hash-table overflow, a bounded
 *    wait that ran out, an index that names no row) are reported through `dev_status`, a
 *    device int32 the caller zeroes beforehand and must read back (poll) when it wants to
 *    know: kernels only ever store a negative wcn_status code into it and it stays set until
 *    the caller zeroes it again.  WCN_ERR_WAIT_EXPIRED overrides the others (the kernel that
 *    stored it gave up half-way): while the word holds it the tensor-core kernels do no work, a
 *    convolution fills the rows it was asked for with NaN and a weight gradient adds nothing.
 *    An out-of-range index is never followed: the access is skipped (the neighbour counts as
 *    absent), the rest of the launch is computed normally and WCN_ERR_BOUNDS is stored if the
 *    word was clean.
 *  - the device the stream belongs to must be the current device of the calling thread
 *    (launch geometry is taken from the current device's properties).
 *  - coordinates are int32 rows (batch, x, y, z).  The batch value INT32_MIN is reserved
 *    (it marks an empty hash slot).
 *
 * Each declaration names the reference interface it replaces (paths relative to the
 * reference project root).
 */
#ifndef WCN_B200_H_
#define WCN_B200_H_

#include <stddef.h>
#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

/* Status codes.  -1..-5 mirror the reference's GemmStatus
 * (warpconvnet/csrc/include/gemm_error_codes.h:5-13); the rest are new. */
enum wcn_status {
  WCN_OK = 0,
  WCN_ERR_PROBLEM_NOT_SUPPORTED = -1,
  WCN_ERR_INITIALIZATION = -2,
  WCN_ERR_EXECUTION = -3,
  WCN_ERR_UNSUPPORTED_CONFIG = -4,
  WCN_ERR_INVALID_PARAMETERS = -5,
  WCN_ERR_HASH_OVERFLOW = -6,
  WCN_ERR_WAIT_EXPIRED = -7,
  WCN_ERR_BOUNDS = -8,
  WCN_ERR_SCRATCH_TOO_SMALL = -9
};

/* Element types of feature / weight tensors. */
enum wcn_dtype { WCN_F32 = 0, WCN_F16 = 1, WCN_BF16 = 2 };

/* Hash functions, in the order of HashMethod
 * (warpconvnet/geometry/coords/search/torch_hashmap.py:17-32). */
enum wcn_hash_method { WCN_HASH_FNV1A = 0, WCN_HASH_CITY = 1, WCN_HASH_MURMUR = 2 };

/* Reductions of wcn_row_reduce, the native part of REDUCTIONS (warpconvnet/ops/reductions.py:13-21). */
enum wcn_reduce_op { WCN_REDUCE_MIN = 0, WCN_REDUCE_MAX = 1, WCN_REDUCE_SUM = 2, WCN_REDUCE_MEAN = 3, WCN_REDUCE_MUL = 4 };

/* Convolution kernels selectable through wcn_conv_fwd's `algo`. */
enum wcn_conv_algo { WCN_CONV_AUTO = 0, WCN_CONV_SIMT = 1, WCN_CONV_TCGEN05 = 2 };

/* Library version (major*10000 + minor*100 + patch). No reference counterpart. */
int wcn_version(void);

/* Human-readable text of a status code.
 * Replaces gemm_status_to_string (warpconvnet/csrc/warpconvnet_pybind.cpp:1220-1226). */
const char* wcn_status_string(int status);

/* ------------------------------------------------------------------ hash table */

/* Bytes of the table buffer for `capacity` slots (16-byte key + 4-byte value per slot, and a
 * 16-byte tail whose first word records whether a key was inserted twice).
 * Replaces the `[capacity, 2] int32` allocation in TorchHashTable.insert
 * (warpconvnet/geometry/coords/search/torch_hashmap.py:142). */
int wcn_hash_table_bytes(int64_t capacity, int64_t* bytes);

/* Clear the table and insert keys[n,4]; the value of a key is its row index (the smallest
 * one when a key occurs more than once).  stride = {sx,sy,sz} floor-divides x,y,z before
 * insertion ({1,1,1} or NULL: keys as given).  Needs n <= capacity.
 * skip_if (device int32, may be NULL): when it holds a non-zero value at the time the kernels run,
 * they do nothing and the table is left unbuilt — for a table that only backs up a brick table
 * (pass wcn_brick_usable_flag(brick_table), built earlier on the same stream): it is filled exactly
 * when wcn_kmap_search_bricks will need it.  A caller that later wants to probe the table itself
 * builds it again with skip_if = NULL.
 * Replaces prepare_key_value_pairs_kernel + insert_kernel_{fnv1a,city,murmur}
 * (warpconvnet/csrc/hashmap_kernels.cu:182-234, 258-270). */
int wcn_hash_build(const int32_t* keys, int64_t n, const int32_t* stride, void* table,
                   int64_t capacity, int hash_method, const int32_t* skip_if, int32_t* dev_status, void* stream);

/* results[i] = value of queries[i] in the table, or -1.
 * Replaces search_kernel_{fnv1a,city,murmur} (warpconvnet/csrc/hashmap_kernels.cu:237-301). */
int wcn_hash_search(const void* table, int64_t capacity, int hash_method, const int32_t* queries,
                    int64_t num_queries, int32_t* results, void* stream);

/* ------------------------------------------------------------------ distinct / strided coordinates */

/* Scratch bytes for wcn_unique_mark / wcn_unique_emit over n rows. */
int wcn_unique_workspace_bytes(int64_t n, int64_t* bytes);

/* Phase 1: with the table built by wcn_hash_build over the same (coords, stride), mark the
 * first occurrence of every distinct row of floor(coords / [1,sx,sy,sz]) and count them
 * into num_unique (device int64).
 * Replaces TorchHashTable.unique_index (torch_hashmap.py:303-322: search of all keys
 * followed by torch.unique) as used by stride_coords
 * (warpconvnet/geometry/coords/ops/stride.py:41-43). */
int wcn_unique_mark(const int32_t* coords, int64_t n, const int32_t* stride, const void* table,
                    int64_t capacity, int hash_method, void* workspace, int64_t* num_unique,
                    void* stream);

/* Phase 2 (after the caller has read num_unique and sized the outputs): write the distinct
 * rows in first-occurrence order to out_coords[num_unique,4], their source rows to
 * unique_index[num_unique], and for every input row the output row it collapsed into to
 * parent[n].  unique_index / parent may be NULL.
 * Replaces the gather `discretized_coords[unique_indices]` and the batch argsort of
 * stride_coords (stride.py:43-48); the order produced here is deterministic. */
int wcn_unique_emit(const int32_t* coords, int64_t n, const int32_t* stride, void* workspace,
                    int32_t* out_coords, int32_t* unique_index, int32_t* parent, void* stream);

/* ------------------------------------------------------------------ kernel map */

/* Scratch bytes for the three kernel-map calls (per-block hit counts). */
int wcn_kmap_workspace_bytes(int64_t num_queries, int32_t num_offsets, int64_t* bytes);

/* nbr[k*M + m] = row of (b, x*sx + i - cx, y*sy + j - cy, z*sz + l - cz) in the table or
 * -1, for k = (i*ky + j)*kz + l and c = size/2 for odd sizes, 0 for even sizes; also the
 * per-block hit counts in `workspace` (NULL: no counts; wcn_kmap_count makes them later if a
 * compact map is ever asked for).  num_offsets limits k to the first num_offsets
 * positions (the reference's skip_symmetric mode passes K/2).
 * Replaces kernel_map_size_4d_{fnv1a,city,murmur}
 * (warpconvnet/csrc/discrete_kernels.cu:264-334, 339-370). */
int wcn_kmap_search(const void* table, int64_t capacity, int hash_method, const int32_t* queries,
                    int64_t num_queries, const int32_t* stride, const int32_t* kernel_size,
                    int32_t num_offsets, int32_t* nbr, void* workspace, void* stream);

/* offsets[k] = number of hits of all offsets < k (device int32 [num_offsets+1]); turns the
 * per-block counts in `workspace` into write positions.
 * Replaces the cumsum/max/cumsum chain of _kernel_map_search_to_result
 * (warpconvnet/geometry/coords/search/torch_discrete.py:103-119). */
int wcn_kmap_scan(void* workspace, int64_t num_queries, int32_t num_offsets, int32_t* offsets,
                  void* stream);

/* wcn_kmap_search with dilated windows and a free window centre: position (i, j, l) of the
 * window probes x*sx + (i - cx)*dx and so on; `dilation` NULL means 1, `center` = {cx,cy,cz}
 * NULL means the default centre (size/2 for odd sizes, 0 for even sizes).
 * Replaces kernel_offsets_from_size with a kernel_dilation / center_offset and the offset-list
 * search _kernel_map_from_offsets (warpconvnet/geometry/coords/search/torch_discrete.py:44-77, 160-241). */
int wcn_kmap_search_dilated(const void* table, int64_t capacity, int hash_method, const int32_t* queries,
                            int64_t num_queries, const int32_t* stride, const int32_t* kernel_size,
                            const int32_t* dilation, const int32_t* center, int32_t num_offsets, int32_t* nbr,
                            void* workspace, void* stream);

/* wcn_kmap_search followed by wcn_kmap_scan, for callers that must not allocate device
 * memory.  Some hosts of this library cannot call cudaMalloc around it: plugins that are
 * handed a fixed arena by their framework and own no allocator, serving loops whose latency
 * budget forbids allocator calls (cudaMalloc synchronises the device), processes whose
 * memory pool is already exhausted or too fragmented for one more block.  For them the
 * per-block hit counts live in a fixed 4 MiB array inside the library image instead of a
 * caller-supplied workspace; the caller passes only inputs (table, queries) and outputs
 * (nbr[num_offsets * num_queries], offsets[num_offsets + 1], both device memory).
 * Limit: num_offsets * ceil(num_queries / 256) + num_offsets + 16 <= 1048576 (about 9.9 M
 * queries for a 3x3x3 window); larger problems return WCN_ERR_SCRATCH_TOO_SMALL and launch
 * nothing.  The entry point calls no allocator of any kind.  The first call on a device
 * looks up the array's device address (cudaGetSymbolAddress) for the CURRENT device, so the
 * device that owns `stream` must be current in the calling thread; make that first call before
 * any stream capture begins (concurrent first calls from several host threads are safe).  The
 * scanned hit counts stay inside the library, so this call yields the dense table and the
 * per-offset totals only: a caller that also wants the compact (in, out) lists runs
 * wcn_kmap_count + wcn_kmap_scan + wcn_kmap_compact with a workspace of its own.  All calls on a device share the one array and it keeps the last
 * call's contents (nothing in it needs clearing between calls), so two calls whose kernels
 * overlap on the GPU — different streams, no ordering between them — race; serialise them.
 * Every GPU that loads the library holds the array until the process exits.
 * No counterpart in the reference (its kernel-map path allocates through CuPy / torch on
 * every call, warpconvnet/geometry/coords/search/torch_discrete.py:312-315, 103-124). */
int wcn_kmap_search_static(const void* table, int64_t capacity, int hash_method,
                           const int32_t* queries, int64_t num_queries, const int32_t* stride,
                           const int32_t* kernel_size, int32_t num_offsets, int32_t* nbr,
                           int32_t* offsets, void* stream);

/* Compact nbr into in_maps / out_maps (length offsets[num_offsets]); within one offset the
 * pairs are in ascending output row.
 * Replaces map_found_indices_to_maps_cuda (warpconvnet/csrc/discrete_kernels.cu:183-213, 250-259). */
int wcn_kmap_compact(const int32_t* nbr, int64_t num_queries, int32_t num_offsets,
                     const void* workspace, const int32_t* offsets, int32_t* in_maps,
                     int32_t* out_maps, void* stream);

/* Dense neighbour table from a compact map: nbr[k*M + out_maps[p]] = in_maps[p] for
 * offsets[k] <= p < offsets[k+1], -1 elsewhere.  Requires out_maps to be distinct within
 * one offset (true of every map the reference builds).
 * Replaces nothing directly: the reference's kernels consume the compact lists
 * (warpconvnet/nn/functional/sparse_conv.py:300-310); this is the layout the
 * output-stationary convolution reads. */
int wcn_nbr_from_maps(const int32_t* in_maps, const int32_t* out_maps, const int32_t* offsets,
                      int32_t num_offsets, int64_t num_pairs, int64_t num_out, int32_t* nbr,
                      void* stream);

/* Neighbour table of the transposed map: nbr_t[k*num_in + i] = m wherever
 * nbr_fwd[k*num_out + m] = i, -1 elsewhere.  Requires each input row to occur at most once
 * per offset (true of every map the reference builds).
 * Replaces the in/out swap `IntSearchResult(in_maps=fwd.out_maps, out_maps=fwd.in_maps, ...)`
 * of transposed convolutions (warpconvnet/nn/functional/sparse_conv.py:1934-1938, 1953-1957). */
int wcn_nbr_transpose(const int32_t* nbr_fwd, int32_t num_offsets, int64_t num_out, int64_t num_in,
                      int32_t* nbr_t, void* stream);

/* Kernel map of a coordinate set onto itself: `keys` are the rows the table was built from
 * (same order), the window is odd (dilated by `dilation`, NULL = 1) and the stride 1, so nbr is [K, num_keys] with
 * K = kx*ky*kz.  Same result as wcn_kmap_search on those arguments.  When the keys are
 * distinct (the table records whether they are) the map is symmetric, nbr[k][m] = i exactly
 * when nbr[K-1-k][i] = m, and only the first half of the offsets and the centre are probed.
 * Leaves no hit counts.
 * Replaces kernel_map_size_4d_* for the submanifold case, i.e. what the reference's
 * skip_symmetric_kernel_map flag hints at (warpconvnet/geometry/coords/search/torch_discrete.py:291-296)
 * but never completes into the full map. */
int wcn_kmap_search_self(const void* table, int64_t capacity, int hash_method, const int32_t* keys,
                         int64_t num_keys, const int32_t* kernel_size, const int32_t* dilation, int32_t* nbr,
                         void* stream);

/* Bytes of the brick table of a coordinate set of n rows (a 32-byte header and one 32-byte entry
 * per slot, 2 n slots allocated, four per brick used). */
int wcn_brick_table_bytes(int64_t n, int64_t* bytes);

/* Brick table of keys[n,4]: one entry per 4x4x4 brick (aligned to `origin`, a DEVICE pointer to
 * three int32, NULL = 0) holding the brick's 64-bit occupancy mask and the row of its first voxel.
 * It is usable when the rows of every brick are consecutive and in Morton order inside the brick
 * — what sorting by the Morton code of (coords - origin) gives (Voxels.sort) — and the rows are
 * distinct; the build checks that on the device and marks the table unusable otherwise, in
 * which case wcn_kmap_search_bricks answers from the voxel table instead.  No host
 * synchronisation.
 * No counterpart in the reference, whose kernel map probes one voxel key per offset
 * (warpconvnet/csrc/discrete_kernels.cu:264-334) whatever the order of the rows; the ordering
 * itself is the reference's (warpconvnet/geometry/types/voxels.py:255-267,
 * warpconvnet/csrc/morton_code.cu:15-22). */
int wcn_brick_build(const int32_t* keys, int64_t n, const int32_t* origin, void* table, void* stream);

/* Device address of the word of a brick table that is non-zero when the table is usable (valid
 * after wcn_brick_build has run on the stream); what wcn_hash_build takes as skip_if.  Host-only,
 * launches nothing.  No counterpart in the reference. */
const int32_t* wcn_brick_usable_flag(const void* brick_table);

/* wcn_kmap_search (same nbr[k*M + m], same offset order and centre rule, dilation 1) answered
 * from a brick table: one thread per query fetches the at most 2x2x2 brick entries its window
 * touches and resolves every offset from them.  Window sizes up to 4 per axis
 * (WCN_ERR_UNSUPPORTED_CONFIG beyond).  `table` / `capacity` / `hash_method` are the voxel table
 * of the same keys (wcn_hash_build), used when the brick table was marked unusable.
 * Replaces kernel_map_size_4d_{fnv1a,city,murmur}
 * (warpconvnet/csrc/discrete_kernels.cu:264-334, 339-370) for Morton-ordered inputs. */
int wcn_kmap_search_bricks(const void* brick_table, const void* table, int64_t capacity, int hash_method,
                           const int32_t* queries, int64_t num_queries, const int32_t* stride,
                           const int32_t* kernel_size, int32_t* nbr, void* stream);

/* Per-block hit counts of a dense neighbour table into `workspace`, exactly what
 * wcn_kmap_search leaves there; for maps that were searched without counts.
 * Replaces the `found >= 0` pass of map_found_indices_to_maps_cuda
 * (warpconvnet/csrc/discrete_kernels.cu:183-213). */
int wcn_kmap_count(const int32_t* nbr, int64_t num_queries, int32_t num_offsets, void* workspace,
                   void* stream);

/* Tile order of a neighbour table: within each window of consecutive output rows (4096 rows for
 * tables of at most 4096 rows, else 16384) the rows are sorted by their neighbour-presence key (a
 * bit per offset, set when nbr[k][m] >= 0; for 27 offsets the centre of the 3x3x3 window is bit 0,
 * then the face, edge and corner offsets, so the rarest ones are the most significant; otherwise bit
 * k; ties by row), so that rows with the same present offsets share a 128-row tile and the
 * convolution skips the (tile, offset) pairs that have no neighbour at all.
 *   out_rows[s]        the output row that slot s of the tiled table stands for (a permutation
 *                      of 0..num_out-1 that moves no row out of its window)
 *   nbr_tiled[k][s]    = nbr[k][out_rows[s]]
 * Pass both to wcn_conv_fwd (nbr = nbr_tiled, out_rows = out_rows); the results are bit
 * identical to the untiled call.  num_offsets <= 32.  Deterministic.
 * No reference counterpart: the reference's implicit GEMM walks per-offset pair lists
 * (warpconvnet/nn/functional/sparse_conv.py:300-310) and never forms output tiles. */
int wcn_kmap_tile_order(const int32_t* nbr, int64_t num_out, int32_t num_offsets, int32_t* out_rows,
                        int32_t* nbr_tiled, void* stream);

/* masks[t] = set of offsets k (bit k) for which some row of [128 t, 128 t + 128) has nbr[k][row] >= 0;
 * ceil(num_out / 128) words, num_offsets <= 32.  Lets a kernel that walks the table in 128-row
 * steps (wcn_conv_wgrad) skip the steps that cannot contribute.  No reference counterpart. */
int wcn_kmap_tile_masks(const int32_t* nbr, int64_t num_out, int32_t num_offsets, uint32_t* masks,
                        void* stream);

/* Table of 4x4x4 cells over keys [n, 4] in any order (32-byte aligned buffer of wcn_cells_bytes; 256 bytes per key are
 * reserved for the rows of a cell, of which as many are touched as there are cells), and windows up to four wide answered
 * from it: nbr as wcn_kmap_search writes it, repeated keys resolving to the smallest row.  `workspace` (may be NULL)
 * receives the per-block hit counts wcn_kmap_scan wants.
 * Replaces the per-offset probes of kernel_map_size_4d (warpconvnet/csrc/discrete_kernels.cu:264-334). */
int wcn_cells_bytes(int64_t n, int64_t* bytes);
int wcn_cells_build(const int32_t* keys, int64_t n, void* table, void* stream);
int wcn_kmap_search_cells(const void* table, int64_t n, const int32_t* queries, int64_t num_queries,
                          const int32_t* stride, const int32_t* kernel_size, int32_t* nbr, void* workspace, void* stream);

/* wcn_kmap_scan that also leaves the offsets [num_offsets + 1] and the device status word in pinned host memory
 * (int32 [num_offsets + 2]), valid once the stream has passed it. */
int wcn_kmap_scan_host(void* workspace, int64_t num_queries, int32_t num_offsets, int32_t* offsets, int32_t* host,
                       const int32_t* dev_status, void* stream);

/* After wcn_unique_mark / wcn_unique_emit over n rows: host (pinned int32 [items + 3]) = number of distinct rows, device
 * status word, distinct rows of batch items 0..items-1, rows of any other item.  hist: int32 [items + 1] scratch.
 * Replaces the bincount behind the output offsets (warpconvnet/geometry/coords/ops/stride.py:48-54). */
int wcn_unique_counts(const int32_t* rows, int64_t n, const void* workspace, int32_t items, int32_t* hist, int32_t* host,
                      const int32_t* dev_status, void* stream);

/* ------------------------------------------------------------------ Morton code */

/* codes[i] = 3-D Morton code of (x - min_xyz[0], y - min_xyz[1], z - min_xyz[2]), x in bit
 * 0, y in bit 1, z in bit 2, up to 21 bits per axis.  coords has `row_ints` int32 per row
 * and the x column at `col0` (3,0 for xyz rows; 4,1 for batch-indexed rows).  `min_xyz` is a
 * DEVICE pointer to three int32 (or NULL for no shift), so the caller's min-reduction needs
 * no round trip to the host.
 * Replaces assign_order_discrete_20bit_kernel_4points (warpconvnet/csrc/morton_code.cu:71-94)
 * and the min subtraction of morton_code (coords/ops/serialization.py:224-225). */
int wcn_morton20(const int32_t* coords, int64_t n, int32_t row_ints, int32_t col0,
                 const int32_t* min_xyz, int64_t* codes, void* stream);

/* ------------------------------------------------------------------ convolution */

/* dst[r, :] = src[idx[r], :]  (rows of `channels` elements; src has num_src rows).  An idx
 * outside [0, num_src) yields a zero row and WCN_ERR_BOUNDS in dev_status (NULL: not reported).
 * Replaces the `comp_in_feats[in_map]` gather of _explicit_gemm_forward_logic
 * (warpconvnet/nn/functional/sparse_conv.py:309). */
int wcn_gather_rows(const void* src, int64_t num_src, const int32_t* idx, void* dst, int64_t num_rows,
                    int32_t channels, int dtype, int32_t* dev_status, void* stream);

/* dst[idx[r], :] += src[r, :]; idx must hold distinct rows (one kernel offset; dst has num_dst
 * rows).  An idx outside [0, num_dst) is skipped and reported like above.
 * Replaces `output_feature_tensor[out_map] += ...` (sparse_conv.py:310). */
int wcn_scatter_add_rows(const void* src, const int32_t* idx, void* dst, int64_t num_dst, int64_t num_rows,
                         int32_t channels, int dtype, int32_t* dev_status, void* stream);

/* Bytes of the packed-weight buffer wcn_conv_fwd needs for (algo, shape, dtype); 0 when
 * the chosen kernel reads the weights as given. */
int wcn_conv_packed_weight_bytes(int algo, int32_t num_offsets, int32_t c_in, int32_t c_out,
                                 int dtype, int64_t* bytes);

/* Re-layout weight[K, c_in, c_out] into the buffer above (K-major tiles for the tensor-core
 * kernel).  No reference counterpart (its kernels read the weights as stored). */
/* wcn_conv_pack_weight from a weight tensor of another dtype (converted as it is packed), of its transpose per offset
 * (transposed != 0: weight is [K, c_out, c_in]) and with the offsets in reverse order (reversed != 0): a gradient's
 * weights in one launch. */
int wcn_conv_pack_weight_from(const void* weight, int src_dtype, int32_t num_offsets, int32_t c_in, int32_t c_out, int dtype,
                              int32_t transposed, int32_t reversed, void* packed, void* stream);
int wcn_conv_pack_weight(int algo, const void* weight, int32_t num_offsets, int32_t c_in,
                         int32_t c_out, int dtype, void* packed, void* stream);

/* Bytes of `workspace` wcn_conv_fwd needs for this problem: 0 in this version (the slices of split_k are added through
 * distributed shared memory), so NULL may be passed.
 * (warpconvnet/csrc/implicit_gemm_split_k.cu:254-258 allocates its partial sums inside the call.) */
int wcn_conv_workspace_bytes(int algo, int64_t num_out, int32_t num_offsets, int32_t c_in, int32_t c_out,
                             int dtype, int out_dtype, int32_t split_k, int64_t* bytes);

/* Bytes of `workspace` with which wcn_conv_fwd runs an fp32 problem on the tensor cores, every number as the exact sum of
 * three bf16 numbers (csrc/conv_split_tcgen05.cu; its results are closer to exact sums than those of the FP32 pipes); 0
 * where it does not.  Any 16-byte aligned device memory, used from the first launch of the call to its last.
 * No reference counterpart. */
int wcn_conv_f32_workspace_bytes(int64_t num_in, int64_t num_out, int32_t num_offsets, int32_t c_in, int32_t c_out, int64_t* bytes);
/* Kernels that this thread's last wcn_conv_fwd or wcn_conv_wgrad_f32 launched (with a workspace or partial sums more than one). */
int wcn_conv_f32_launches(void);

/* Output-stationary sparse convolution with a fused epilogue:
 *   acc[s, :] = sum_k feats[nbr[k*M + s], :] @ weight[k]      (rows with nbr < 0 skipped, fp32 accumulation)
 *   m = out_rows[s]           (out_rows NULL: m = s; else a permutation of 0..M-1, see
 *                              wcn_kmap_tile_order, with nbr being that call's nbr_tiled)
 *   y = acc * scale + shift   (scale NULL: y = acc + shift; both NULL: y = acc)
 *   y += residual[m, :]       (residual NULL: skipped; residual has the output dtype)
 *   y = max(y, 0)             (relu != 0)
 *   out[m, :] = (out dtype) y
 * feats / weight share `dtype`; scale / shift are fp32 [c_out].  Each output row is written
 * once by the block that owns it: no atomics, bit-reproducible.
 * feats_ld / residual_ld / out_ld are the distances between consecutive rows of the three
 * matrices in elements (0 = dense: c_in / c_out), so a matrix may be a column block of a wider
 * one (a skip connection's half of a concatenated buffer); rows must start on 16-byte boundaries
 * for the tensor-core kernel.  nbr entries >= num_in count as absent and raise WCN_ERR_BOUNDS.
 * num_in and M are below 2^31 (row numbers are 32-bit); larger values return WCN_ERR_INVALID_PARAMETERS.
 * algo WCN_CONV_TCGEN05 needs dtype f16/bf16, c_in >= 16, c_in % 8 == 0, c_out % 16 == 0, 16 <= c_out <= 256
 * and `packed_weight` from wcn_conv_pack_weight; WCN_CONV_AUTO picks it when those hold and
 * packed_weight is not NULL, else the SIMT kernel.
 * split_k: the tensor-core kernel may divide the kernel offsets of a 128-row block among the S CTAs of a cluster (slice s
 * owns the offsets k with k % S == s), whose fp32 sums are added in slice order before the epilogue: for problems with
 * fewer row blocks than multiprocessors.  0 = the library decides, 1 = never, 2.. = that many slices (at most 8); a
 * negative value divides the OUTPUT COLUMNS into -split_k blocks instead (a tuning aid).  `workspace` must hold
 * wcn_conv_workspace_bytes(...) for the same arguments (NULL / 0 when that is 0); fp32 problems under WCN_CONV_AUTO take one
 * of wcn_conv_f32_workspace_bytes(...), with the same meaning of split_k > 0, and run on the FP32 pipes without.
 * With split_k = 1 a row's sums do not depend on which other rows a launch has (asked with the same num_out, that query gives
 * the same answer for all of them).  Results are the same bits on every run for a given S and, in fp32, with the workspace
 * given or not given each time (the two round differently: a caller that goes on without one for want of memory gets the
 * FP32 pipes' bits); different S round differently (fp32 sums are grouped by slice).
 * Replaces implicit_gemm (warpconvnet/csrc/warpconvnet_pybind.cpp:732-837,
 * warpconvnet/csrc/implicit_gemm.cu:44-267) and cutlass_gemm_AD_gather_scatter with its
 * split_k_slices argument (warpconvnet_pybind.cpp:396-509,
 * warpconvnet/csrc/cutlass_gemm_gather_scatter.cu:176-464), the per-offset loop around them
 * (warpconvnet/nn/functional/sparse_conv.py:396-413, 516-544), the bias add
 * (sparse_conv.py:1794-1795) and the BatchNorm1d / ReLU / residual-add / concatenation chain of
 * the model blocks (examples/mink_unet.py:36-47, 129-141, 340-358). */
int wcn_conv_fwd(int algo, const void* feats, int64_t num_in, int64_t feats_ld, const void* weight,
                 const void* packed_weight, const int32_t* nbr, const int32_t* out_rows, int64_t num_out,
                 int32_t num_offsets, int32_t c_in, int32_t c_out, int dtype, const float* scale,
                 const float* shift, const void* residual, int64_t residual_ld, int relu, void* out,
                 int64_t out_ld, int out_dtype, int32_t split_k, void* workspace, int64_t workspace_bytes,
                 int32_t* dev_status, void* stream);

/* Pooling over a kernel map: out[m, :] = op over the offsets k with nbr[k*M + m] >= 0 of
 * feats[nbr[k*M + m], :] (fp32 accumulation, offsets in ascending order; rows without a neighbour
 * become 0; mean divides by the number of neighbours).  With the transposed table of a
 * non-overlapping pooling it is the un-pooling gather.  nbr entries >= num_in count as absent
 * and raise WCN_ERR_BOUNDS in dev_status (NULL: not reported).
 * Replaces kernel_map.to_csr() + row_reduction / torch_scatter.segment_csr of sparse_reduce
 * (warpconvnet/nn/functional/sparse_pool.py:87-92, warpconvnet/ops/reductions.py:36-70) and the
 * argsort + gather of sparse_unpool (sparse_pool.py:168-172). */
int wcn_row_reduce(const void* feats, int64_t num_in, const int32_t* nbr, int64_t num_out, int32_t num_offsets,
                   int32_t channels, int dtype, int op, void* out, int32_t* dev_status, void* stream);

/* The same, leaving what its gradient needs (each may be NULL): `arg` [num_out, channels] of arg_bytes = 1 (at most
 * 255 offsets) or 2 bytes per element (min, max: the first offset that attained the result, all ones where there is
 * none) and `count` [num_out] (mean: neighbours of the row, at least 1). */
int wcn_row_reduce_train(const void* feats, int64_t num_in, const int32_t* nbr, int64_t num_out, int32_t num_offsets,
                         int32_t channels, int dtype, int op, void* out, void* arg, int32_t arg_bytes, float* count,
                         int32_t* dev_status, void* stream);

/* Gradient of a pooling with respect to its features, over the transposed table nbr_t [num_offsets, num_in]:
 * grad_in[i, :] = sum over the offsets k with m = nbr_t[k*num_in + i] >= 0 of grad_out[m, :] (divided by count[m] when
 * `count` is given; where arg[m] == k only, when `arg` is given).  fp32 accumulation in order of k. */
int wcn_row_reduce_backward(const void* grad_out, int64_t num_out, const int32_t* nbr_t, int64_t num_in,
                            int32_t num_offsets, int32_t channels, int dtype, const void* arg, int32_t arg_bytes,
                            const float* count, void* grad_in, int32_t* dev_status, void* stream);

/* Convolution in which every output row has exactly one (input row, kernel offset) pair, run from the
 * INPUT side on the tensor cores: a 1x1x1 convolution (optionally writing through a row permutation)
 * and a transposed convolution whose window equals its stride (2x2x2, stride 2).  For input row j and
 * offset k, out[dst_rows[k * num_in + j], :] = epilogue(feats[j, :] @ weight[k]); entries < 0 name no
 * output row.  dst_rows == NULL (num_offsets must be 1) means dst = j.  The caller guarantees that no
 * output row is named twice (it would be written twice, last writer wins) — for the stride-2 case
 * dst_rows is the [8, num_coarse] neighbour table of the matching strided convolution.
 * Feature rows arrive through TMA tiles (16-byte aligned base and pitch), weights (packed by
 * wcn_conv_pack_weight at width c_out_packed, a multiple of 16 >= c_out whose extra columns are zero)
 * stay in shared memory; fp16 / bf16 features, c_in % 32 == 0, c_out_packed <= 256.
 * The reference runs these layers through the same gather-GEMM-scatter as every other convolution
 * (warpconvnet/nn/functional/sparse_conv.py:358-415 with the swapped kernel map of :1916-1945). */
int wcn_conv_rows_supported(int32_t num_offsets, int32_t c_in, int32_t c_out_packed, int dtype, int out_dtype,
                            int32_t* supported);
int wcn_conv_rows_fwd(const void* feats, int64_t num_in, int64_t feats_ld, const void* packed_weight,
                      const int32_t* dst_rows, int64_t num_out, int32_t num_offsets, int32_t c_in,
                      int32_t c_out_packed, int32_t c_out, int dtype, const float* scale, const float* shift,
                      const void* residual, int64_t residual_ld, int relu, void* out, int64_t out_ld,
                      int out_dtype, int32_t* dev_status, void* stream);

/* Weight gradient of the convolution above, accumulated into grad_weight[K, c_in, c_out] (fp32; the
 * caller zeroes it):
 *   grad_weight[k] += feats[nbr[k*M + m], :]^T (outer) grad_out[m, :]   over rows m with nbr >= 0
 * feats / grad_out share `dtype` (f16 or bf16), fp32 accumulation on the tensor cores; the partial
 * sums of different row ranges are added with atomics, so the last bits vary from run to run.
 * Needs c_in >= 16, c_in % 8 == 0, c_out % 16 == 0, c_out <= 256; else WCN_ERR_UNSUPPORTED_CONFIG (callers
 * take wcn_conv_wgrad_pairs).  (`nbr`, `out_rows`) is the pair wcn_conv_fwd takes: the plain table
 * with out_rows NULL, or the tiled one with its row order (grad_out is then read at out_rows[s]);
 * `tile_masks` (from wcn_kmap_tile_masks on the same table, or NULL) lets the kernel skip the 128-row
 * steps in which the offsets of a CTA have no neighbour.
 * Replaces cutlass_gemm_trAB_gather (warpconvnet/csrc/warpconvnet_pybind.cpp:511-624) and
 * split_k_implicit_gemm (warpconvnet/csrc/implicit_gemm_split_k.cu:63-393) with the per-offset loop
 * around them (warpconvnet/nn/functional/sparse_conv.py:591-604). */
int wcn_conv_wgrad(const void* feats, int64_t num_in, const void* grad_out, const int32_t* nbr,
                   const int32_t* out_rows, const uint32_t* tile_masks, int64_t num_out, int32_t num_offsets, int32_t c_in, int32_t c_out, int dtype,
                   float* grad_weight, int32_t* dev_status, void* stream);

/* The same gradient of fp32 tensors on the tensor cores, every number as the exact sum of three bf16 numbers: grad_weight
 * (16-byte aligned, like the other matrices and the workspace) is written, the same bits on every run.  c_in and c_out are
 * multiples of 4 from 16 on, num_offsets at most 32, tile_masks must be given; 0 bytes: not taken. */
int wcn_conv_wgrad_f32_workspace_bytes(int64_t num_in, int64_t num_out, int32_t num_offsets, int32_t c_in, int32_t c_out, int64_t* bytes);
int wcn_conv_wgrad_f32(const float* feats, int64_t num_in, const float* grad_out, const int32_t* nbr, const int32_t* out_rows,
                       const uint32_t* tile_masks, int64_t num_out, int32_t num_offsets, int32_t c_in, int32_t c_out,
                       float* grad_weight, void* workspace, int64_t workspace_bytes, int32_t* dev_status, void* stream);

/* The same gradient on the FP32 pipes, for any dtype and widths (fp32 tensors, a 3-channel stem): grad_weight is
 * written, not accumulated into, from partial sums of row ranges added in order (the same bits on every run).
 * `workspace`: wcn_conv_wgrad_pairs_workspace_bytes bytes (0: none needed). */
int wcn_conv_wgrad_pairs_workspace_bytes(int64_t num_out, int32_t num_offsets, int32_t c_in, int32_t c_out, int64_t* bytes);
int wcn_conv_wgrad_pairs(const void* feats, int64_t num_in, const void* grad_out, const int32_t* nbr,
                         const int32_t* out_rows, int64_t num_out, int32_t num_offsets, int32_t c_in, int32_t c_out,
                         int dtype, float* grad_weight, void* workspace, int64_t workspace_bytes, int32_t* dev_status,
                         void* stream);

/* ------------------------------------------------------------------ Morton order, pyramid, maps of all levels */

/* Rows of a batch of voxel sets in Morton order, one cooperative launch:
 *   perm [n] int64      sorted row -> caller's row, stable by (batch item, code)
 *   codes [n] int64     Morton code of the caller's rows about the corner
 *   rows [n, 4] int32   sorted (batch, x, y, z), 16-byte aligned
 *   info [8] int32      [0..2] the corner: the per-axis minimum rounded down to a multiple of 16; [3] bits per axis of
 *                       the codes; [4] 1 when no two positions share a code (extent below 2^21)
 *   feats_sorted        rows of feat_row_bytes (even; feats NULL: none) in sorted order
 * `offsets` is a HOST array [batches + 1] of row offsets; at most 255 batch items (else WCN_ERR_UNSUPPORTED_CONFIG).
 * Replaces the per-batch argsort of warpconvnet/coords/ops/serialization.py:60-254 behind Voxels.sort
 * (geometry/types/voxels.py:255-267). */
int wcn_morton_sort_workspace_bytes(int64_t n, int64_t* bytes);
int wcn_morton_sort(const int32_t* coords, int64_t n, const int64_t* offsets, int32_t batches, int64_t* codes,
                    int64_t* perm, int32_t* rows, int32_t* info, const void* feats, void* feats_sorted,
                    int32_t feat_row_bytes, void* workspace, int32_t* dev_status, void* stream);

/* The coarser levels of rows sorted by wcn_morton_sort: level l (1..levels, at most 4) holds the distinct rows of
 * floor(row / 2^l) in first-occurrence order, as wcn_unique_emit gives them.
 *   out [levels, n, 4], first [levels, n]   rows of each level and, per row, its first row on the level below
 *   counts [24]   [0..6] distinct cells of 2^s voxels about the corner, [7] non-zero when two rows are equal,
 *                 [8 + 4 l ..] the corner of level l + 1 (a copy in 16-byte steps)
 *   host          HOST-mapped (pinned) int64 [levels * (batches + 1) + 2]: row offsets of every level, then 1 when the
 *                 levels are usable (rows distinct, codes whole), then the device status word.  Written by the kernel:
 *                 valid once the stream has passed it.
 * Replaces stride_coords level by level (warpconvnet/geometry/coords/ops/stride.py:17-54). */
int wcn_pyramid_workspace_bytes(int64_t n, int64_t* bytes);
int wcn_pyramid(const int32_t* rows, int64_t n, const int32_t* info, const int64_t* offsets, int32_t batches,
                int32_t levels, int32_t* out, int32_t* first, int32_t* counts, int64_t* host, void* workspace,
                const int32_t* dev_status, void* stream);

/* One level of wcn_level_maps. */
typedef struct {
  const int32_t* rows;        /* [n, 4] of wcn_morton_sort (level 0) or wcn_pyramid */
  int64_t n;
  void* bricks;               /* wcn_level_brick_bytes(n) bytes of scratch, 32-byte aligned */
  int32_t* order;             /* [n] slot -> row of the tile order; NULL: slots are rows */
  int32_t* nbr;               /* [27, n] 3x3x3 neighbour table, slots in tile order */
  int32_t* child;             /* [8, n] row of the level below at each 2x2x2 offset, -1 where none; NULL: not wanted */
  const int32_t* first_child; /* [n] of wcn_pyramid (child only) */
  const int32_t* rows_below;  /* [n_below, 4] (child only) */
  int64_t n_below;
  int64_t level;              /* 0..4 */
} wcn_level;

/* 3x3x3 maps in tile order and children tables of up to five levels, a launch per stage for all of them.  The rows must
 * be what wcn_pyramid called usable.  (nbr, order) is a pair for wcn_conv_fwd, child the [8, n] table of the 2x2x2
 * stride-2 convolution and of wcn_conv_rows_fwd on the way back up.
 * Tables of up to small_window_rows rows are ordered in windows of 4 096 rows, larger ones in windows of 16 384 (which
 * leave about 7 % fewer (tile, offset) pairs; one keeps a block busy for 25 us, a small one for 9).
 * Replaces generate_kernel_map per layer geometry (warpconvnet/geometry/coords/search/torch_discrete.py:365-466). */
int wcn_level_brick_bytes(int64_t n, int64_t* bytes);
int wcn_level_maps(const wcn_level* levels, int32_t num_levels, const int32_t* info, const int32_t* counts,
                   int32_t small_window_rows, void* stream);

/* ------------------------------------------------------------------ a network as one call */

/* One convolution of wcn_net_run: columns [src_col, src_col + c_in) of buffer src to columns [dst_col, ..) of buffer dst,
 * + columns [res_col, ..) of buffer res (res < 0: none). */
typedef struct {
  int32_t kind;        /* 0: wcn_conv_fwd over table `table`; 1: wcn_conv_rows_fwd, dst_rows = nbr of `table` (-1: identity) */
  int32_t table;
  int32_t level_in, level_out;
  int32_t num_offsets, c_in, c_out, c_out_packed, relu;
  int32_t src, src_col, dst, dst_col, res, res_col;
  int32_t reserved;
  const void* weight;
  const void* packed;
  const float* scale;
  const float* shift;
} wcn_net_op;
typedef struct { void* data; int64_t ld; } wcn_net_buffer;                       /* rows of ld elements */
typedef struct { const int32_t* nbr; const int32_t* out_rows; } wcn_net_table;

/* Enqueues the convolutions in order, all tensors of one 16-bit dtype; `rows` are the row counts per level.  Weights,
 * scales and tables must have been written before the call (its launches overlap and read them early).  The reference runs the same layers from Python, one module at a time
 * (warpconvnet/nn/modules/sequential.py:14-62, examples/mink_unet.py:212-413). */
int wcn_net_run(const wcn_net_op* ops, int32_t num_ops, const int64_t* rows, const wcn_net_buffer* buffers,
                const wcn_net_table* tables, int dtype, int32_t* dev_status, void* stream);

/* sums[j] = sum of column j of x [n, channels] (contiguous 16-byte aligned rows that are whole 16-byte pieces, 4096 bytes at
 * most; fp32 sums, the same bits on every run): the gradient of a layer's bias.  workspace: the bytes that the query gives
 * (0: not taken).  Stands for the reduction that autograd makes of sparse_conv.py:1794-1795. */
int wcn_column_sums_workspace_bytes(int64_t n, int32_t channels, int dtype, int64_t* bytes);
int wcn_column_sums(const void* x, int64_t n, int32_t channels, int dtype, float* sums, void* workspace, void* stream);

/* ------------------------------------------------------------------ batch normalisation in training */

/* y = relu(batch_norm(x) + residual) of [n, channels] rows (residual, relu optional), rounded to the dtype after the
 * normalisation and after the addition.  mean / rstd [channels] are left for the backward pass; running_mean / running_var
 * (may be NULL) and *num_batches (may be NULL) are updated as nn.BatchNorm1d does with a momentum.  eps and momentum are
 * given as the bits of a float.  `counter`: one zero word, zero again afterwards (one per stream).
 * backward: dx (may be NULL) and, with a residual behind a ReLU, its gradient; sums [2, channels] = d beta, d gamma;
 * y: the forward's result where a residual was added, else NULL.
 * WCN_ERR_UNSUPPORTED_CONFIG: n < 2, more than 1024 channels, or rows that are no whole number of 16-byte pieces.
 * Stands for the nn.BatchNorm1d / addition / nn.ReLU chain of examples/mink_unet.py:36-47, 129-141. */
int wcn_batch_norm_workspace_bytes(int64_t n, int32_t channels, int dtype, int64_t* bytes);
int wcn_batch_norm_train(const void* x, int64_t n, int32_t channels, int dtype, const float* gamma, const float* beta,
                         uint32_t eps_bits, uint32_t momentum_bits, float* running_mean, float* running_var,
                         int64_t* num_batches, const void* residual, int relu, void* y, float* mean, float* rstd,
                         void* workspace, uint32_t* counter, void* stream);
int wcn_batch_norm_backward(const void* x, const void* dy, const void* y, int64_t n, int32_t channels, int dtype,
                            const float* gamma, const float* beta, const float* mean, const float* rstd, int relu, void* dx,
                            void* dresidual, float* sums, void* workspace, uint32_t* counter, void* stream);

/* ------------------------------------------------------------------ self test */

/* Checks the library's bounded device-side waits: launches one small kernel that waits, with a
 * limit of `limit_cycles` SM clock cycles (1e3 .. 2e9), for a barrier phase that nothing can
 * complete.  The wait must give up, store WCN_ERR_WAIT_EXPIRED in dev_status and let the kernel
 * end normally; gave_up (device int32, may be NULL) receives 1 when it did.  The context stays
 * usable.  No counterpart in the reference (its kernels have no device-side waits). */
int wcn_selftest_bounded_wait(int64_t limit_cycles, int32_t* dev_status, int32_t* gave_up, void* stream);

#ifdef __cplusplus
}
#endif
#endif /* WCN_B200_H_ */
