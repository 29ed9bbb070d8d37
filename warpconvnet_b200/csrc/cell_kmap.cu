// Kernel maps of coordinate sets in any row order through a table of 4x4x4 cells.
//
// A voxel-keyed hash table answers one window position per probe: 14 to 27 dependent random reads per query, bound by
// the latency and sector rate of L2.  Here the table has one 32-byte entry per occupied 4x4x4 cell (key, 64-bit occupancy
// mask, number of the cell) and the rows of its voxels in 64 consecutive words, so a window touches at most 2x2x2
// entries, whose masks say which positions exist, and then reads only the rows of those: for a room scan 3.4 entries and
// 9.8 rows (a few 32-byte sectors) instead of 27 probes.  Rows need no order; repeated voxels resolve to the smallest row.
//
// Built in three light passes over the keys: claim the cells, set the mask bits and store the rows, and - only if some
// voxel occurred twice, which the second pass notices - take the smallest row of each.
// Measured (1 M room voxels in random order, 3x3x3): build 10 + 22 + 24 us, search 96 us with its hit counts; the voxel
// table took 54 us, its mirrored search 235 us and the counts 80 us.
#include "wcn_common.cuh"

namespace {

constexpr int THREADS = 256;

struct __align__(32) Cell {
  int4 key;                  // (batch, cell x, y, z); key.x == WCN_EMPTY_BATCH: empty
  unsigned long long mask;   // bit p set: the voxel at position p exists
  int32_t id;                // its rows are rows[64 * id ..]
  int32_t pad;
};

struct __align__(32) CellHeader {
  int32_t cells;             // cells claimed so far
  int32_t repeated;          // some voxel occurs more than once
  int32_t pad[6];
};

__host__ __device__ inline int64_t cell_cap(int64_t n) { return n * 2 > 64 ? n * 2 : 64; }

__device__ __forceinline__ uint32_t cell_pos(int x, int y, int z) {
  return (uint32_t)((x & 1) | ((y & 1) << 1) | ((z & 1) << 2) | ((x & 2) << 2) | ((y & 2) << 3) | ((z & 2) << 4));
}
__device__ __forceinline__ int4 cell_of(int4 c) { return make_int4(c.x, c.y >> 2, c.z >> 2, c.w >> 2); }  // arithmetic shift = floor
__device__ __forceinline__ uint32_t home(int4 key, uint32_t cap) { return wcn_slot(wcn_hash4<WCN_HASH_CITY>(key), cap); }

__global__ void cell_clear_kernel(CellHeader* hdr, Cell* cells, int64_t cap) {
  const int64_t i = (int64_t)blockIdx.x * THREADS + threadIdx.x;
  if (i < cap) {
    reinterpret_cast<int4*>(cells + i)[0] = make_int4(WCN_EMPTY_BATCH, 0, 0, 0);
    reinterpret_cast<int4*>(cells + i)[1] = make_int4(0, 0, 0, 0);
  }
  if (i == 0) hdr->cells = hdr->repeated = 0;
}

// Claim the cell of every row.  The claims of a warp take consecutive numbers from one atomic.
__global__ void cell_claim_kernel(const int4* __restrict__ keys, int64_t n, CellHeader* hdr, Cell* cells, uint32_t cap) {
  const int64_t i = (int64_t)blockIdx.x * THREADS + threadIdx.x;
  const int lane = threadIdx.x & 31;
  uint32_t mine = 0xFFFFFFFFu;
  if (i < n) {
    const int4 me = cell_of(__ldg(&keys[i]));
    uint32_t slot = home(me, cap);
    for (uint32_t probe = 0; probe < cap; ++probe) {
      int4* kp = &cells[slot].key;
      int4 cur = __ldcg(kp);
      if (cur.x == WCN_EMPTY_BATCH) {
        const unsigned long long clo = (uint32_t)WCN_EMPTY_BATCH;
        const unsigned long long vlo = ((unsigned long long)(uint32_t)me.y << 32) | (uint32_t)me.x;
        const unsigned long long vhi = ((unsigned long long)(uint32_t)me.w << 32) | (uint32_t)me.z;
        unsigned long long olo, ohi;
        asm volatile(
            "{\n\t.reg .b128 c, v, o;\n\t"
            "mov.b128 c, {%2, %3};\n\tmov.b128 v, {%4, %5};\n\t"
            "atom.global.relaxed.gpu.cas.b128 o, [%6], c, v;\n\t"
            "mov.b128 {%0, %1}, o;\n\t}"
            : "=l"(olo), "=l"(ohi)
            : "l"(clo), "l"(0ull), "l"(vlo), "l"(vhi), "l"(kp)
            : "memory");
        cur = make_int4((int)(uint32_t)olo, (int)(uint32_t)(olo >> 32), (int)(uint32_t)ohi, (int)(uint32_t)(ohi >> 32));
        if (cur.x == WCN_EMPTY_BATCH) { mine = slot; break; }
      }
      if (wcn_key_eq(cur, me)) break;
      slot = slot + 1 == cap ? 0u : slot + 1;
    }
  }
  const uint32_t claims = __ballot_sync(0xFFFFFFFFu, mine != 0xFFFFFFFFu);
  if (claims) {
    const int leader = __ffs(claims) - 1;
    int first = 0;
    if (lane == leader) first = atomicAdd(&hdr->cells, __popc(claims));
    first = __shfl_sync(0xFFFFFFFFu, first, leader);
    if (mine != 0xFFFFFFFFu) cells[mine].id = first + __popc(claims & ((1u << lane) - 1u));
  }
}

__device__ __forceinline__ const Cell* find(const Cell* __restrict__ cells, uint32_t cap, int4 key) {
  uint32_t slot = home(key, cap);
  for (uint32_t probe = 0; probe < cap; ++probe) {
    const int4 k = __ldg(&cells[slot].key);
    if (k.x == WCN_EMPTY_BATCH) return nullptr;
    if (wcn_key_eq(k, key)) return cells + slot;
    slot = slot + 1 == cap ? 0u : slot + 1;
  }
  return nullptr;
}

__global__ void cell_fill_kernel(const int4* __restrict__ keys, int64_t n, CellHeader* hdr, Cell* cells, uint32_t cap,
                                 int32_t* __restrict__ rows) {
  const int64_t i = (int64_t)blockIdx.x * THREADS + threadIdx.x;
  if (i >= n) return;
  const int4 c = __ldg(&keys[i]);
  Cell* cell = const_cast<Cell*>(find(cells, cap, cell_of(c)));
  if (!cell) return;
  const uint32_t p = cell_pos(c.y & 3, c.z & 3, c.w & 3);
  const unsigned long long old = atomicOr(&cell->mask, 1ull << p);
  if ((old >> p) & 1ull) hdr->repeated = 1;
  else rows[(int64_t)cell->id * 64 + p] = (int32_t)i;
}

__global__ void cell_smallest_kernel(const int4* __restrict__ keys, int64_t n, const CellHeader* __restrict__ hdr,
                                     const Cell* __restrict__ cells, uint32_t cap, int32_t* rows) {
  if (__ldg(&hdr->repeated) == 0) return;
  for (int64_t i = (int64_t)blockIdx.x * THREADS + threadIdx.x; i < n; i += (int64_t)gridDim.x * THREADS) {
    const int4 c = __ldg(&keys[i]);
    const Cell* cell = find(cells, cap, cell_of(c));
    if (cell) atomicMin(&rows[(int64_t)cell->id * 64 + cell_pos(c.y & 3, c.z & 3, c.w & 3)], (int32_t)i);
  }
}

// One thread per query.  KS: the window's width when it is the same along the axes and known at compile time (2 or 3).
template <int KS>
__global__ void __launch_bounds__(THREADS)
kmap_search_cells_kernel(const Cell* __restrict__ cells, uint32_t cap, const int32_t* __restrict__ rows,
                         const int4* __restrict__ queries, int64_t M, int sx, int sy, int sz, int kx_, int ky_, int kz_,
                         int32_t* __restrict__ nbr, int* __restrict__ block_counts) {
  __shared__ unsigned long long s_mask[8][THREADS];
  __shared__ int s_id[8][THREADS];
  __shared__ int s_count[64];
  const int kx = KS ? KS : kx_, ky = KS ? KS : ky_, kz = KS ? KS : kz_;
  const int tid = threadIdx.x, lane = tid & 31;
  const int64_t m = (int64_t)blockIdx.x * THREADS + tid;
  const bool live = m < M;
  if (block_counts) {
    if (tid < 64) s_count[tid] = 0;
    __syncthreads();
  }
  int rx = 0, ry = 0, rz = 0;
  if (live) {
    const int4 q = __ldg(&queries[m]);
    rx = q.y * sx - ((kx & 1) ? kx / 2 : 0);
    ry = q.z * sy - ((ky & 1) ? ky / 2 : 0);
    rz = q.w * sz - ((kz & 1) ? kz / 2 : 0);
    const int bx = rx >> 2, by = ry >> 2, bz = rz >> 2;
    const bool two_x = ((rx + kx - 1) >> 2) != bx, two_y = ((ry + ky - 1) >> 2) != by, two_z = ((rz + kz - 1) >> 2) != bz;
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const int ix = t & 1, iy = (t >> 1) & 1, iz = t >> 2;
      unsigned long long mk = 0ull;
      int id = 0;
      if ((!ix || two_x) && (!iy || two_y) && (!iz || two_z)) {
        const int4 key = make_int4(q.x, bx + ix, by + iy, bz + iz);
        uint32_t slot = home(key, cap);
        for (uint32_t probe = 0; probe < cap; ++probe) {
          const int4* e = reinterpret_cast<const int4*>(cells + slot);
          const int4 k = __ldg(e), d = __ldg(e + 1);  // both halves of the entry together
          if (k.x == WCN_EMPTY_BATCH) break;
          if (wcn_key_eq(k, key)) {
            mk = ((unsigned long long)(uint32_t)d.y << 32) | (uint32_t)d.x;
            id = d.z;
            break;
          }
          slot = slot + 1 == cap ? 0u : slot + 1;
        }
      }
      s_mask[t][tid] = mk;
      s_id[t][tid] = id;
    }
  }
  const int bx = rx >> 2, by = ry >> 2, bz = rz >> 2;
  int32_t* dst = nbr + m;
  int k = 0;
#pragma unroll
  for (int i = 0; i < kx; ++i) {
    const int x = rx + i, tx = (x >> 2) != bx;
    const uint32_t px = cell_pos(x & 3, 0, 0);
#pragma unroll
    for (int j = 0; j < ky; ++j) {
      const int y = ry + j, txy = tx | (((y >> 2) != by) << 1);
      const uint32_t pxy = px | cell_pos(0, y & 3, 0);
#pragma unroll
      for (int l = 0; l < kz; ++l, dst += M, ++k) {
        const int z = rz + l, t = txy | (((z >> 2) != bz) << 2);
        const uint32_t p = pxy | cell_pos(0, 0, z & 3);
        int found = -1;
        if (live && ((s_mask[t][tid] >> p) & 1ull)) found = __ldg(&rows[(int64_t)s_id[t][tid] * 64 + p]);
        if (live) *dst = found;
        if (block_counts) {
          const uint32_t have = __ballot_sync(0xFFFFFFFFu, found >= 0);
          if (lane == 0 && have) atomicAdd(&s_count[k], __popc(have));
        }
      }
    }
  }
  if (block_counts) {
    __syncthreads();
    for (int c = tid; c < kx * ky * kz; c += THREADS) block_counts[(int64_t)c * gridDim.x + blockIdx.x] = s_count[c];
  }
}

// Distinct rows per batch item, item counts into hist[items].
__global__ void batch_count_kernel(const int4* __restrict__ rows, const int* __restrict__ total, int items, int* __restrict__ hist) {
  const int n = *total;
  for (int i0 = blockIdx.x * THREADS; i0 < n; i0 += gridDim.x * THREADS) {
    const int i = i0 + threadIdx.x;
    int b = -1;
    if (i < n) {
      b = __ldg(&rows[i]).x;
      if (b < 0 || b >= items) b = items;  // counted apart: the caller takes another path
    }
    const uint32_t same = __match_any_sync(0xFFFFFFFFu, b);
    if (b >= 0 && (int)(threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(&hist[b], __popc(same));
  }
}

__global__ void publish_kernel(const int* __restrict__ total, const int* __restrict__ hist, int n, const int32_t* dev_status, int32_t* host) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) host[2 + i] = hist[i];
  if (threadIdx.x == 0) {
    host[0] = *total;
    host[1] = *(volatile const int32_t*)dev_status;
  }
}

inline unsigned blocks_for(int64_t n) { return (unsigned)((n + THREADS - 1) / THREADS); }

}  // namespace

extern "C" int wcn_cells_bytes(int64_t n, int64_t* bytes) {
  if (n < 0 || !bytes) return WCN_ERR_INVALID_PARAMETERS;
  *bytes = (int64_t)sizeof(CellHeader) + cell_cap(n) * (int64_t)sizeof(Cell) + n * 64 * (int64_t)sizeof(int32_t);
  return WCN_OK;
}

extern "C" int wcn_cells_build(const int32_t* keys, int64_t n, void* table, void* stream) {
  if (!table || n < 0 || n >= 0x3FFFFFFFll || (n > 0 && !keys)) return WCN_ERR_INVALID_PARAMETERS;
  if ((reinterpret_cast<uintptr_t>(table) & 31) || (reinterpret_cast<uintptr_t>(keys) & 15)) return WCN_ERR_INVALID_PARAMETERS;
  cudaStream_t st = wcn_stream(stream);
  CellHeader* hdr = reinterpret_cast<CellHeader*>(table);
  Cell* cells = reinterpret_cast<Cell*>(hdr + 1);
  const int64_t cap = cell_cap(n);
  int32_t* rows = reinterpret_cast<int32_t*>(cells + cap);
  const int4* k4 = reinterpret_cast<const int4*>(keys);
  cell_clear_kernel<<<blocks_for(cap), THREADS, 0, st>>>(hdr, cells, cap);
  if (n > 0) {
    cell_claim_kernel<<<blocks_for(n), THREADS, 0, st>>>(k4, n, hdr, cells, (uint32_t)cap);
    cell_fill_kernel<<<blocks_for(n), THREADS, 0, st>>>(k4, n, hdr, cells, (uint32_t)cap, rows);
    const unsigned most = (unsigned)wcn_num_sms() * 8;
    cell_smallest_kernel<<<blocks_for(n) < most ? blocks_for(n) : most, THREADS, 0, st>>>(k4, n, hdr, cells, (uint32_t)cap, rows);
  }
  WCN_CHECK_LAUNCH();
  return WCN_OK;
}

extern "C" int wcn_kmap_search_cells(const void* table, int64_t n, const int32_t* queries, int64_t num_queries,
                                     const int32_t* stride, const int32_t* kernel_size, int32_t* nbr, void* workspace,
                                     void* stream) {
  if (!table || !kernel_size || n < 0 || num_queries < 0) return WCN_ERR_INVALID_PARAMETERS;
  int sx = 1, sy = 1, sz = 1;
  if (stride) { sx = stride[0]; sy = stride[1]; sz = stride[2]; }
  const int kx = kernel_size[0], ky = kernel_size[1], kz = kernel_size[2];
  if (sx <= 0 || sy <= 0 || sz <= 0 || kx <= 0 || ky <= 0 || kz <= 0) return WCN_ERR_INVALID_PARAMETERS;
  if (kx > 4 || ky > 4 || kz > 4) return WCN_ERR_UNSUPPORTED_CONFIG;  // a wider window spans three cells
  if (num_queries == 0) return WCN_OK;
  if (!queries || !nbr || (reinterpret_cast<uintptr_t>(queries) & 15) || (reinterpret_cast<uintptr_t>(table) & 31))
    return WCN_ERR_INVALID_PARAMETERS;
  const Cell* cells = reinterpret_cast<const Cell*>(reinterpret_cast<const CellHeader*>(table) + 1);
  const int64_t cap = cell_cap(n);
  const int32_t* rows = reinterpret_cast<const int32_t*>(cells + cap);
  cudaStream_t st = wcn_stream(stream);
  const int ks = (kx == ky && ky == kz && (kx == 2 || kx == 3)) ? kx : 0;
#define WCN_CELLS_LAUNCH(KS)                                                                                             \
  kmap_search_cells_kernel<KS><<<blocks_for(num_queries), THREADS, 0, st>>>(cells, (uint32_t)cap, rows,                  \
                                                                           reinterpret_cast<const int4*>(queries), num_queries, \
                                                                           sx, sy, sz, kx, ky, kz, nbr, (int*)workspace)
  if (ks == 3) WCN_CELLS_LAUNCH(3);
  else if (ks == 2) WCN_CELLS_LAUNCH(2);
  else WCN_CELLS_LAUNCH(0);
#undef WCN_CELLS_LAUNCH
  WCN_CHECK_LAUNCH();
  return WCN_OK;
}

extern "C" int wcn_unique_counts(const int32_t* rows, int64_t n, const void* workspace, int32_t items, int32_t* hist,
                                 int32_t* host, const int32_t* dev_status, void* stream) {
  if (!workspace || !hist || !host || !dev_status || n <= 0 || items < 1 || !rows) return WCN_ERR_INVALID_PARAMETERS;
  const int* total = wcn_unique_total(workspace, n);
  cudaStream_t st = wcn_stream(stream);
  if (cudaMemsetAsync(hist, 0, (size_t)(items + 1) * sizeof(int), st) != cudaSuccess) return WCN_ERR_EXECUTION;
  const unsigned most = (unsigned)wcn_num_sms() * 4;
  batch_count_kernel<<<blocks_for(n) < most ? blocks_for(n) : most, THREADS, 0, st>>>(reinterpret_cast<const int4*>(rows), total, items, hist);
  publish_kernel<<<1, THREADS, 0, st>>>(total, hist, items + 1, dev_status, host);
  WCN_CHECK_LAUNCH();
  return WCN_OK;
}
