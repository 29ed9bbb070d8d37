// Kernel maps of every level of a Morton-sorted coordinate pyramid at once: the 3x3x3 maps in tile order and the
// children of every coarse row (the 2x2x2 stride-2 maps).
//
// Level by level these are eight kernels each (brick table count / clear / insert, search, presence masks, window
// sort, permuted copy, stride-2 search), most of them a few microseconds of latency for the coarse levels; here each
// stage is one launch over all levels.  Two passes over memory are gone as well: the sort key of a row is computed by
// a first walk over the bricks that stores nothing else, and the table is written once, in tile order, by a second
// walk in that order (before: table written, read for the masks, read and written again permuted).  A coarse row's
// children are the consecutive rows that start at its first child: no search.
//
// The caller vouches that the rows of every level are distinct and in Morton order about the corner (the pyramid kernel
// has checked it); with other rows the tables are wrong, but every access stays in bounds.
#include "tile_order.cuh"
#include "wcn_common.cuh"

namespace {

constexpr int THREADS = 256;
constexpr int MAX_LEVELS = 5;

struct __align__(32) Brick {
  int4 key;                  // (batch, brick x, y, z about the corner); key.x == WCN_EMPTY_BATCH: empty
  unsigned long long mask;   // bit p set: the voxel at position p of the brick exists
  int32_t base;              // row of the brick's first voxel
  int32_t pad;
};

struct Level {
  const int4* rows;
  int n;
  Brick* bricks;
  uint32_t cap_max;
  int32_t* order;            // sort keys, then slot -> row (null: rows in their own order)
  int32_t* nbr;              // [27][n]
  int32_t* child;            // [8][n] rows of the level below (null: none)
  const int32_t* first_child;
  const int4* rows_below;
  int n_below;
  int shift;                 // level number: the corner is shifted by it, bricks are counts[shift + 2]
};

struct LevelsParams {
  Level level[MAX_LEVELS];
  const int32_t* info;       // corner of level 0
  const int32_t* counts;     // distinct cells per shift
};

// Position of a voxel inside its brick = the low six bits of its Morton code (x in bit 0).
__device__ __forceinline__ uint32_t brick_pos(int x, int y, int z) {
  return (uint32_t)((x & 1) | ((y & 1) << 1) | ((z & 1) << 2) | ((x & 2) << 2) | ((y & 2) << 3) | ((z & 2) << 4));
}

__device__ __forceinline__ uint32_t used_slots(const LevelsParams& p, const Level& v) {
  const uint32_t want = max(64u, (uint32_t)__ldg(&p.counts[v.shift + 2]) * 4u);  // a quarter full at most
  return min(want, v.cap_max);
}

__device__ __forceinline__ uint32_t home_slot(int4 key, uint32_t cap) { return wcn_slot(wcn_hash4<WCN_HASH_CITY>(key), cap); }

struct Corner { int x, y, z; };
__device__ __forceinline__ Corner corner_of(const LevelsParams& p, const Level& v) {
  return {__ldg(&p.info[0]) >> v.shift, __ldg(&p.info[1]) >> v.shift, __ldg(&p.info[2]) >> v.shift};
}
__device__ __forceinline__ int4 brick_of(int4 c, const Corner& o) {
  return make_int4(c.x, (c.y - o.x) >> 2, (c.z - o.y) >> 2, (c.w - o.z) >> 2);
}

__global__ void level_clear_kernel(const LevelsParams p) {
  const Level& v = p.level[blockIdx.y];
  const uint32_t cap = used_slots(p, v);
  for (uint32_t i = blockIdx.x * THREADS + threadIdx.x; i < cap; i += gridDim.x * THREADS)
    v.bricks[i].key = make_int4(WCN_EMPTY_BATCH, 0, 0, 0);
}

// The first row of every brick collects the positions of its run, eight rows in flight, and inserts the brick.
__global__ void level_insert_kernel(const LevelsParams p) {
  const Level& v = p.level[blockIdx.y];
  const int i = blockIdx.x * THREADS + threadIdx.x;
  if (i >= v.n) return;
  const Corner o = corner_of(p, v);
  const int4 me = brick_of(__ldg(&v.rows[i]), o);
  if (i > 0 && wcn_key_eq(me, brick_of(__ldg(&v.rows[i - 1]), o))) return;
  unsigned long long mask = 0;
  bool more = true;
  for (int j0 = i; more && j0 < v.n && j0 < i + 64; j0 += 8) {
    int4 c[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) c[u] = __ldg(&v.rows[min(j0 + u, v.n - 1)]);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      more = more && j0 + u < v.n && wcn_key_eq(me, brick_of(c[u], o));
      if (more) mask |= 1ull << brick_pos((c[u].y - o.x) & 3, (c[u].z - o.y) & 3, (c[u].w - o.z) & 3);
    }
  }
  const uint32_t cap = used_slots(p, v);
  uint32_t slot = home_slot(me, cap);
  for (uint32_t probe = 0; probe < cap; ++probe) {
    int4* kp = &v.bricks[slot].key;
    unsigned long long olo = 0, ohi;
    if (__ldcg(kp).x == WCN_EMPTY_BATCH) {
      const unsigned long long clo = (uint32_t)WCN_EMPTY_BATCH;
      const unsigned long long vlo = ((unsigned long long)(uint32_t)me.y << 32) | (uint32_t)me.x;
      const unsigned long long vhi = ((unsigned long long)(uint32_t)me.w << 32) | (uint32_t)me.z;
      asm volatile(
          "{\n\t.reg .b128 c, v, o;\n\t"
          "mov.b128 c, {%2, %3};\n\tmov.b128 v, {%4, %5};\n\t"
          "atom.global.relaxed.gpu.cas.b128 o, [%6], c, v;\n\t"
          "mov.b128 {%0, %1}, o;\n\t}"
          : "=l"(olo), "=l"(ohi)
          : "l"(clo), "l"(0ull), "l"(vlo), "l"(vhi), "l"(kp)
          : "memory");
      if (olo == clo && ohi == 0) {  // claimed: this thread alone writes the rest of the entry
        v.bricks[slot].mask = mask;
        v.bricks[slot].base = i;
        return;
      }
    }
    slot = slot + 1 == cap ? 0u : slot + 1;
  }
}

// The up to 2 x 2 x 2 bricks a 3x3x3 window around a row touches, in shared memory (indexed at run time).
struct Window {
  unsigned long long (*mask)[THREADS];
  int (*base)[THREADS];
  int rx, ry, rz;  // first position of the window about the corner
};

__device__ __forceinline__ void fetch_window(const Level& v, const Corner& o, uint32_t cap, int4 q, Window& w) {
  w.rx = q.y - 1 - o.x; w.ry = q.z - 1 - o.y; w.rz = q.w - 1 - o.z;
  const int bx = w.rx >> 2, by = w.ry >> 2, bz = w.rz >> 2;
  const bool two_x = ((w.rx + 2) >> 2) > bx, two_y = ((w.ry + 2) >> 2) > by, two_z = ((w.rz + 2) >> 2) > bz;
#pragma unroll
  for (int t = 0; t < 8; ++t) {
    const int ix = t & 1, iy = (t >> 1) & 1, iz = t >> 2;
    unsigned long long mk = 0ull;
    int bs = 0;
    if ((!ix || two_x) && (!iy || two_y) && (!iz || two_z)) {
      const int4 key = make_int4(q.x, bx + ix, by + iy, bz + iz);
      uint32_t slot = home_slot(key, cap);
      for (uint32_t probe = 0; probe < cap; ++probe) {
        const int4* e = reinterpret_cast<const int4*>(v.bricks + slot);
        const int4 k = __ldg(e), d = __ldg(e + 1);
        if (k.x == WCN_EMPTY_BATCH) break;
        if (wcn_key_eq(k, key)) {
          mk = ((unsigned long long)(uint32_t)d.y << 32) | (uint32_t)d.x;
          bs = d.z;
          break;
        }
        slot = slot + 1 == cap ? 0u : slot + 1;
      }
    }
    w.mask[t][threadIdx.x] = mk;
    w.base[t][threadIdx.x] = bs;
  }
}

// Calls f(k, brick, position, mask) for every offset k of the window.
template <typename F> __device__ __forceinline__ void each_offset(const Window& w, F f) {
  const int bx = w.rx >> 2, by = w.ry >> 2, bz = w.rz >> 2;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const int x = w.rx + i, tx = (x >> 2) - bx;
    const uint32_t px = brick_pos(x & 3, 0, 0);
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const int y = w.ry + j, txy = tx | (((y >> 2) - by) << 1);
      const uint32_t pxy = px | brick_pos(0, y & 3, 0);
#pragma unroll
      for (int l = 0; l < 3; ++l) {
        const int z = w.rz + l, t = txy | (((z >> 2) - bz) << 2);
        f((i * 3 + j) * 3 + l, t, pxy | brick_pos(0, 0, z & 3), w.mask[t][threadIdx.x]);
      }
    }
  }
}

// Sort key of every row.
__global__ void __launch_bounds__(THREADS)
level_key_kernel(const LevelsParams p) {
  __shared__ unsigned long long s_mask[8][THREADS];
  __shared__ int s_base[8][THREADS];
  const Level& v = p.level[blockIdx.y];
  const int m = blockIdx.x * THREADS + threadIdx.x;
  if (m >= v.n || !v.order) return;
  Window w{s_mask, s_base, 0, 0, 0};
  fetch_window(v, corner_of(p, v), used_slots(p, v), __ldg(&v.rows[m]), w);
  uint32_t key = 0;
  each_offset(w, [&](int k, int, uint32_t pos, unsigned long long mk) { key |= (uint32_t)((mk >> pos) & 1ull) << presence_bit27(k); });
  v.order[m] = (int32_t)key;
}

// One block per window of every level.
template <int W>
__global__ void __launch_bounds__(kTileOrderThreads)
level_sort_kernel(const LevelsParams p, int window_min_rows, int window_max_rows) {
  extern __shared__ __align__(16) uint8_t sort_smem[];
  const Level& v = p.level[blockIdx.y];
  if (!v.order || v.n < window_min_rows || v.n > window_max_rows || (int64_t)blockIdx.x * W >= v.n) return;
  sort_window<W>(v.order, v.n, 27, blockIdx.x, sort_smem);
}

// nbr[k][s] = row of offset k around row order[s].
__global__ void __launch_bounds__(THREADS)
level_search_kernel(const LevelsParams p) {
  __shared__ unsigned long long s_mask[8][THREADS];
  __shared__ int s_base[8][THREADS];
  const Level& v = p.level[blockIdx.y];
  const int s = blockIdx.x * THREADS + threadIdx.x;
  if (s >= v.n) return;
  const int m = v.order ? __ldg(&v.order[s]) : s;
  Window w{s_mask, s_base, 0, 0, 0};
  fetch_window(v, corner_of(p, v), used_slots(p, v), __ldg(&v.rows[m]), w);
  int32_t* dst = v.nbr + s;
  const int64_t n = v.n;
  each_offset(w, [&](int k, int t, uint32_t pos, unsigned long long mk) {
    int found = -1;
    if ((mk >> pos) & 1ull) found = w.base[t][threadIdx.x] + __popcll(mk & ((1ull << pos) - 1ull));
    dst[k * n] = found;
  });
}

__global__ void level_child_kernel(const LevelsParams p) {
  const Level& v = p.level[blockIdx.y];
  const int j = blockIdx.x * THREADS + threadIdx.x;
  if (!v.child || j >= v.n) return;
  const int begin = __ldg(&v.first_child[j]), end = j + 1 < v.n ? __ldg(&v.first_child[j + 1]) : v.n_below;
  int rows[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) rows[k] = -1;
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const int r = begin + u;
    if (r < end && r < v.n_below) {
      const int4 c = __ldg(&v.rows_below[r]);
      const int k = ((c.y & 1) * 2 + (c.z & 1)) * 2 + (c.w & 1);
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (q == k) rows[q] = r;
    }
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) v.child[(int64_t)k * v.n + j] = rows[k];
}

template <int W> int launch_sort(const LevelsParams& p, int levels, int lo, int hi, int windows, cudaStream_t st) {
  static bool configured[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return WCN_ERR_INITIALIZATION;
  if (!configured[dev]) {
    if (cudaFuncSetAttribute(level_sort_kernel<W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sort_window_bytes<W>()) != cudaSuccess) {
      (void)cudaGetLastError();
      return WCN_ERR_INITIALIZATION;
    }
    configured[dev] = true;
  }
  level_sort_kernel<W><<<dim3((unsigned)windows, (unsigned)levels), kTileOrderThreads, sort_window_bytes<W>(), st>>>(p, lo, hi);
  return cudaGetLastError() == cudaSuccess ? WCN_OK : WCN_ERR_EXECUTION;
}

}  // namespace

extern "C" int wcn_level_brick_bytes(int64_t n, int64_t* bytes) {
  if (n < 0 || !bytes) return WCN_ERR_INVALID_PARAMETERS;
  *bytes = (n * 2 > 64 ? n * 2 : 64) * (int64_t)sizeof(Brick);
  return WCN_OK;
}

extern "C" int wcn_level_maps(const wcn_level* levels, int32_t num_levels, const int32_t* info, const int32_t* counts,
                              int32_t small_window_rows, void* stream) {
  if (!levels || num_levels < 1 || num_levels > MAX_LEVELS || !info || !counts || small_window_rows < 0) return WCN_ERR_INVALID_PARAMETERS;
  LevelsParams p = {};
  p.info = info; p.counts = counts;
  int64_t most = 0, small_windows = 0, large_windows = 0;
  bool tiled = false, children = false;
  for (int l = 0; l < num_levels; ++l) {
    const wcn_level& q = levels[l];
    Level& v = p.level[l];
    if (q.n <= 0 || q.n >= 0x3FFFFFFFll || !q.rows || !q.bricks || !q.nbr || q.level < 0 || q.level > 4 ||
        (reinterpret_cast<uintptr_t>(q.rows) & 15) || (reinterpret_cast<uintptr_t>(q.bricks) & 31) ||
        (q.child && (!q.first_child || !q.rows_below || q.n_below <= 0)))
      return WCN_ERR_INVALID_PARAMETERS;
    v.rows = reinterpret_cast<const int4*>(q.rows); v.n = (int)q.n;
    v.bricks = reinterpret_cast<Brick*>(q.bricks); v.cap_max = (uint32_t)(q.n * 2 > 64 ? q.n * 2 : 64);
    v.order = q.order; v.nbr = q.nbr; v.child = q.child; v.first_child = q.first_child;
    v.rows_below = reinterpret_cast<const int4*>(q.rows_below); v.n_below = (int)q.n_below; v.shift = q.level;
    most = q.n > most ? q.n : most;
    if (q.order) {
      tiled = true;
      if (q.n <= small_window_rows) small_windows = small_windows > (q.n + kTileWindowSmall - 1) / kTileWindowSmall ? small_windows : (q.n + kTileWindowSmall - 1) / kTileWindowSmall;
      else large_windows = large_windows > (q.n + kTileWindowLarge - 1) / kTileWindowLarge ? large_windows : (q.n + kTileWindowLarge - 1) / kTileWindowLarge;
    }
    children |= q.child != nullptr;
  }
  cudaStream_t st = wcn_stream(stream);
  const dim3 grid((unsigned)((most + THREADS - 1) / THREADS), (unsigned)num_levels);
  level_clear_kernel<<<grid, THREADS, 0, st>>>(p);
  level_insert_kernel<<<grid, THREADS, 0, st>>>(p);
  if (tiled) {
    level_key_kernel<<<grid, THREADS, 0, st>>>(p);
    int rc = WCN_OK;
    if (large_windows) rc = launch_sort<kTileWindowLarge>(p, num_levels, small_window_rows + 1, INT_MAX, (int)large_windows, st);
    if (rc == WCN_OK && small_windows) rc = launch_sort<kTileWindowSmall>(p, num_levels, 0, small_window_rows, (int)small_windows, st);
    if (rc != WCN_OK) return rc;
  }
  level_search_kernel<<<grid, THREADS, 0, st>>>(p);
  if (children) level_child_kernel<<<grid, THREADS, 0, st>>>(p);
  WCN_CHECK_LAUNCH();
  return WCN_OK;
}
