// Morton order of a batch of voxel sets, and the coordinates of the coarser levels of the sorted rows.
//
// Sort.  One cooperative kernel: per-axis minimum and maximum, codes, a least-significant-digit radix sort of
// (batch, code) by 8-bit digits, and in the last pass the sorted rows themselves.  As separate kernels (torch.min,
// codes, two argsorts of eight and one digit passes, three gathers) a 20 000-voxel scene spends 0.2 ms on launches
// and passes over constant digits; here the number of passes follows from the coordinates that are there, and a pass
// is two grid barriers.  A block owns a contiguous chunk of rows, a warp a contiguous part of it, so ranks from
// __match_any_sync in lane order make the sort stable.
//
// Coarser levels.  Rows sorted by Morton code about a corner that is a multiple of 2^s have the rows of every 2^s cell
// next to each other, so the distinct rows of floor(c / 2^s) are the rows whose predecessor lies in another cell: no
// hash table, and the first child of every coarse row comes with it.
#include "wcn_common.cuh"

namespace {

constexpr int SORT_THREADS = 1024, SORT_WARPS = SORT_THREADS / 32;
constexpr int SORT_PER_LANE = 8;                                   // rows a lane holds at a time
constexpr int SORT_TILE = SORT_THREADS * SORT_PER_LANE;            // rows a block ranks at a time
constexpr int SORT_MAX_BLOCKS = 592;
constexpr int SORT_MAX_BATCH = 255;
constexpr long long SORT_WAIT_CYCLES = 4000000000ll;

struct SortParams {
  const int32_t* coords;   // [n][3]
  int64_t n;
  int64_t* codes;          // [n], caller's row order
  int64_t* perm;           // [n], sorted row -> caller's row
  int4* rows;              // [n], sorted (batch, x, y, z)
  int32_t* info;           // [8]: corner x y z, bits per axis, 1 if every code is the whole position, status
  const char* feats;       // rows of feat_units * unit bytes, or null
  char* feats_sorted;
  int feat_units, unit;
  unsigned long long* keys[2];
  uint32_t* index[2];
  uint32_t* hist;          // [blocks][256]
  int32_t* bounds;         // [blocks][6]
  uint32_t* barrier;       // zeroed by the host
  int32_t* dev_status;
  int batches;
  int32_t offsets[SORT_MAX_BATCH + 1];
};

__device__ __forceinline__ unsigned long long spread3(unsigned long long n) {
  n &= 0x1FFFFFull;
  n = (n | (n << 32)) & 0x001F00000000FFFFull;
  n = (n | (n << 16)) & 0x001F0000FF0000FFull;
  n = (n | (n << 8)) & 0x100F00F00F00F00Full;
  n = (n | (n << 4)) & 0x10C30C30C30C30C3ull;
  n = (n | (n << 2)) & 0x1249249249249249ull;
  return n;
}

// All blocks of the (cooperatively launched) grid meet.  Bounded: false once a block gave up.
__device__ __forceinline__ bool grid_meet(uint32_t* counter, uint32_t round, int32_t* dev_status) {
  __shared__ int met;
  __syncthreads();
  if (threadIdx.x == 0) {
    met = 1;
    __threadfence();
    const uint32_t target = round * gridDim.x;
    if (atomicAdd(counter, 1u) + 1u < target) {
      const long long t0 = clock64();
      while (*(volatile uint32_t*)counter < target) {
        if (clock64() - t0 > SORT_WAIT_CYCLES) {
          atomicExch(dev_status, (int)WCN_ERR_WAIT_EXPIRED);
          met = 0;
          break;
        }
      }
    }
    __threadfence();
  }
  __syncthreads();
  return met != 0;
}

__device__ __forceinline__ int batch_of(const int32_t* offsets, int batches, int i) {
  int lo = 0, hi = batches;  // largest b with offsets[b] <= i
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (offsets[mid] <= i) lo = mid; else hi = mid;
  }
  return lo;
}

__global__ void __launch_bounds__(SORT_THREADS, 1)
morton_sort_kernel(const SortParams p) {
  __shared__ uint16_t cnt[SORT_WARPS][256];   // rows of a digit per warp, then their rank before the warp
  __shared__ uint32_t base[256];              // next output row of a digit
  __shared__ uint32_t total[256];
  __shared__ int32_t red[SORT_WARPS][6];
  __shared__ int32_t box[6];
  __shared__ int32_t offs[SORT_MAX_BATCH + 1];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, blk = blockIdx.x, blocks = gridDim.x;
  const int64_t chunk = ((p.n + blocks - 1) / blocks + 31) / 32 * 32;
  const int64_t lo = min(p.n, chunk * blk), hi = min(p.n, lo + chunk);
  uint32_t round = 0;
  for (int i = tid; i <= p.batches; i += SORT_THREADS) offs[i] = p.offsets[i];

  // ---- extent of the coordinates
  int32_t mn[3] = {INT_MAX, INT_MAX, INT_MAX}, mx[3] = {INT_MIN, INT_MIN, INT_MIN};
  for (int64_t i = lo + tid; i < hi; i += SORT_THREADS) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const int32_t v = __ldg(&p.coords[i * 3 + a]);
      mn[a] = min(mn[a], v);
      mx[a] = max(mx[a], v);
    }
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    mn[a] = __reduce_min_sync(0xFFFFFFFFu, mn[a]);
    mx[a] = __reduce_max_sync(0xFFFFFFFFu, mx[a]);
    if (lane == 0) { red[warp][a] = mn[a]; red[warp][3 + a] = mx[a]; }
  }
  __syncthreads();
  if (tid < 6) {
    int32_t v = red[0][tid];
    for (int w = 1; w < SORT_WARPS; ++w) v = tid < 3 ? min(v, red[w][tid]) : max(v, red[w][tid]);
    p.bounds[blk * 6 + tid] = v;
  }
  if (!grid_meet(p.barrier, ++round, p.dev_status)) return;
  if (warp < 6) {
    int32_t v = warp < 3 ? INT_MAX : INT_MIN;
    for (int b = lane; b < blocks; b += 32) {
      const int32_t u = __ldcg(&p.bounds[b * 6 + warp]);
      v = warp < 3 ? min(v, u) : max(v, u);
    }
    v = warp < 3 ? __reduce_min_sync(0xFFFFFFFFu, v) : __reduce_max_sync(0xFFFFFFFFu, v);
    if (lane == 0) box[warp] = v;
  }
  __syncthreads();
  // the corner the codes are taken from: the minimum rounded down to a multiple of 16
  const int ox = box[0] & ~15, oy = box[1] & ~15, oz = box[2] & ~15;
  const uint32_t span = max((uint32_t)(box[3] - ox), max((uint32_t)(box[4] - oy), (uint32_t)(box[5] - oz)));
  const bool whole = span < (1u << 21);               // else positions 2^21 apart share a code
  const int axis_bits = whole ? (span ? 32 - __clz((int)span) : 1) : 21;
  const int code_bits = 3 * axis_bits;
  const int batch_bits = p.batches > 1 ? 32 - __clz(p.batches - 1) : 0;
  // (batch, code) in one 64-bit key: with 63 code bits there is room for one batch bit; more batches than that are
  // ordered by the digits of the batch index alone, taken from the row index, after those of the code
  const int key_bits = code_bits + batch_bits <= 64 ? code_bits + batch_bits : code_bits;
  const int code_passes = (key_bits + 7) / 8;
  const int passes = code_passes + (key_bits == code_bits ? (batch_bits + 7) / 8 : 0);
  if (blk == 0 && tid == 0) {
    p.info[0] = ox; p.info[1] = oy; p.info[2] = oz; p.info[3] = axis_bits; p.info[4] = whole ? 1 : 0;
  }
  for (int64_t i = lo + tid; i < hi; i += SORT_THREADS) {
    const int32_t x = __ldg(&p.coords[i * 3]), y = __ldg(&p.coords[i * 3 + 1]), z = __ldg(&p.coords[i * 3 + 2]);
    const unsigned long long code = spread3((unsigned long long)(uint32_t)(x - ox)) |
                                    (spread3((unsigned long long)(uint32_t)(y - oy)) << 1) |
                                    (spread3((unsigned long long)(uint32_t)(z - oz)) << 2);
    p.codes[i] = (int64_t)code;
    unsigned long long key = code;
    if (key_bits > code_bits) key |= (unsigned long long)batch_of(offs, p.batches, (int)i) << code_bits;
    p.keys[0][i] = key;
  }
  __syncthreads();

  auto digit_of = [&](unsigned long long key, uint32_t idx, int pass) -> int {
    if (pass < code_passes) return (int)((key >> (8 * pass)) & 255u);
    return (batch_of(offs, p.batches, (int)idx) >> (8 * (pass - code_passes))) & 255;
  };

  for (int pass = 0; pass < passes; ++pass) {
    const unsigned long long* kin = p.keys[pass & 1];
    unsigned long long* kout = p.keys[(pass & 1) ^ 1];
    const uint32_t* iin = p.index[pass & 1];
    uint32_t* iout = p.index[(pass & 1) ^ 1];
    const bool last = pass == passes - 1;
    auto load = [&](int64_t i, unsigned long long& key, uint32_t& idx) {  // written by other blocks: not through L1
      key = __ldcg(&kin[i]);
      idx = pass ? __ldcg(&iin[i]) : (uint32_t)i;
    };
    // ---- rows of every digit in this block
    if (tid < 256) total[tid] = 0;
    __syncthreads();
    for (int64_t i0 = lo; i0 < hi; i0 += SORT_THREADS) {
      const int64_t i = i0 + tid;
      const bool live = i < hi;
      unsigned long long key = 0;
      uint32_t idx = 0;
      if (live) load(i, key, idx);
      const int d = live ? digit_of(key, idx, pass) : 256;
      const uint32_t same = __match_any_sync(0xFFFFFFFFu, d);
      if (live && lane == __ffs(same) - 1) atomicAdd(&total[d], (uint32_t)__popc(same));
    }
    __syncthreads();
    if (tid < 256) p.hist[blk * 256 + tid] = total[tid];
    if (!grid_meet(p.barrier, ++round, p.dev_status)) return;
    // ---- first output row of every digit of this block: four threads a digit, each every fourth block
    {
      const int d = tid & 255, part = tid >> 8;
      uint32_t before = 0, all = 0;
#pragma unroll 8
      for (int b = part; b < blocks; b += 4) {
        const uint32_t v = __ldcg(&p.hist[b * 256 + d]);
        all += v;
        if (b < blk) before += v;
      }
      if (tid < 256) { base[tid] = 0; total[tid] = 0; }
      __syncthreads();
      atomicAdd(&base[d], before);
      atomicAdd(&total[d], all);
      __syncthreads();
      if (warp == 0) {  // exclusive scan of the totals over the digits, eight per lane
        uint32_t v[8], sum = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) { v[j] = total[lane * 8 + j]; sum += v[j]; }
        uint32_t incl = sum;
#pragma unroll
        for (int s = 1; s < 32; s <<= 1) {
          const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, incl, s);
          if (lane >= s) incl += o;
        }
        uint32_t run = incl - sum;
#pragma unroll
        for (int j = 0; j < 8; ++j) { base[lane * 8 + j] += run; run += v[j]; }
      }
      __syncthreads();
    }
    // ---- scatter, SORT_TILE rows at a time; a warp ranks 32 * SORT_PER_LANE consecutive rows
    for (int64_t t0 = lo; t0 < hi; t0 += SORT_TILE) {
      for (int i = tid; i < SORT_WARPS * 256 / 2; i += SORT_THREADS) reinterpret_cast<uint32_t*>(&cnt[0][0])[i] = 0;
      __syncthreads();
      unsigned long long key[SORT_PER_LANE];
      uint32_t idx[SORT_PER_LANE];
      uint16_t rank[SORT_PER_LANE];
      // the tile is dealt to the warps evenly, so that a short tile still uses all of them
      const int64_t rows = min((int64_t)SORT_TILE, hi - t0);
      const int per_warp = (int)((rows + 32 * SORT_WARPS - 1) / (32 * SORT_WARPS)) * 32;
      const int64_t w0 = t0 + (int64_t)warp * per_warp;
      const int64_t w1 = min(hi, w0 + per_warp);
#pragma unroll
      for (int j = 0; j < SORT_PER_LANE; ++j) {
        const int64_t i = w0 + j * 32 + lane;
        key[j] = 0; idx[j] = 0;
        if (i < w1) load(i, key[j], idx[j]);
      }
#pragma unroll
      for (int j = 0; j < SORT_PER_LANE; ++j) {
        const bool live = w0 + j * 32 + lane < w1;
        const int d = live ? digit_of(key[j], idx[j], pass) : 256;
        const uint32_t same = __match_any_sync(0xFFFFFFFFu, d);
        const int leader = __ffs(same) - 1;
        uint32_t before = 0;
        if (live && lane == leader) {
          before = cnt[warp][d];
          cnt[warp][d] = (uint16_t)(before + __popc(same));
        }
        before = __shfl_sync(0xFFFFFFFFu, before, leader);
        rank[j] = (uint16_t)(before + __popc(same & ((1u << lane) - 1u)));
        __syncwarp();
      }
      __syncthreads();
      if (tid < 256) {  // rows of the digit in the warps before
        uint32_t run = 0;
#pragma unroll 8
        for (int w = 0; w < SORT_WARPS; ++w) {
          const uint32_t v = cnt[w][tid];
          cnt[w][tid] = (uint16_t)run;
          run += v;
        }
        total[tid] = run;
      }
      __syncthreads();
#pragma unroll
      for (int j = 0; j < SORT_PER_LANE; ++j) {
        if (w0 + j * 32 + lane >= w1) continue;
        const int d = digit_of(key[j], idx[j], pass);
        const int64_t to = (int64_t)base[d] + cnt[warp][d] + rank[j];
        if (!last) {
          kout[to] = key[j];
          iout[to] = idx[j];
        } else {
          const int64_t i = idx[j];
          p.perm[to] = i;
          p.rows[to] = make_int4(batch_of(offs, p.batches, (int)i), __ldg(&p.coords[i * 3]), __ldg(&p.coords[i * 3 + 1]),
                                 __ldg(&p.coords[i * 3 + 2]));
          if (p.feats) {
            if (p.unit == 4) {
              for (int u = 0; u < p.feat_units; ++u)
                reinterpret_cast<uint32_t*>(p.feats_sorted)[to * p.feat_units + u] =
                    __ldg(reinterpret_cast<const uint32_t*>(p.feats) + i * p.feat_units + u);
            } else {
              for (int u = 0; u < p.feat_units; ++u)
                reinterpret_cast<uint16_t*>(p.feats_sorted)[to * p.feat_units + u] =
                    __ldg(reinterpret_cast<const uint16_t*>(p.feats) + i * p.feat_units + u);
            }
          }
        }
      }
      __syncthreads();
      if (tid < 256) base[tid] += total[tid];
    }
    if (!last && !grid_meet(p.barrier, ++round, p.dev_status)) return;
  }
}

inline int sort_blocks(int64_t n) {
  int64_t b = (n + 2047) / 2048;  // at least two rows a lane
  const int sms = wcn_num_sms() < SORT_MAX_BLOCKS ? wcn_num_sms() : SORT_MAX_BLOCKS;
  return (int)(b < sms ? b : sms);
}

// ------------------------------------------------------------------ coarser levels

constexpr int PYR_THREADS = 256;
constexpr int PYR_SHIFTS = 6;   // cells of 2, 4, .., 64 voxels are counted

struct PyramidParams {
  int groups, per_block;   // groups of PYR_THREADS rows, and how many of them a block of the second kernel takes
  const int4* rows;         // [n] sorted
  const int32_t* info;      // of the sort: corner, ...
  int64_t n;
  int levels;               // strided levels to emit
  int32_t* block_counts;    // [PYR_SHIFTS][blocks]
  int32_t* counts;          // [24] device: rows per shift 0..6, 1 if two rows are equal, corners of the levels
  int4* out[4];             // [n] each: floor(row / 2^(l+1))
  int32_t* first[4];        // [n] each: first row of the level below
  int64_t* host;            // [levels][batches + 1] row offsets, then usable flag, status word (pinned host memory)
  const int32_t* dev_status;
  int batches;
  int32_t offsets[SORT_MAX_BATCH + 1];
};

// Highest differing coordinate bit between a row and its predecessor about the corner: the row starts a new cell at
// shift s when any bit from s up differs (or the batch does).
__device__ __forceinline__ uint32_t step_bits(const PyramidParams& p, int64_t i, int ox, int oy, int oz, int4* row) {
  const int4 c = __ldg(&p.rows[i]);
  *row = c;
  if (i == 0) return 0xFFFFFFFFu;
  const int4 q = __ldg(&p.rows[i - 1]);
  if (q.x != c.x) return 0xFFFFFFFFu;
  return ((uint32_t)(c.y - ox) ^ (uint32_t)(q.y - ox)) | ((uint32_t)(c.z - oy) ^ (uint32_t)(q.z - oy)) |
         ((uint32_t)(c.w - oz) ^ (uint32_t)(q.w - oz));
}

__global__ void __launch_bounds__(PYR_THREADS)
pyramid_count_kernel(const PyramidParams p) {
  const int64_t i = (int64_t)blockIdx.x * PYR_THREADS + threadIdx.x;
  const int ox = __ldg(&p.info[0]), oy = __ldg(&p.info[1]), oz = __ldg(&p.info[2]);
  int4 row;
  const uint32_t d = i < p.n ? step_bits(p, i, ox, oy, oz, &row) : 0u;
#pragma unroll
  for (int s = 1; s <= PYR_SHIFTS; ++s) {
    const int c = __syncthreads_count((d >> s) != 0);
    if (threadIdx.x == 0) p.block_counts[(s - 1) * gridDim.x + blockIdx.x] = c;
  }
  if (i < p.n && d == 0) p.counts[7] = 1;  // equal to the row before
}

// Every block adds up the counts of all groups of rows before its own, so large sets give a block several groups
// (`per_block`): 1.2 M rows, a group each: 64 us, four: 41, sixteen: 46.
__global__ void __launch_bounds__(PYR_THREADS)
pyramid_emit_kernel(const PyramidParams p) {
  constexpr int WARPS = PYR_THREADS / 32, PARTS = WARPS / PYR_SHIFTS > 0 ? WARPS / PYR_SHIFTS : 1;
  __shared__ int32_t before_s[PYR_SHIFTS], all_s[PYR_SHIFTS];
  __shared__ int32_t warp_c[PYR_SHIFTS][WARPS];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ox = __ldg(&p.info[0]), oy = __ldg(&p.info[1]), oz = __ldg(&p.info[2]);
  const int group0 = (int)blockIdx.x * p.per_block;
  if (tid < PYR_SHIFTS) before_s[tid] = all_s[tid] = 0;
  __syncthreads();
  for (int w = warp; w < PYR_SHIFTS * PARTS; w += WARPS) {
    const int s = w / PARTS, part = w % PARTS;
    int before = 0, all = 0;
#pragma unroll 4
    for (int b = part * 32 + lane; b < p.groups; b += 32 * PARTS) {
      const int v = __ldg(&p.block_counts[s * p.groups + b]);
      all += v;
      if (b < group0) before += v;
    }
    before = __reduce_add_sync(0xFFFFFFFFu, before);
    all = __reduce_add_sync(0xFFFFFFFFu, all);
    if (lane == 0) { atomicAdd(&before_s[s], before); atomicAdd(&all_s[s], all); }
  }
  for (int q = 0; q < p.per_block && group0 + q < p.groups; ++q) {
    const int64_t i = (int64_t)(group0 + q) * PYR_THREADS + tid;
    int4 row = make_int4(0, 0, 0, 0);
    const bool live = i < p.n;
    const uint32_t d = live ? step_bits(p, i, ox, oy, oz, &row) : 0u;
    uint32_t heads[PYR_SHIFTS];
#pragma unroll
    for (int s = 0; s < PYR_SHIFTS; ++s) {
      heads[s] = __ballot_sync(0xFFFFFFFFu, (d >> (s + 1)) != 0);
      if (lane == 0) warp_c[s][warp] = __popc(heads[s]);
    }
    __syncthreads();
    int rank_below = (int)i;
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      if (l >= p.levels) break;
      int rank = before_s[l] + __popc(heads[l] & ((1u << lane) - 1u));
      for (int w = 0; w < warp; ++w) rank += warp_c[l][w];
      if (live && ((d >> (l + 1)) != 0)) {
        const int s = l + 1;
        p.out[l][rank] = make_int4(row.x, row.y >> s, row.z >> s, row.w >> s);
        p.first[l][rank] = rank_below;
        rank_below = rank;
      }
      if (live) {  // batch items start where their first row does (an empty one where the next does)
        const bool start = i == 0 || d == 0xFFFFFFFFu;
        if (start)
          for (int b = 0; b <= p.batches; ++b)
            if (p.offsets[b] == (int32_t)i) p.host[(int64_t)l * (p.batches + 1) + b] = rank;
      }
    }
    __syncthreads();
    if (tid < PYR_SHIFTS)
      for (int w = 0; w < WARPS; ++w) before_s[tid] += warp_c[tid][w];
    __syncthreads();
  }
  if (blockIdx.x == 0 && tid == 0) {
    p.counts[0] = (int32_t)p.n;
    for (int l = 0; l < p.levels; ++l) {
      p.counts[8 + 4 * l] = ox >> (l + 1); p.counts[9 + 4 * l] = oy >> (l + 1); p.counts[10 + 4 * l] = oz >> (l + 1);
    }
#pragma unroll
    for (int s = 0; s < PYR_SHIFTS; ++s) p.counts[s + 1] = all_s[s];
    for (int l = 0; l < p.levels; ++l)
      for (int b = 0; b <= p.batches; ++b)
        if (p.offsets[b] == (int32_t)p.n) p.host[(int64_t)l * (p.batches + 1) + b] = all_s[l];
    p.host[(int64_t)p.levels * (p.batches + 1)] = (p.counts[7] == 0 && __ldg(&p.info[4]) != 0) ? 1 : 0;
    p.host[(int64_t)p.levels * (p.batches + 1) + 1] = *(volatile const int32_t*)p.dev_status;
  }
}

}  // namespace

extern "C" int wcn_morton_sort_workspace_bytes(int64_t n, int64_t* bytes) {
  if (n < 0 || !bytes) return WCN_ERR_INVALID_PARAMETERS;
  *bytes = 24 * ((n + 31) / 32 * 32) + (int64_t)SORT_MAX_BLOCKS * (256 + 6) * 4 + 512;
  return WCN_OK;
}

extern "C" int wcn_morton_sort(const int32_t* coords, int64_t n, const int64_t* offsets, int32_t batches, int64_t* codes,
                               int64_t* perm, int32_t* rows, int32_t* info, const void* feats, void* feats_sorted,
                               int32_t feat_row_bytes, void* workspace, int32_t* dev_status, void* stream) {
  if (n < 0 || n >= 0x7FFFFFFFll || batches < 1 || !offsets) return WCN_ERR_INVALID_PARAMETERS;
  if (batches > SORT_MAX_BATCH) return WCN_ERR_UNSUPPORTED_CONFIG;
  if (n == 0) return WCN_OK;
  if (!coords || !codes || !perm || !rows || !info || !workspace || !dev_status || (reinterpret_cast<uintptr_t>(rows) & 15) ||
      (reinterpret_cast<uintptr_t>(workspace) & 15))
    return WCN_ERR_INVALID_PARAMETERS;
  if (feats && (!feats_sorted || feat_row_bytes <= 0 || feat_row_bytes % 2)) return WCN_ERR_INVALID_PARAMETERS;
  SortParams p;
  p.coords = coords; p.n = n; p.codes = codes; p.perm = perm; p.rows = reinterpret_cast<int4*>(rows); p.info = info;
  const bool words = feat_row_bytes % 4 == 0 && !(reinterpret_cast<uintptr_t>(feats) & 3) && !(reinterpret_cast<uintptr_t>(feats_sorted) & 3);
  p.feats = (const char*)feats; p.feats_sorted = (char*)feats_sorted; p.unit = words ? 4 : 2; p.feat_units = feat_row_bytes / p.unit;
  const int64_t padded = (n + 31) / 32 * 32;
  char* ws = (char*)workspace;
  p.barrier = (uint32_t*)ws;
  ws += 512;
  p.keys[0] = (unsigned long long*)ws; p.keys[1] = p.keys[0] + padded;
  p.index[0] = (uint32_t*)(p.keys[1] + padded); p.index[1] = p.index[0] + padded;
  p.hist = p.index[1] + padded;
  p.bounds = (int32_t*)(p.hist + SORT_MAX_BLOCKS * 256);
  p.dev_status = dev_status; p.batches = batches;
  for (int b = 0; b <= batches; ++b) {
    if (offsets[b] < 0 || offsets[b] > n) return WCN_ERR_INVALID_PARAMETERS;
    p.offsets[b] = (int32_t)offsets[b];
  }
  cudaStream_t st = wcn_stream(stream);
  if (cudaMemsetAsync(p.barrier, 0, 4, st) != cudaSuccess) return WCN_ERR_EXECUTION;
  void* args[] = {&p};
  // cooperative: the blocks meet at grid barriers, so they must all be resident (one per multiprocessor at most)
  if (cudaLaunchCooperativeKernel((const void*)morton_sort_kernel, dim3((unsigned)sort_blocks(n)), dim3(SORT_THREADS), args, 0, st) != cudaSuccess) {
    (void)cudaGetLastError();
    return WCN_ERR_EXECUTION;
  }
  return WCN_OK;
}

extern "C" int wcn_pyramid_workspace_bytes(int64_t n, int64_t* bytes) {
  if (n < 0 || !bytes) return WCN_ERR_INVALID_PARAMETERS;
  *bytes = ((n + PYR_THREADS - 1) / PYR_THREADS * PYR_SHIFTS + 64) * 4;
  return WCN_OK;
}

extern "C" int wcn_pyramid(const int32_t* rows, int64_t n, const int32_t* info, const int64_t* offsets, int32_t batches,
                           int32_t levels, int32_t* out, int32_t* first, int32_t* counts, int64_t* host, void* workspace,
                           const int32_t* dev_status, void* stream) {
  if (n <= 0 || n >= 0x7FFFFFFFll || batches < 1 || levels < 1 || levels > 4 || !offsets) return WCN_ERR_INVALID_PARAMETERS;
  if (batches > SORT_MAX_BATCH) return WCN_ERR_UNSUPPORTED_CONFIG;
  if (!rows || !info || !out || !first || !counts || !host || !workspace || !dev_status || (reinterpret_cast<uintptr_t>(rows) & 15) ||
      (reinterpret_cast<uintptr_t>(out) & 15))
    return WCN_ERR_INVALID_PARAMETERS;
  PyramidParams p;
  p.rows = reinterpret_cast<const int4*>(rows); p.info = info; p.n = n; p.levels = levels;
  p.block_counts = (int32_t*)workspace; p.counts = counts; p.host = host; p.dev_status = dev_status; p.batches = batches;
  for (int l = 0; l < 4; ++l) {
    p.out[l] = l < levels ? reinterpret_cast<int4*>(out) + (int64_t)l * n : nullptr;
    p.first[l] = l < levels ? first + (int64_t)l * n : nullptr;
  }
  for (int b = 0; b <= batches; ++b) {
    if (offsets[b] < 0 || offsets[b] > n) return WCN_ERR_INVALID_PARAMETERS;
    p.offsets[b] = (int32_t)offsets[b];
  }
  cudaStream_t st = wcn_stream(stream);
  if (cudaMemsetAsync(counts, 0, 8 * sizeof(int32_t), st) != cudaSuccess) return WCN_ERR_EXECUTION;
  const unsigned blocks = (unsigned)((n + PYR_THREADS - 1) / PYR_THREADS);
  pyramid_count_kernel<<<blocks, PYR_THREADS, 0, st>>>(p);
  p.groups = (int)blocks;
  p.per_block = blocks >= 512 ? 4 : 1;
  pyramid_emit_kernel<<<(blocks + p.per_block - 1) / p.per_block, PYR_THREADS, 0, st>>>(p);
  WCN_CHECK_LAUNCH();
  return WCN_OK;
}
