// Weight gradient of fp32 tensors on the 5th-generation tensor cores:
//     dW[k][ci][co] = sum over rows m with a neighbour at offset k of X[nbr[k][m]][ci] * dY[m][co]
// with every number as the exact sum of three bf16 numbers and six of the nine products kept, added in fp32 every 32 rows:
// see conv_split_tcgen05.cu for what that is worth and for the numbers that have no three parts.
//
// Three launches.  The first writes the three parts of X's rows, and of dY's rows in the order of the table, 32 rows at a time
// as the swizzled images that shared memory wants (a bulk copy per part; rows past the end are zeros).  The second: the
// M = 128 side of an instruction holds four "chunks" of 32 channels of X gathered through one offset each, consecutive chunks
// (offset-major) forming a group: two offsets at C_in = 64.  A CTA owns a group, up to 128 columns and a range of 128-row
// tiles, of which it takes those where the group's offsets have a neighbour at all (tile masks).  Four gather warps copy a
// chunk each (cp.async, absent rows zero-filled), one thread adds the dY images, two issue the instructions of a slot of 32
// rows in turns into one of four accumulators, and eight warps add every accumulator to the sums in their registers.  The
// ranges leave partial sums, which the third launch adds in order: the same bits on every run.
//
// Bound by the rate of narrow instructions (12 of 57 clocks at N = 64 per slot; the tensor pipe is busy for 37 % of the time) and
// the spread of the groups: an inner offset is in every tile, a corner in few; the inner ones start first.  Measured (us,
// conv_wgrad_pairs.cu / all three launches, L2 flushed): 60 000 room voxels, 64 -> 64 181 / 107, 128 -> 128 681 / 165, 96 -> 48 339 / 144; 2 000: 64 -> 64 52 / 26;
// outdoors, 60 000: 64 -> 64 118 / 93, 128 -> 128 525 / 149.  Distance from sums in 64 bits: 1.7e-7 against 6.2e-7, 2.0e-7 against
// 1.1e-6.  Table entries asked for one slot ahead instead of a tile ahead: 126 us instead of 79 for the second launch.
#include "wcn_common.cuh"
#include "tcgen05_common.cuh"
#include "split_bf16.cuh"

extern thread_local int wcn_f32_launches;   // api.cu

namespace {

constexpr int WS_ROWS = 32;                           // rows of a slot
constexpr int WS_CHUNK = WS_ROWS * 64;                // bytes of one part of 32 rows x 32 channels
constexpr int WS_CHUNKS = 4;                          // chunks of a group
constexpr int WS_A = 3 * WS_CHUNKS * WS_CHUNK;        // bytes of a slot's X
constexpr int WS_MAX_N = 128, WS_ACCS = 4, WS_MAX_SLOTS = 6;
constexpr int WS_MAX_TILES = 512;                     // 128-row tiles of a range
constexpr int WS_EPI = 256, WS_GATHER = 128;          // warps 0..7 and 8..11
constexpr int WS_MMA_WARP = 12, WS_ISSUERS = 2, WS_DY_WARP = 14, WS_THREADS = 480;
constexpr size_t WS_SMEM = 226 * 1024;
constexpr int WS_PLANE_BLOCKS = 1024;                 // of the first launch at most

struct WsParams {
  const char* planes;       // [num_in][3][cp] bf16
  const char* images;       // [tiles][4][3][gchunks] images of 32 rows x 32 channels
  const float* feats;       // (these two for sums that are not finite)
  const float* gout;
  const int32_t* nbr;
  const int32_t* out_rows;
  const uint32_t* masks;    // offsets present in every 128 rows of nbr
  int64_t M;
  int K, c_in, cp, c_out, num_in, gchunks;
  int groups, blocks, block_n, tiles, per_range, slots;
  float* dst;               // [ranges][K][c_in][c_out]
  int32_t* dev_status;
};

struct WsControl {
  uint64_t full[WS_MAX_SLOTS], empty[WS_MAX_SLOTS];
  uint64_t acc_full[WS_ACCS], acc_empty[WS_ACCS];
  uint32_t tmem;
  int32_t count;
  int32_t tile[WS_MAX_TILES];   // tiles of the range that the group has anything in
  uint32_t again[2][WS_CHUNKS]; // fours of columns (of the two halves) of a chunk with sums that are not finite
  uint32_t odd[2][128];         // those of a row
};

__global__ void __launch_bounds__(256)
wgrad_planes_kernel(const float* __restrict__ feats, int64_t num_in, int c_in, int cp, const float* __restrict__ gout, int64_t M, int c_out,
                    int gchunks, int tiles, const int32_t* __restrict__ out_rows, char* __restrict__ planes, char* __restrict__ images) {
  launch_dependents();
  const int per_x = cp / 8, per_g = gchunks * 4;
  const int64_t x_items = num_in * per_x, total = x_items + (int64_t)tiles * 128 * per_g;
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < total; i += (int64_t)gridDim.x * 256) {
    float v[8];
    if (i < x_items) {
      const int64_t r = i / per_x;
      const int c = (int)(i - r * per_x) * 8;
      load_eight(feats + r * c_in, c, c_in, v);
      store_parts(v, planes + r * 6 * cp + c * 2, (int64_t)cp * 2);
    } else {
      const int64_t q = i - x_items, m = q / per_g;
      const int c = (int)(q - m * per_g) * 8;
      if (m < M) {
        const int64_t r = out_rows ? (int64_t)__ldg(&out_rows[m]) : m;
        load_eight(gout + r * c_out, c, c_out, v);
      } else {
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = 0.f;
      }
      const int64_t apart = (int64_t)gchunks * WS_CHUNK;
      store_parts(v, images + (m / WS_ROWS) * 3 * apart + (c / 32) * WS_CHUNK + tile_offset<64>((int)(m % WS_ROWS), (c % 32) / 8), apart);
    }
  }
}

__global__ void __launch_bounds__(WS_THREADS, 1)
conv_wgrad_split_kernel(const WsParams p) {
  extern __shared__ uint8_t smem_raw[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int BN = p.block_n, b_bytes = BN * 64, slot_bytes = WS_A + 3 * b_bytes;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  WsControl* ctl = reinterpret_cast<WsControl*>(smem_raw + (base - smem_u32(smem_raw)) + p.slots * slot_bytes);
  auto bar = [](uint64_t* b) { return smem_u32(b); };
  // groups from the middle outwards (the inner offsets are in every tile)
  const int block = (int)blockIdx.x % p.blocks, turn = ((int)blockIdx.x / p.blocks) % p.groups, range = (int)blockIdx.x / (p.blocks * p.groups);
  const int middle = (p.groups - 1) / 2;
  const int group = (turn & 1) ? middle + (turn + 1) / 2 : middle - turn / 2;
  const int bn = min(BN, p.gchunks * 32 - block * BN);   // (the last column block may be narrower)
  const int cpc = p.cp / 32, chunks = p.K * cpc;
  const int t0 = range * p.per_range, t1 = min(p.tiles, t0 + p.per_range);
  uint32_t offsets = 0;
#pragma unroll
  for (int w = 0; w < WS_CHUNKS; ++w)
    if (group * WS_CHUNKS + w < chunks) offsets |= 1u << ((group * WS_CHUNKS + w) / cpc);

  if (warp == 0) {
    if (lane < p.slots) { mbar_init(bar(&ctl->full[lane]), WS_GATHER + 1); mbar_init(bar(&ctl->empty[lane]), 1); }
    if (lane < WS_ACCS) { mbar_init(bar(&ctl->acc_full[lane]), 1); mbar_init(bar(&ctl->acc_empty[lane]), WS_EPI / 32); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    int n = 0;
    for (int t = t0; t < t1; t += 32) {
      const bool there = t + lane < t1 && (__ldg(&p.masks[t + lane]) & offsets);
      const uint32_t b = __ballot_sync(0xFFFFFFFFu, there);
      if (there) ctl->tile[n + __popc(b & ((1u << lane) - 1u))] = t + lane;
      n += __popc(b);
    }
    if (lane == 0) ctl->count = n;
    if (lane < 2 * WS_CHUNKS) ctl->again[lane / WS_CHUNKS][lane % WS_CHUNKS] = 0;
  } else if (warp == WS_MMA_WARP) {
    tmem_alloc(smem_u32(&ctl->tmem), 512);
  }
  // (everything above runs while the parts are written; tables, masks and rows are older than that launch)
  wait_for_primary();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = ctl->tmem;
  const int steps = ctl->count * 4;
  bool ok = true, redo = false;

  if (warp >= 8 && warp < WS_MMA_WARP) {
    // ================================================================ gather: a chunk per warp
    const int w = warp - 8, q = group * WS_CHUNKS + w;
    const bool mine = q < chunks;
    const int k = mine ? q / cpc : 0, c = mine ? q % cpc : 0;
    const int sub = lane >> 2, chunk = lane & 3;       // a copy instruction covers eight rows of 64 bytes
    const uint32_t at = w * WS_CHUNK + tile_offset<64>(sub, chunk);
    const char* from = p.planes + c * 64 + chunk * 16;
    const int64_t row_bytes = (int64_t)p.cp * 6;
    const int32_t* table = p.nbr + (int64_t)k * p.M;
    int slot = 0, phase = 0;
    bool bad = false;
    // The rows of a tile are asked for a tile ahead: a load waits behind the copies that are queued, longer than a slot takes.
    int next[4];
    auto rows_of = [&](int t) {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int64_t m = t * 4 < steps && mine ? (int64_t)ctl->tile[t] * 128 + u * WS_ROWS + lane : p.M;
        next[u] = m < p.M ? __ldg(table + m) : -1;
      }
    };
    rows_of(0);
    for (int t = 0; t * 4 < steps && ok; ++t) {
      int rows[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        rows[u] = next[u];
        if (rows[u] >= p.num_in) { rows[u] = -1; bad = true; }
      }
      rows_of(t + 1);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int r = rows[u];
        if (!mbar_wait(bar(&ctl->empty[slot]), phase ^ 1, p.dev_status)) { ok = false; break; }
        __syncwarp();
        if (mine) {
          const uint32_t dst = base + slot * slot_bytes + at;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int rj = __shfl_sync(0xFFFFFFFFu, r, 8 * j + sub);
            const char* src = from + (int64_t)max(rj, 0) * row_bytes;
#pragma unroll
            for (int s = 0; s < 3; ++s) cp_async16(dst + s * (WS_CHUNKS * WS_CHUNK) + j * 512, src + s * p.cp * 2, rj >= 0 ? 16u : 0u);
          }
        }
        cp_async_arrive(bar(&ctl->full[slot]));
        if (++slot == p.slots) { slot = 0; phase ^= 1; }
      }
    }
    cp_async_drain();
    if (bad) wcn_report_bounds(p.dev_status);
  } else if (warp == WS_DY_WARP) {
    // ================================================================ dY
    if (elect_one()) {
      int slot = 0, phase = 0;
      const int64_t part = (int64_t)p.gchunks * WS_CHUNK;
      for (int i = 0; i < steps; ++i) {
        if (!mbar_wait(bar(&ctl->empty[slot]), phase ^ 1, p.dev_status)) { ok = false; break; }
        const uint32_t dst = base + slot * slot_bytes + WS_A, full = bar(&ctl->full[slot]);
        const char* src = p.images + ((int64_t)ctl->tile[i >> 2] * 4 + (i & 3)) * 3 * part + (int64_t)block * b_bytes;
        mbar_expect_tx(full, (uint32_t)(3 * bn * 64));
#pragma unroll
        for (int s = 0; s < 3; ++s) bulk_copy_g2s(dst + s * b_bytes, src + s * part, (uint32_t)(bn * 64), full);
        if (++slot == p.slots) { slot = 0; phase ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == WS_MMA_WARP || warp == WS_MMA_WARP + 1) {
    // ================================================================ tensor-core instructions, slots in turns
    if (elect_one()) {
      // fp32 accumulate, bf16, A and B MN-major (bits 15, 16), N = bn, M = 128
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((uint32_t)(bn >> 3) << 17) | (8u << 24);
      int slot = 0, phase = 0, ab = 0, aphase = 0;
      for (int i = 0; i < steps; ++i) {
        if ((i & 1) == warp - WS_MMA_WARP) {
          if (!mbar_wait(bar(&ctl->acc_empty[ab]), aphase ^ 1, p.dev_status) ||
              !mbar_wait(bar(&ctl->full[slot]), phase, p.dev_status)) { ok = false; break; }
          tc_fence_after();
          const uint64_t a = smem_desc_mn<64>(base + slot * slot_bytes, WS_CHUNK), b = smem_desc_mn<64>(base + slot * slot_bytes + WS_A, WS_CHUNK);
          const uint32_t d = tmem + ab * WS_MAX_N;
#pragma unroll
          for (int q = 0; q < 6; ++q)
#pragma unroll
            for (int ks = 0; ks < WS_ROWS / 16; ++ks)   // 16 rows = two 8-row atoms further down the tiles
              umma_f16(d, a + (uint64_t)(split_a(q) * ((WS_CHUNKS * WS_CHUNK) >> 4) + ks * 64), b + (uint64_t)(split_b(q) * (b_bytes >> 4) + ks * 64),
                       idesc, q + ks > 0 ? 1u : 0u);
          umma_commit(bar(&ctl->empty[slot]));
          umma_commit(bar(&ctl->acc_full[ab]));
        }
        if (++slot == p.slots) { slot = 0; phase ^= 1; }
        if (++ab == WS_ACCS) { ab = 0; aphase ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp < 8) {
    // ================================================================ sums: a row of the group per thread, half of its columns
    const int half = warp >> 2, mid = ((bn / 16 + 1) / 2) * 16;
    const int c_begin = half ? mid : 0, cols = half ? bn - mid : mid;   // at most 64 columns a thread
    float sum[64];
#pragma unroll
    for (int i = 0; i < 64; ++i) sum[i] = 0.f;
    int ab = 0, aphase = 0;
    for (int i = 0; i < steps; ++i) {
      ok = mbar_wait(bar(&ctl->acc_full[ab]), aphase, p.dev_status);
      if (!__all_sync(0xFFFFFFFFu, ok)) { ok = false; break; }
      tc_fence_after();
      const uint32_t at = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(ab * WS_MAX_N + c_begin);
#pragma unroll
      for (int c = 0; c < 64; c += 32) {
        if (c < cols) {
          uint32_t v[2][16];
          tmem_ld16(at + c, v[0]);
          if (c + 16 < cols) tmem_ld16(at + c + 16, v[1]);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j) sum[c + j] += __uint_as_float(v[0][j]);
          if (c + 16 < cols) {
#pragma unroll
            for (int j = 0; j < 16; ++j) sum[c + 16 + j] += __uint_as_float(v[1][j]);
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(&ctl->acc_empty[ab]));
      if (++ab == WS_ACCS) { ab = 0; aphase ^= 1; }
    }
    const int q = group * WS_CHUNKS + (warp & 3), k = q / cpc, ci = (q % cpc) * 32 + lane;
    const int n0 = block * BN + c_begin;
    float* dst = p.dst + (((int64_t)range * p.K + k) * p.c_in + ci) * p.c_out + n0;
    uint32_t mine = 0;   // fours of columns with a sum that is not finite
    if (q < chunks && ci < p.c_in) {
      const bool poison = !ok || *(volatile const int32_t*)p.dev_status == (int)WCN_ERR_WAIT_EXPIRED;
#pragma unroll
      for (int c = 0; c < 64; c += 4)
        if (c < cols && n0 + c < p.c_out) {
          const float nan = __int_as_float(0x7FC00000);
          if (poison) *reinterpret_cast<float4*>(dst + c) = make_float4(nan, nan, nan, nan);
          else if (!(fmaf(sum[c], 0.f, sum[c + 1] * 0.f) + fmaf(sum[c + 2], 0.f, sum[c + 3] * 0.f) == 0.f)) mine |= 1u << (c / 4);
          else *reinterpret_cast<float4*>(dst + c) = make_float4(sum[c] * kSumScale, sum[c + 1] * kSumScale, sum[c + 2] * kSumScale, sum[c + 3] * kSumScale);
        }
    }
    const uint32_t any = __reduce_or_sync(0xFFFFFFFFu, mine);
    redo = any != 0;
    if (redo) {
      ctl->odd[half][tid & 127] = mine;
      if (lane == 0) ctl->again[half][warp & 3] = any;
    }
  }
  tc_fence_before();
  redo = __syncthreads_or(redo);
  // A number without three parts, or one beside an absent row (0 times infinity): such sums are made again on the FMA pipes
  // from the present pairs, up to eight fours of a chunk at a time.  All warps take slots of 32 rows in turns, their sums
  // are added in order through the ring, which nothing uses any more (60 000 room voxels, 64 -> 64, 101 us: 357 with a NaN in
  // a row of X and one of dY, 930 with nothing else, 175 in conv_wgrad_pairs.cu; one thread per sum walking all rows took
  // 20 000, an epilogue warp on its own 808 and 1 629).
  float* part = reinterpret_cast<float*>(smem_raw + (base - smem_u32(smem_raw)));
  for (int i = 0; redo && i < 2 * WS_CHUNKS; ++i) {
    const int half = i / WS_CHUNKS, w = i % WS_CHUNKS, q = group * WS_CHUNKS + w, k = q / cpc, ci = (q % cpc) * 32 + lane;
    const int n0 = block * BN + (half ? ((bn / 16 + 1) / 2) * 16 : 0);
    for (uint32_t rest = ctl->again[half][w]; rest;) {
      int col[8], fours = 0;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        col[j] = rest ? (__ffs(rest) - 1) * 4 : 0;
        fours += rest ? 1 : 0;
        rest &= rest - 1;
      }
      float4 acc[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int t = warp; t < steps; t += WS_THREADS / 32) {
        const int64_t m = (int64_t)ctl->tile[t >> 2] * 128 + (t & 3) * WS_ROWS + lane;
        const int r = m < p.M ? __ldg(&p.nbr[(int64_t)k * p.M + m]) : -1;
        const int64_t at = m < p.M && p.out_rows ? (int64_t)__ldg(&p.out_rows[m]) : m;
        for (uint32_t have = __ballot_sync(0xFFFFFFFFu, r >= 0 && r < p.num_in); have;) {   // (others are reported by the gather warps)
          float x[4];
          const float* g[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int row = have ? __ffs(have) - 1 : -1;
            have &= have - 1;
            const int64_t from = __shfl_sync(0xFFFFFFFFu, r, max(row, 0)), to = __shfl_sync(0xFFFFFFFFu, at, max(row, 0));
            x[u] = row >= 0 && ci < p.c_in ? __ldg(&p.feats[from * p.c_in + ci]) : 0.f;
            g[u] = row >= 0 ? p.gout + to * p.c_out + n0 : nullptr;
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if (j >= fours) break;
            float4 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = g[u] ? __ldg(reinterpret_cast<const float4*>(g[u] + col[j])) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              acc[j].x = fmaf(x[u], v[u].x, acc[j].x);
              acc[j].y = fmaf(x[u], v[u].y, acc[j].y);
              acc[j].z = fmaf(x[u], v[u].z, acc[j].z);
              acc[j].w = fmaf(x[u], v[u].w, acc[j].w);
            }
          }
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (j < fours) reinterpret_cast<float4*>(part)[(warp * 8 + j) * 32 + lane] = acc[j];
      __syncthreads();
      int c = 0;
#pragma unroll
      for (int j = 0; j < 8; ++j) c = warp == j ? col[j] : c;
      if (warp < fours && ((ctl->odd[half][w * 32 + lane] >> (c / 4)) & 1u)) {
        float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int from = 0; from < WS_THREADS / 32; ++from) {
          const float4 v = reinterpret_cast<const float4*>(part)[(from * 8 + warp) * 32 + lane];
          y.x += v.x; y.y += v.y; y.z += v.z; y.w += v.w;
        }
        *reinterpret_cast<float4*>(p.dst + (((int64_t)range * p.K + k) * p.c_in + ci) * p.c_out + n0 + c) = y;
      }
      __syncthreads();
    }
  }
  if (warp == WS_MMA_WARP) tmem_dealloc(tmem, 512);
}

__global__ void wgrad_sum_kernel(const float4* __restrict__ partial, int ranges, int64_t n, float4* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float4 s = __ldcg(&partial[i]);
#pragma unroll 8
  for (int r = 1; r < ranges; ++r) {
    const float4 v = __ldcg(&partial[r * n + i]);
    s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
  }
  out[i] = s;
}

struct WsPlan {
  int cp, gchunks, groups, blocks, block_n, tiles, ranges, per_range;
  size_t planes, images, partial;
};

WsPlan plan_ws(int64_t num_in, int64_t M, int K, int c_in, int c_out) {
  WsPlan q;
  q.cp = (c_in + 31) / 32 * 32;
  q.gchunks = (c_out + 31) / 32;
  q.groups = (K * (q.cp / 32) + WS_CHUNKS - 1) / WS_CHUNKS;
  q.blocks = (q.gchunks + 3) / 4;   // as few as there can be: each gathers all rows of X again (64 -> 160 columns in five: 435 us, two 263)
  q.block_n = (q.gchunks + q.blocks - 1) / q.blocks * 32;
  q.blocks = (q.gchunks * 32 + q.block_n - 1) / q.block_n;
  q.tiles = (int)((M + 127) / 128);
  // Three CTAs a multiprocessor or more (they differ in what they have to do), of at least four tiles each.
  const int64_t work = (int64_t)q.groups * q.blocks;
  int64_t ranges = (3 * (int64_t)wcn_num_sms() + work - 1) / work;
  const int64_t most = (q.tiles + 3) / 4, least = (q.tiles + WS_MAX_TILES - 1) / WS_MAX_TILES;
  if (ranges > most) ranges = most;
  if (ranges < least) ranges = least;
  q.per_range = (int)((q.tiles + ranges - 1) / ranges);
  q.ranges = (q.tiles + q.per_range - 1) / q.per_range;
  q.planes = (size_t)num_in * q.cp * 6;
  q.images = (size_t)q.tiles * 12 * q.gchunks * WS_CHUNK;
  q.partial = q.ranges > 1 ? (size_t)q.ranges * K * c_in * c_out * 4 : 0;
  return q;
}

bool wgrad_split_supported(int64_t num_in, int64_t M, int K, int c_in, int c_out) {
  return num_in > 0 && M > 0 && M < 0x3FFFFFFFll && num_in < 0x7FFFFFFFll && K >= 1 && K <= 32 && c_in >= 16 && c_out >= 16 &&
         c_in % 4 == 0 && c_out % 4 == 0 && c_in <= 4096 && c_out <= 4096;
}

}  // namespace

extern "C" int wcn_conv_wgrad_f32_workspace_bytes(int64_t num_in, int64_t num_out, int32_t num_offsets, int32_t c_in, int32_t c_out,
                                                  int64_t* bytes) {
  if (!bytes || num_in < 0 || num_out < 0 || num_offsets <= 0 || c_in <= 0 || c_out <= 0) return WCN_ERR_INVALID_PARAMETERS;
  *bytes = 0;
  // Few offsets stay on the FP32 pipes (8 of them, 60 000 rows of 64 -> 64: 50 us / 42 in a room, 32 / 74 outdoors: the three
  // parts are as much to write as the gradient is to read), and narrow layers, where the two take the same time (32 -> 32,
  // 27 offsets, 60 000 rows: 79 / 69, outdoors 58 / 64).
  // So do a few rows of a large matrix, all of whose rows would be split (see wcn_conv_f32_workspace_bytes).
  const double area = (double)c_in * c_out;
  if (num_in > 8 * num_out && 2e-6 * (double)num_in * ((c_in + 31) / 32 * 32) > 25. + 3.7e-7 * area * (double)num_out) return WCN_OK;
  if (num_offsets < 16 || area < 2048 || !wgrad_split_supported(num_in, num_out, num_offsets, c_in, c_out)) return WCN_OK;
  const WsPlan q = plan_ws(num_in, num_out, num_offsets, c_in, c_out);
  *bytes = (int64_t)(q.planes + q.images + q.partial);
  return WCN_OK;
}

extern "C" int wcn_conv_wgrad_f32(const float* feats, int64_t num_in, const float* grad_out, const int32_t* nbr, const int32_t* out_rows,
                                  const uint32_t* tile_masks, int64_t num_out, int32_t num_offsets, int32_t c_in, int32_t c_out,
                                  float* grad_weight, void* workspace, int64_t workspace_bytes, int32_t* dev_status, void* stream) {
  if (!wgrad_split_supported(num_in, num_out, num_offsets, c_in, c_out)) return WCN_ERR_UNSUPPORTED_CONFIG;
  auto odd = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) != 0; };
  if (!feats || !grad_out || !nbr || !tile_masks || !grad_weight || !workspace || !dev_status || odd(feats) || odd(grad_out) ||
      odd(grad_weight) || odd(workspace))
    return WCN_ERR_INVALID_PARAMETERS;
  const WsPlan q = plan_ws(num_in, num_out, num_offsets, c_in, c_out);
  if (workspace_bytes < (int64_t)(q.planes + q.images + q.partial)) return WCN_ERR_INVALID_PARAMETERS;
  static bool configured[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return WCN_ERR_INITIALIZATION;
  if (!configured[dev]) {
    if (cudaFuncSetAttribute(conv_wgrad_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WS_SMEM) != cudaSuccess) {
      (void)cudaGetLastError();
      return WCN_ERR_INITIALIZATION;
    }
    configured[dev] = true;
  }
  cudaStream_t st = wcn_stream(stream);
  char* ws = (char*)workspace;
  WsParams p = {};
  p.planes = ws; p.images = p.planes + q.planes;
  p.feats = feats; p.gout = grad_out; p.nbr = nbr; p.out_rows = out_rows; p.masks = tile_masks;
  p.M = num_out; p.K = num_offsets; p.c_in = c_in; p.cp = q.cp; p.c_out = c_out; p.num_in = (int)num_in; p.gchunks = q.gchunks;
  p.groups = q.groups; p.blocks = q.blocks; p.block_n = q.block_n; p.tiles = q.tiles; p.per_range = q.per_range;
  p.dst = q.ranges > 1 ? (float*)(ws + q.planes + q.images) : grad_weight;
  p.dev_status = dev_status;
  const size_t slot = WS_A + 3 * (size_t)q.block_n * 64, fixed = 1024 + sizeof(WsControl) + 64;
  p.slots = (int)((WS_SMEM - fixed) / slot);
  if (p.slots > WS_MAX_SLOTS) p.slots = WS_MAX_SLOTS;
  const int64_t ctas = (int64_t)q.ranges * q.groups * q.blocks;
  if (ctas > 0x7FFFFFFFll) return WCN_ERR_UNSUPPORTED_CONFIG;
  const int64_t items = num_in * (q.cp / 8) + (int64_t)q.tiles * 128 * q.gchunks * 4;
  int64_t blocks = (items + 511) / 512;
  if (blocks > WS_PLANE_BLOCKS) blocks = WS_PLANE_BLOCKS;
  wgrad_planes_kernel<<<(unsigned)blocks, 256, 0, st>>>(feats, num_in, c_in, q.cp, grad_out, num_out, c_out, q.gchunks, q.tiles, out_rows,
                                                        (char*)p.planes, (char*)p.images);
  WCN_CHECK_LAUNCH();
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctas); cfg.blockDim = dim3(WS_THREADS); cfg.dynamicSmemBytes = fixed + p.slots * slot; cfg.stream = st;
  cfg.attrs = &attr; cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, conv_wgrad_split_kernel, p) != cudaSuccess) {
    (void)cudaGetLastError();
    return WCN_ERR_EXECUTION;
  }
  wcn_f32_launches = q.ranges == 1 ? 2 : 3;
  if (q.ranges == 1) return WCN_OK;
  const int64_t n = (int64_t)num_offsets * c_in * c_out / 4;
  wgrad_sum_kernel<<<(unsigned)((n + 127) / 128), 128, 0, st>>>((const float4*)p.dst, q.ranges, n, (float4*)grad_weight);
  WCN_CHECK_LAUNCH();
  return WCN_OK;
}
