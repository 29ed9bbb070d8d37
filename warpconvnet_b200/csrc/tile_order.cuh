// Tile order: what the kernels that group output rows by their neighbour pattern share.  Everything is in an unnamed
// namespace: each translation unit gets its own copy.
#pragma once
#include "wcn_common.cuh"

namespace {

constexpr int kTileWindowSmall = 4096, kTileWindowLarge = 16384;
constexpr int kTileOrderThreads = 1024;

// Rows of a window of a table of M rows in tile order: the large window above 4096 rows, in a network above 65 536.  (For the
// order in which a convolution begins its tiles; a table with other windows gives the same results.)
inline int tile_window(int64_t M, bool network) { return M > (network ? 65536 : 4096) ? kTileWindowLarge : kTileWindowSmall; }

// Sort key of a row from which of its K offsets have a neighbour (bit k of `present`).  For a 3x3x3 window the centre
// comes in bit 0, then the 6 face, 12 edge and 8 corner offsets, so that the rarest offsets are the most significant
// bits and rows that share them end up in the same tiles (2-4 % fewer (tile, offset) pairs than offsets in index
// order).  Only the order of the rows depends on it.
__device__ __forceinline__ constexpr int presence_bit27(int k) {
  const int ax = (k / 9 != 1) + ((k / 3) % 3 != 1) + (k % 3 != 1);   // 0 centre, 1 face, 2 edge, 3 corner
  int pos = 0;   // offsets of a lower class, and earlier ones of the same class, come first
  for (int q = 0; q < 27; ++q) {
    const int aq = (q / 9 != 1) + ((q / 3) % 3 != 1) + (q % 3 != 1);
    pos += (aq < ax) || (aq == ax && q < k);
  }
  return pos;
}

// Pass 2: one block per window sorts its rows by (mask, row) and replaces the masks by the row
// order.  Stable least-significant-digit radix sort of the permutation, 7 bits per pass
// (ceil(K / 7) passes): a warp owns 128 consecutive positions, ranks equal digits with
// match_any (lane order = position order, so the sort is stable and deterministic), the
// per-(digit, warp) counts are scanned digit-major by the block, and rows scatter to their place.
constexpr int kDigitBits = 7, kDigits = 1 << kDigitBits;

template <int kTileWindow>
__device__ __forceinline__ void sort_window(int32_t* __restrict__ rows_io, int64_t M, int K, int64_t window, uint8_t* sort_smem) {
  uint32_t* mask_s = reinterpret_cast<uint32_t*>(sort_smem);                       // mask of local row r (never moves)
  uint16_t (*perm_s)[kTileWindow] = reinterpret_cast<uint16_t (*)[kTileWindow]>(mask_s + kTileWindow);  // current / next order
  uint16_t* cnt = reinterpret_cast<uint16_t*>(perm_s + 2);                         // [digit][warp] counts, then start positions
  uint32_t* warp_sums = reinterpret_cast<uint32_t*>(cnt + kDigits * 32);
  constexpr int kBatches = kTileWindow / kTileOrderThreads;                        // rows per thread
  const int64_t base = window * kTileWindow;
  const int n = (int)min((int64_t)kTileWindow, M - base);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < kTileWindow; i += kTileOrderThreads) {
    mask_s[i] = i < n ? (uint32_t)rows_io[base + i] : 0xFFFFFFFFu;  // padding sorts last (ties: stable)
    perm_s[0][i] = (uint16_t)i;
  }
  int cur = 0;
  const int passes = (K + kDigitBits - 1) / kDigitBits;
  for (int pass = 0; pass < passes; ++pass) {
    const int shift = pass * kDigitBits;
    for (int i = threadIdx.x; i < kDigits * 32; i += kTileOrderThreads) cnt[i] = 0;
    __syncthreads();
    // rank inside (warp, digit); positions of a warp: warp * (32 * kBatches) + batch*32 + lane
    uint16_t row[kBatches];
    int dig[kBatches], rank[kBatches];
#pragma unroll
    for (int b = 0; b < kBatches; ++b) {
      row[b] = perm_s[cur][warp * (32 * kBatches) + b * 32 + lane];
      dig[b] = (int)((mask_s[row[b]] >> shift) & (kDigits - 1));
      const unsigned same = __match_any_sync(0xFFFFFFFFu, dig[b]);
      const int r = __popc(same & ((1u << lane) - 1u));
      const int leader = __ffs(same) - 1;
      int before = 0;
      if (r == 0) {  // the first lane of each digit updates the warp's count
        before = cnt[dig[b] * 32 + warp];
        cnt[dig[b] * 32 + warp] = (uint16_t)(before + __popc(same));
      }
      before = __shfl_sync(0xFFFFFFFFu, before, leader);
      rank[b] = before + r;
      __syncwarp();  // the next batch reads the counts written here
    }
    __syncthreads();
    // exclusive scan of the counts in (digit, warp) order: 4 consecutive entries per thread
    {
      constexpr int kPer = kDigits * 32 / kTileOrderThreads;
      uint32_t v[kPer], sum = 0;
#pragma unroll
      for (int j = 0; j < kPer; ++j) { v[j] = cnt[threadIdx.x * kPer + j]; sum += v[j]; }
      uint32_t incl = sum;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, incl, d);
        if (lane >= d) incl += o;
      }
      if (lane == 31) warp_sums[warp] = incl;
      __syncthreads();
      if (warp == 0) {
        const uint32_t w = warp_sums[lane];
        uint32_t wi = w;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, wi, d);
          if (lane >= d) wi += o;
        }
        warp_sums[lane] = wi - w;
      }
      __syncthreads();
      uint32_t run = warp_sums[warp] + incl - sum;
#pragma unroll
      for (int j = 0; j < kPer; ++j) { cnt[threadIdx.x * kPer + j] = (uint16_t)run; run += v[j]; }
    }
    __syncthreads();
#pragma unroll
    for (int b = 0; b < kBatches; ++b) perm_s[cur ^ 1][cnt[dig[b] * 32 + warp] + rank[b]] = row[b];
    cur ^= 1;
    __syncthreads();
  }
  for (int i = threadIdx.x; i < n; i += kTileOrderThreads) rows_io[base + i] = (int32_t)(base + perm_s[cur][i]);
}

template <int W> constexpr size_t sort_window_bytes() { return (size_t)W * 4 + 2 * (size_t)W * 2 + kDigits * 32 * 2 + 32 * 4; }

}  // namespace
