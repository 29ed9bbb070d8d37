// Output-stationary sparse convolution on the 5th-generation tensor cores.
//
// A CTA (one per SM) works through units of G x 128 consecutive output rows.  Each 128-row sub-tile owns one fp32
// accumulator in tensor memory (the 128 TMEM lanes of an M = 128 tcgen05.mma); the accumulators are double-buffered when
// they fit, so the epilogue of one unit overlaps the main loop of the next.  Five warp roles, connected by mbarrier rings:
//  * eight index warps choose the NEXT unit (fixed strides, or claimed from the hardware's queue of CTAs not yet started),
//    read its neighbour table and stage, for every sub-tile and every offset at which it has any neighbour, the list of
//    128 input rows;
//  * all roles then walk  offsets with a neighbour x channel slices : one thread fetches the weight slice of (offset,
//    channel slice) ONCE per unit with a bulk copy (the packed weights hold the swizzled shared-memory image), and four
//    gather warps per sub-tile copy the 128 neighbour rows of the feature matrix into a K-major swizzled tile of that
//    sub-tile's own ring (16-byte cp.async, whole row segments per request, absent rows zero-filled); the copies signal
//    the ring's mbarrier themselves when they land;
//  * one thread per sub-tile issues tcgen05.mma and releases ring slots with tcgen05.commit;
//  * four epilogue warps per sub-tile read the accumulators with tcgen05.ld, apply scale/shift (folded BatchNorm or bias),
//    residual add and ReLU, convert and store every output row exactly once.  No atomics, bit-reproducible.
//
// What bounds it, and what the layout buys (B200, 500 000 rows of a 1 cm room, 9.2 neighbours a row, L2 flushed).  The
// tensor cores are far from busy below 256 channels: a slot passes through four single-thread or single-warp streams, a
// barrier round trip costs 350 to 450 clocks, and with one ring for both sub-tiles and both issuers in step the streams
// waited for each other (no copies, no instructions and no stores at all still took 486 of 631 us at C = 256).  A ring and
// four gather warps per sub-tile, issuing threads that share nothing but the weight slots and look at the next barriers
// early, instructions issued behind elect.sync, lists of present offsets only (their 27 KB became row slots) and claimed
// units: C = 32 / 64 / 96 / 128 / 256 from 94 / 133 / 158 / 201 / 636 us to 86 / 118 / 152 / 186 / 520 us (256: 1.17
// PFLOP/s); outdoor scene, 128 -> 96 bf16, 777 777 rows: 449 -> 422 us (whole calls in turn, with what follows);
// MinkUNet-34 over 1.2 M voxels: 4.77 -> 4.50 ms.  Then a shorter way to the first copy of a launch - the first unit's neighbour loads issued before the barriers are set up, a
// single unit's table published without a rendezvous of the index warps, no look at the status word on the way (the epilogue
// reads it and writes NaN where an earlier launch gave up): C = 32 / 64 / 96 81 / 113 / 144 us, the network over one
// scene of 20 000 voxels 928 -> 855 us, over 1.2 M 4.41 ms.  Then the order of the units (supertile_of) and claims that wait
// until the unit before last is done: a multiprocessor was idle for 15 to 17 % of a layer, 500 000 rows of 64 / 128 / 256
// channels 113 / 187 / 547 -> 104 / 170 / 499 us, the network over 150 000 / 1.2 M voxels 1 318 / 4 589 -> 1 273 / 4 449.
//
// Problems with fewer 128-row tiles than multiprocessors divide the kernel offsets of a tile among the S CTAs of a
// cluster ("split-K over kernel offsets": slice s owns the offsets k with k % S == s, which deals the frequent central
// ones evenly).  Each CTA leaves its fp32 accumulators in its shared memory, where the ring was, and adds 1 / S of the
// rows over all slices through distributed shared memory, in slice order, with the epilogue behind it: no workspace, no
// second kernel, no atomics and the same bits on every run.
//
// Launches of one network overlap (programmatic dependent launch): everything up to the first read of a feature row -
// barriers, tensor memory, neighbour tables, weight slices, all written before the network's first launch - runs while
// the previous layer finishes.
//
// Every wait is bounded: a wait that runs out stores WCN_ERR_WAIT_EXPIRED in the
// device status word, the other waits notice it and the CTA leaves through the
// normal exit path (tensor memory released).
#include "wcn_common.cuh"
#include "tcgen05_common.cuh"
#include "tile_order.cuh"
#include <atomic>

namespace {

constexpr int BLOCK_M = 128;
constexpr int MAX_G = 2;              // sub-tiles per supertile (one per MMA issuer)
constexpr int MAX_RING = 12;          // slots per ring
constexpr int MAX_OFFSETS = 27;
constexpr int MAX_SLICES = 8;         // CTAs of a (portable) cluster
constexpr int EPI_THREADS = 256;      // warps 0..7: TMEM lane quarter = warp index & 3, one sub-tile per four warps
constexpr int IDX_THREADS = 256;      // warps 8..15: neighbour-table staging, four warps per sub-tile
constexpr int GATHER_WARP0 = 16;      // warps 16..23: row gathers, four per sub-tile
constexpr int GATHER_THREADS = 256;
constexpr int MMA_WARP = 24;          // warps 24, 25: MMA issuers, one per sub-tile; warp 24 owns TMEM
constexpr int MMA_ISSUERS = 2;
constexpr int WEIGHT_WARP = 26;       // weight bulk copies
constexpr int THREADS = 864;
constexpr int SMEM_LIMIT = 226 * 1024;  // dynamic shared memory the kernels opt in to
constexpr int TAIL_WINDOWS = 12;      // windows of the tile order that are begun together, at the end of a launch

struct ConvTcParams {
  const char* feats;
  bool wide_out, wide_res;   // rows of `out` / `residual` start on 32-byte boundaries
  const char* wpacked;
  const int32_t* nbr;
  const int32_t* out_rows;  // slot -> output row, or null for the identity
  int64_t M, num_in;
  int64_t in_ld_bytes;      // distance between consecutive feature rows, bytes
  int64_t out_ld, res_ld;   // distance between consecutive output / residual rows, elements
  int K, c_in, c_out;       // c_in: padded to the packed weights' channel slices
  int row_bytes;            // bytes of a feature row (the channels beyond are filled with zeros)
  const float* scale;
  const float* shift;
  const void* residual;
  int relu;
  void* out;
  int32_t* dev_status;
  int block_n;      // output columns per CTA (blockIdx.y selects the column block)
  int G;            // sub-tiles per supertile: 1 or 2
  int nbuf;         // accumulator sets in TMEM: 1 or 2
  int cols;         // TMEM columns per accumulator (power of two >= block_n)
  int sa, sb;       // ring depths (row slots of each sub-tile, weight slots)
  int kbc;          // channel slices per ring slot (a slot holds kbc K-major tiles side by side)
  int64_t supertiles;
  int S;            // offset slices per supertile (split-K over kernel offsets); 1 = none
  int64_t units;    // supertiles * S work units, walked by the persistent CTAs (S > 1: one each)
  bool claim;       // one CTA per unit was launched: a CTA claims further units from the hardware's queue
  int window, tail; // supertiles of a window of the tile order (0: rows in no such order), windows of the launch's tail
};

// Row lists (128 input rows of one sub-tile at one offset) staged per sub-tile: two units of ordinary density where K is
// large, two of any density where it is small.
__host__ __device__ inline int staged_lists(int K) { return K >= 27 ? K : (2 * K < 27 ? 2 * K : 27); }

// The supertile that comes `turn`-th.  The tile order puts the rows with the fewest neighbours first in a window and those
// with the most last, so that a supertile takes between a fifth of the mean time and three times as long.  Taken as they
// lie, the last to begin were the longest: one multiprocessor finished while the others had been idle for 15 to 17 % of a
// layer of 500 000 rows.  So every window is begun with its last supertile, windows from the last to the first, and the first
// `tail` windows come together at the end, the longest supertiles of all of them first: what begins last is short.  (All
// windows together would gather from the whole feature matrix at once.)
__device__ __forceinline__ int64_t supertile_of(const ConvTcParams& p, int64_t turn) {
  if (p.window == 0) return turn;
  const int64_t head = p.supertiles - (int64_t)p.tail * p.window;
  if (turn < head) return p.supertiles - 1 - turn;
  const int j = (int)(turn - head), place = j / p.tail, w = j - place * p.tail;
  return (int64_t)w * p.window + (p.window - 1 - place);
}

// Offsets of slice s of S: the k with k % S == s.
__device__ __forceinline__ uint32_t slice_mask(int s, int S) {
  if (S <= 1) return 0xFFFFFFFFu;
  uint32_t m = 0;
  for (int k = s; k < 32; k += S) m |= 1u << k;
  return m;
}

__device__ __forceinline__ void cluster_meet() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ float4 ld_cluster(uint32_t addr, uint32_t rank) {
  float4 v;
  asm volatile(
      "{\n\t.reg .b32 r;\n\tmapa.shared::cluster.u32 r, %4, %5;\n\t"
      "ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [r];\n\t}"
      : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
      : "r"(addr), "r"(rank)
      : "memory");
  return v;
}

// 32 bytes in one request: a whole sector per lane.  Every thread of the epilogue writes its own row,
// so a store instruction touches 32 different lines; with 16-byte pieces the L2 gets two half-sector
// writes per sector, with 32-byte ones a single full-sector write.
__device__ __forceinline__ void st_global_32B(void* p, const uint32_t* v) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]),
               "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}

__device__ __forceinline__ void ld_global_32B(const void* p, uint32_t* v) {
  asm volatile("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "l"(p));
}

// Sixteen elements; `wide`: the address is 32-byte aligned (rows start on 32-byte boundaries).
template <typename TO> __device__ __forceinline__ void load_raw16(const TO* p, TO* v, bool wide) {
  uint32_t* w = reinterpret_cast<uint32_t*>(v);
  if (wide) {
#pragma unroll
    for (int i = 0; i < (int)sizeof(TO) / 2; ++i) ld_global_32B(reinterpret_cast<const char*>(p) + 32 * i, w + 8 * i);
  } else {
#pragma unroll
    for (int i = 0; i < (int)sizeof(TO); ++i) {
      const uint4 x = __ldg(reinterpret_cast<const uint4*>(p) + i);
      w[4 * i] = x.x; w[4 * i + 1] = x.y; w[4 * i + 2] = x.z; w[4 * i + 3] = x.w;
    }
  }
}
template <typename TO> __device__ __forceinline__ void store16(TO* p, const float (&y)[16], bool wide) {
  __align__(32) TO v[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = wcn_from_float<TO>(y[i]);
  const uint32_t* w = reinterpret_cast<const uint32_t*>(v);
  if (wide) {
#pragma unroll
    for (int i = 0; i < (int)sizeof(TO) / 2; ++i) st_global_32B(reinterpret_cast<char*>(p) + 32 * i, w + 8 * i);
  } else {
#pragma unroll
    for (int i = 0; i < (int)sizeof(TO); ++i)
      reinterpret_cast<uint4*>(p)[i] = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
  }
}

// Up to N active offsets taken from the low end of `rest` (bit k = offset k still to do);
// ku[u] = -1 beyond the last one.  Returns how many were taken.
template <int N> __device__ __forceinline__ int pop_offsets(uint32_t& rest, int (&ku)[N]) {
  int n = 0;
#pragma unroll
  for (int u = 0; u < N; ++u) {
    ku[u] = -1;
    if (rest) {
      ku[u] = __ffs(rest) - 1;
      rest &= rest - 1;
      n = u + 1;
    }
  }
  return n;
}

// Ring cursor: slot index and the parity of the phase the slot is in.
struct Ring {
  int slot, phase, depth;
  __device__ __forceinline__ void advance() {
    if (++slot == depth) { slot = 0; phase ^= 1; }
  }
};

// Control block in shared memory.  Everything a unit's roles need to know about it - which unit it is, which offsets its
// sub-tiles have, where their neighbour rows were staged - is published by the index warps in one of two `info` entries.
struct Control {
  uint64_t a_full[MAX_G][MAX_RING], a_empty[MAX_G][MAX_RING];
  uint64_t b_full[MAX_RING], b_empty[MAX_RING];
  uint64_t acc_full[2][MAX_G], acc_empty[2][MAX_G];
  uint64_t info_full[2], info_empty[2];
  uint64_t idx_sync;              // rendezvous of the index threads (bounded, unlike bar.sync)
  uint64_t claim_full;            // a claimed unit has arrived in `claim`
  __align__(16) uint64_t claim[2];
  int64_t info_unit[2];           // the unit; < 0: no more units
  uint32_t info_mask[2][MAX_G];   // non-empty offsets of each sub-tile
  int info_entry[2][MAX_G];       // first staged row list of each sub-tile
  uint32_t mask_acc[3][MAX_G];    // index warps' scratch while building the masks
  uint32_t tmem_holder;
  int32_t out_row[2][MAX_G * BLOCK_M];          // output row of each slot, -1 past the end
  __align__(16) float sc[256], sh[256];         // this CTA's columns of the epilogue scale / shift (1 / 0 when absent)
};

// The hardware's work queue (cluster launch control): a running CTA claims a CTA of its grid that has not started yet
// and does that one's unit itself.  Units differ in their number of offsets; dealt in fixed strides they left the
// multiprocessors idle for about 15 % of a 256-channel layer, claimed one by one they leave only the last unit.
__device__ __forceinline__ void claim_next(uint32_t dst, uint32_t bar) {
  mbar_expect_tx(bar, 16u);
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(dst),
               "r"(bar)
               : "memory");
}
__device__ __forceinline__ int64_t claimed_unit(const uint64_t (&c)[2]) {
  uint32_t got, x;
  asm volatile(
      "{\n\t.reg .b128 h;\n\t.reg .pred p;\n\tmov.b128 h, {%2, %3};\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\n\tselp.u32 %0, 1, 0, p;\n\tmov.u32 %1, 0;\n\t"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %1, h;\n\t}"
      : "=r"(got), "=r"(x)
      : "l"(*(volatile const uint64_t*)&c[0]), "l"(*(volatile const uint64_t*)&c[1])
      : "memory");
  return got ? (int64_t)x : -1;
}

// ------------------------------------------------------------------ kernel

template <int BK, int KBC, bool SPAN, bool BF16, typename TO, bool RES>
__global__ void __launch_bounds__(THREADS, 1)
conv_tcgen05_kernel(const ConvTcParams p) {
  constexpr int RB = BK * 2;         // bytes per tile row
  constexpr int CH = RB / 16;        // 16-byte chunks per tile row
  constexpr int RPI = 32 / CH;       // tile rows covered by one warp-wide copy instruction
  constexpr int A_BYTES = BLOCK_M * RB;
  extern __shared__ uint8_t smem_raw[];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int G = p.G, BN = p.block_n, K = p.K, NBUF = p.nbuf;
  const int n0 = blockIdx.y * BN;
  const int KB = p.c_in / BK;
  const int B_BYTES = BN * RB;         // one weight tile
  constexpr int A_SLOT = KBC * A_BYTES;  // KBC channel slices per ring slot (KBC divides c_in / BK)
  const int B_SLOT = KBC * B_BYTES;
  const int ENTRIES = G * staged_lists(K);

  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t a_base = base;
  const uint32_t b_base = a_base + G * p.sa * A_SLOT;
  const uint32_t misc = b_base + p.sb * B_SLOT;
  uint8_t* misc_gen = gen + (misc - base);
  Control* ctl = reinterpret_cast<Control*>(misc_gen);
  int32_t* rows_idx = reinterpret_cast<int32_t*>(misc_gen + sizeof(Control));  // [ENTRIES][128]
  auto bar = [](uint64_t* b) { return smem_u32(b); };

  // One rendezvous behind the whole set-up (an earlier form, a thread at a time behind two, took 2 000 clocks: a microsecond
  // of each of the sixty launches of a small network).
  if (!p.claim) launch_dependents();
  // The index warps' share of a unit: 128 rows of one sub-tile in four warps (for a single sub-tile four take the even and
  // four the odd offsets).  The first unit's loads are on their way while the barriers are set up.
  const int itid = tid - EPI_THREADS, irow = itid & (BLOCK_M - 1);
  const uint32_t mine = G == 2 ? 0xFFFFFFFFu : itid >= BLOCK_M ? 0xAAAAAAAAu : 0x55555555u;   // this thread's offsets
  const bool single = !p.claim && (int64_t)gridDim.x >= p.units;                               // one unit per CTA
  int r[MAX_OFFSETS];
  int32_t out_row = -1;
  auto load_lists = [&](int64_t unit) {
    const int64_t st = p.S > 1 ? unit / p.S : unit;
    const uint32_t kmask = slice_mask((int)(unit - st * p.S), p.S) & mine;
    const int64_t m = (st * G + (G == 2 ? itid >> 7 : 0)) * BLOCK_M + irow;
    const int32_t* at = p.nbr + m;
#pragma unroll
    for (int k = 0; k < MAX_OFFSETS; ++k)
      r[k] = k < K && ((kmask >> k) & 1u) && m < p.M ? __ldg(at + (int64_t)k * p.M) : -1;
    out_row = m < p.M ? (p.out_rows ? __ldg(&p.out_rows[m]) : (int32_t)m) : -1;
  };
  const bool indexing = warp >= EPI_THREADS / 32 && warp < GATHER_WARP0;
  const int64_t first = p.S > 1 ? (int64_t)blockIdx.x : supertile_of(p, blockIdx.x);
  if (indexing) load_lists(first);
  const uint32_t tmem_total = (uint32_t)(NBUF * G * p.cols);
  if (warp == 0) {
    for (int g = 0; g < G; ++g)
      if (lane < p.sa) { mbar_init(bar(&ctl->a_full[g][lane]), GATHER_THREADS / G); mbar_init(bar(&ctl->a_empty[g][lane]), 1); }
    if (lane < p.sb) { mbar_init(bar(&ctl->b_full[lane]), 1); mbar_init(bar(&ctl->b_empty[lane]), G); }
    if (lane < 2) {
      for (int g = 0; g < G; ++g) { mbar_init(bar(&ctl->acc_full[lane][g]), 1); mbar_init(bar(&ctl->acc_empty[lane][g]), EPI_THREADS / G); }
      mbar_init(bar(&ctl->info_full[lane]), IDX_THREADS);
      mbar_init(bar(&ctl->info_empty[lane]), EPI_THREADS / 32 + G + 1 + GATHER_THREADS / 32);  // epilogue warps, MMA threads, weight thread, gather warps
    }
    if (lane == 2) mbar_init(bar(&ctl->claim_full), 1);
    if (lane < 3) ctl->mask_acc[lane][0] = ctl->mask_acc[lane][1] = 0;
    if (lane < 2) ctl->info_mask[0][lane] = 0;
    if (lane == 3) mbar_init(bar(&ctl->idx_sync), IDX_THREADS);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  } else if (warp == MMA_WARP) {
    tmem_alloc(smem_u32(&ctl->tmem_holder), tmem_total < 32 ? 32u : tmem_total);
  } else if (warp >= GATHER_WARP0 && warp < MMA_WARP) {
    for (int i = tid - GATHER_WARP0 * 32; i < BN; i += GATHER_THREADS) {
      ctl->sc[i] = p.scale ? __ldg(&p.scale[n0 + i]) : 1.f;
      ctl->sh[i] = p.shift ? __ldg(&p.shift[n0 + i]) : 0.f;
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  bool ok = true;
  const uint32_t tmem_base = ctl->tmem_holder;

  if (indexing) {
    // ================================================================ index warps
    // Choose the next unit and stage what the other roles need of it, one unit ahead of the copies: the output row of
    // every slot, the offsets each sub-tile has any neighbour at, and for each of those the 128 input rows (-1 where a row
    // has none), as row lists in a ring of G * K entries - room for two units of ordinary density, where two complete
    // tables would take another 27 KB from the row slots.  Only the offsets of the unit's slice are read; the others
    // are absent for every role.  An index that does not name a feature row is treated as absent and reported
    // (WCN_ERR_BOUNDS).
    // This role paces narrow layers (few bytes per unit), and what it waits for is latency: four warps per sub-tile (or,
    // for a single sub-tile, four for the even and four for the odd offsets), one vote per warp.  A CTA's first
    // unit and those of fixed strides are loaded before the wait for a free entry; a claimed unit waits for the entry, then for
    // the claim, then loads (see below what claims further ahead cost).  54 loads and 54 votes in four warps took 14 000 clocks per unit, three times
    // what the copies of a 32-channel layer take.
    const int g = G == 2 ? itid >> 7 : 0;
    const int num_in = (int)p.num_in;
    int sphase = 0, entry = 0, before = 0;   // next free entry; entries of the unit before
    int n = 0, acc = 0;                      // units staged; scratch of this unit's masks
    int cphase = 0;
    bool bad = false;
    int64_t unit = first, turn = blockIdx.x;
    if (single) {
      // A complete table of the one unit: nothing to compact, so the warps need not meet (a microsecond of the few that
      // such a launch takes).
      uint32_t has = 0;
#pragma unroll
      for (int k = 0; k < MAX_OFFSETS; ++k) {
        if (r[k] >= num_in) { r[k] = -1; bad = true; }
        has |= r[k] >= 0 ? 1u << k : 0u;
        if (k < K && ((mine >> k) & 1u)) rows_idx[(g * K + k) * BLOCK_M + irow] = r[k];
      }
      has = __reduce_or_sync(0xFFFFFFFFu, has);
      if (lane == 0 && has) atomicOr(&ctl->info_mask[0][g], has);
      if (mine & 1u) ctl->out_row[0][g * BLOCK_M + irow] = out_row;
      if (itid == 0) { ctl->info_unit[0] = unit; ctl->info_unit[1] = -1; }
      mbar_arrive(bar(&ctl->info_full[0]));
      mbar_arrive(bar(&ctl->info_full[1]));
      unit = -1;
    }
    while (ok && !single) {
      const int ib = n & 1;
      if (n > 0) {  // the unit after the one just staged
        if (!p.claim) {
          turn += gridDim.x;
          unit = turn < p.units ? supertile_of(p, turn) : -1;
        } else {
          // Not before the unit before last is done: a multiprocessor then holds the unit it works on and the next one, and
          // those that are left go to whoever is free.  (Claimed two ahead, the last units waited in the queues of busy
          // multiprocessors: with the order of the supertiles, 500 000 rows of 96 / 128 / 256 channels 143 / 187 / 547 -> 130 /
          // 170 / 499 us, 80 000 rows of 64 channels 38 -> 34.)
          if (!mbar_wait(bar(&ctl->info_empty[ib]), ((n >> 1) & 1) ^ 1, p.dev_status)) { ok = false; break; }
          if (itid == 0) {
            // (every index thread has read the last claim: they met since)
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            claim_next(bar(&ctl->claim[0]), bar(&ctl->claim_full));
          }
          // (a claim on its way writes this CTA's shared memory: it has to arrive before the CTA leaves)
          if (!mbar_wait(bar(&ctl->claim_full), cphase, p.dev_status)) {
            (void)mbar_wait(bar(&ctl->claim_full), cphase, p.dev_status);
            ok = false;
            break;
          }
          cphase ^= 1;
          unit = claimed_unit(ctl->claim);
          // (not before: the next launch's CTAs would be placed ahead of this grid's that have not started, and wait there
          // for the few multiprocessors left to it)
          if (unit < 0) launch_dependents();
          else unit = supertile_of(p, unit);
        }
      }
      if (unit < 0) {
        if (!mbar_wait(bar(&ctl->info_empty[ib]), ((n >> 1) & 1) ^ 1, p.dev_status)) { ok = false; break; }
        if (itid == 0) ctl->info_unit[ib] = -1;
        mbar_arrive(bar(&ctl->info_full[ib]));
        break;
      }
      if (n > 0) load_lists(unit);
      if (!mbar_wait(bar(&ctl->info_empty[ib]), ((n >> 1) & 1) ^ 1, p.dev_status)) { ok = false; break; }
      uint32_t has = 0;
#pragma unroll
      for (int k = 0; k < MAX_OFFSETS; ++k) {
        if (r[k] >= num_in) { r[k] = -1; bad = true; }
        has |= r[k] >= 0 ? 1u << k : 0u;
      }
      has = __reduce_or_sync(0xFFFFFFFFu, has);
      if (lane == 0 && has) atomicOr(&ctl->mask_acc[acc][g], has);
      if (mine & 1u) ctl->out_row[ib][g * BLOCK_M + irow] = out_row;
      // all index threads meet (bounded: a thread that gave up does not arrive, the others time out)
      mbar_arrive(bar(&ctl->idx_sync));
      if (!mbar_wait(bar(&ctl->idx_sync), sphase, p.dev_status)) { ok = false; break; }
      sphase ^= 1;
      const uint32_t m0 = ctl->mask_acc[acc][0], m1 = ctl->mask_acc[acc][1];
      // The scratch is used in turns of three: what is cleared here was read before this rendezvous and is next added to
      // after the following one.
      acc = acc == 2 ? 0 : acc + 1;
      if (itid == 0) { const int c = acc == 2 ? 0 : acc + 1; ctl->mask_acc[c][0] = ctl->mask_acc[c][1] = 0; }
      const int need = __popc(m0) + __popc(m1);
      // the entries of the unit before last are free (info_empty above); those of the last unit only if it has been read
      if (before + need > ENTRIES && !mbar_wait(bar(&ctl->info_empty[ib ^ 1]), ((n - 1) >> 1) & 1, p.dev_status)) { ok = false; break; }
      before = need;
      int second = entry + __popc(m0);
      if (second >= ENTRIES) second -= ENTRIES;
      if (itid == 0) {
        ctl->info_unit[ib] = unit;
        ctl->info_mask[ib][0] = m0;
        ctl->info_mask[ib][1] = m1;
        ctl->info_entry[ib][0] = entry;
        ctl->info_entry[ib][1] = second;
      }
      const uint32_t own = g == 0 ? m0 : m1;
      int32_t* at = rows_idx + (g == 0 ? entry : second) * BLOCK_M + irow;
      int32_t* const end = rows_idx + ENTRIES * BLOCK_M;
#pragma unroll
      for (int k = 0; k < MAX_OFFSETS; ++k) {
        if ((own >> k) & 1u) {
          if ((mine >> k) & 1u) *at = r[k];
          at += BLOCK_M;
          if (at >= end) at -= ENTRIES * BLOCK_M;
        }
      }
      entry = second + __popc(m1);
      if (entry >= ENTRIES) entry -= ENTRIES;
      mbar_arrive(bar(&ctl->info_full[ib]));  // (256 arrivals publish the lists)
      ++n;
    }
    if (bad) wcn_report_bounds(p.dev_status);
  } else if (warp == WEIGHT_WARP) {
    // ================================================================ weight loader
    if (elect_one()) {
      Ring rb{0, 0, p.sb};
      for (int n = 0; ok; ++n) {
        const int ib = n & 1;
        if (!mbar_wait(bar(&ctl->info_full[ib]), (n >> 1) & 1, p.dev_status)) { ok = false; break; }
        const bool last = ctl->info_unit[ib] < 0;
        uint32_t rest = ctl->info_mask[ib][0] | ctl->info_mask[ib][1];
        mbar_arrive(bar(&ctl->info_empty[ib]));  // only the masks were needed
        if (last) break;
        // One channel slice per offset (KB == 1) and KBC > 1: a ring slot spans KBC consecutive
        // ACTIVE OFFSETS instead of KBC channel slices of one offset, so narrow layers get the same
        // fat slots as wide ones.  All roles take the offsets off the mask in the same groups.
        while (SPAN && rest && ok) {
          int ku[KBC];
          const int nu = pop_offsets<KBC>(rest, ku);
          if (!mbar_wait(bar(&ctl->b_empty[rb.slot]), rb.phase ^ 1, p.dev_status)) { ok = false; break; }
          const uint32_t fullb = bar(&ctl->b_full[rb.slot]);
          mbar_expect_tx(fullb, (uint32_t)(nu * B_BYTES));
#pragma unroll
          for (int u = 0; u < KBC; ++u)
            if (ku[u] >= 0)
              bulk_copy_g2s(b_base + rb.slot * B_SLOT + u * B_BYTES,
                            p.wpacked + ((int64_t)ku[u] * p.c_out + n0) * RB, (uint32_t)B_BYTES, fullb);
          rb.advance();
        }
        while (!SPAN && rest && ok) {
          const int k = __ffs(rest) - 1;
          rest &= rest - 1;
          const char* bsrc_k = p.wpacked + ((int64_t)k * KB * p.c_out + n0) * RB;
          for (int kb0 = 0; kb0 < KB; kb0 += KBC) {
            // weight tiles (offset k, channel slices kb0..): bulk copies onto one barrier, shared by all sub-tiles
            if (!mbar_wait(bar(&ctl->b_empty[rb.slot]), rb.phase ^ 1, p.dev_status)) { ok = false; break; }
            const uint32_t fullb = bar(&ctl->b_full[rb.slot]);
            mbar_expect_tx(fullb, (uint32_t)(KBC * B_BYTES));
#pragma unroll
            for (int u = 0; u < KBC; ++u)
              bulk_copy_g2s(b_base + rb.slot * B_SLOT + u * B_BYTES, bsrc_k + (int64_t)(kb0 + u) * p.c_out * RB,
                            (uint32_t)B_BYTES, fullb);
            rb.advance();
          }
        }
      }
    }
    __syncwarp();
  } else if (warp >= GATHER_WARP0 && warp < MMA_WARP) {
    // ================================================================ gather warps
    // Four warps and a ring of row slots per sub-tile (all eight for the one sub-tile of a small problem).
    wait_for_primary();  // the feature rows are the previous launch's
    const int gwarp = warp - GATHER_WARP0;
    const int g = G == 2 ? gwarp >> 2 : 0;
    const int row0 = G == 2 ? (gwarp & 3) * 32 : gwarp * 16;  // this warp's 32 (16) rows of the tile
    constexpr int NJ = 16 / RPI;                               // copy instructions per 16 rows and channel slice
    const int sub_row = lane / CH, chunk = lane % CH;
    uint32_t aoff[2 * NJ];  // this thread's fixed (row, chunk) positions inside an A tile
#pragma unroll
    for (int j = 0; j < 2 * NJ; ++j) aoff[j] = tile_offset<RB>((row0 + j * RPI + sub_row) & (BLOCK_M - 1), chunk);
    const char* feats = p.feats + chunk * 16;
    const int valid = p.row_bytes - chunk * 16;   // a slice that starts at or beyond it has no channels for this thread
    Ring ra{0, 0, p.sa};
    const uint32_t ring = a_base + g * p.sa * A_SLOT;
    for (int n = 0; ok; ++n) {
      const int ib = n & 1;
      if (!mbar_wait(bar(&ctl->info_full[ib]), (n >> 1) & 1, p.dev_status)) { ok = false; break; }
      if (ctl->info_unit[ib] < 0) break;
      const uint32_t own = ctl->info_mask[ib][g];
      uint32_t rest = SPAN ? own | ctl->info_mask[ib][1] | ctl->info_mask[ib][0] : own;
      int e = ctl->info_entry[ib][g];
      const int32_t* tab = rows_idx + row0 + sub_row;
      // the addresses of this thread's rows, and which of them are there
      auto rows_of = [&](int entry, const char* (&src)[2 * NJ], uint32_t& have) {
        have = 0;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (h < G) {
#pragma unroll
            for (int j = h * NJ; j < (h + 1) * NJ; ++j) {
              const int r = tab[entry * BLOCK_M + j * RPI];
              have |= (r >= 0 ? 1u : 0u) << j;
              src[j] = feats + (int64_t)max(r, 0) * p.in_ld_bytes;
            }
          }
        }
      };
      auto copy = [&](uint32_t dst, const char* const (&src)[2 * NJ], uint32_t have, int at) {
        if (BK == 32 && at >= valid) { have = 0; at = 0; }   // (rows that fill their slices to the end run with BK = 64 too)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (h < G) {
#pragma unroll
            for (int j = h * NJ; j < (h + 1) * NJ; ++j)
              cp_async16(dst + aoff[j], src[j] + at, ((have >> j) & 1u) * 16u);
          }
        }
      };
      while (SPAN && rest && ok) {  // slots that span offsets (see the weight loader)
        int ku[KBC];
        pop_offsets<KBC>(rest, ku);
        uint32_t used = 0;
#pragma unroll
        for (int u = 0; u < KBC; ++u)
          if (ku[u] >= 0) used |= ((own >> ku[u]) & 1u) << u;
        if (!used) continue;
        if (!mbar_wait(bar(&ctl->a_empty[g][ra.slot]), ra.phase ^ 1, p.dev_status)) { ok = false; break; }
        const uint32_t dst = ring + ra.slot * A_SLOT;
#pragma unroll
        for (int u = 0; u < KBC; ++u) {
          if ((used >> u) & 1u) {  // parts of offsets this sub-tile does not have stay unused
            const char* src[2 * NJ];
            uint32_t have;
            rows_of(single ? g * K + ku[u] : e, src, have);
            if (++e == ENTRIES) e = 0;
            copy(dst + u * A_BYTES, src, have, 0);
          }
        }
        cp_async_arrive(bar(&ctl->a_full[g][ra.slot]));
        ra.advance();
      }
      while (!SPAN && rest && ok) {
        const int k = __ffs(rest) - 1;
        rest &= rest - 1;
        const char* src[2 * NJ];
        uint32_t have;
        rows_of(single ? g * K + k : e, src, have);
        if (++e == ENTRIES) e = 0;
        for (int kb0 = 0; kb0 < KB; kb0 += KBC) {
          if (!mbar_wait(bar(&ctl->a_empty[g][ra.slot]), ra.phase ^ 1, p.dev_status)) { ok = false; break; }
          const uint32_t dst = ring + ra.slot * A_SLOT;
#pragma unroll
          for (int u = 0; u < KBC; ++u)  // the row's next channel slices are contiguous in memory
            copy(dst + u * A_BYTES, src, have, (kb0 + u) * RB);
          cp_async_arrive(bar(&ctl->a_full[g][ra.slot]));  // hardware arrives when this thread's copies land
          ra.advance();
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(&ctl->info_empty[ib]));  // this warp is done with the staged lists
    }
    cp_async_drain();
  } else if (warp >= MMA_WARP && warp < MMA_WARP + MMA_ISSUERS) {
    // ================================================================ MMA issuers
    // One thread per sub-tile.  They share the weight slots - both observe and release every one, because a parity wait is
    // only meaningful for a thread that is never a whole lap away - and nothing else.  A barrier operation costs a single
    // thread 50 to 100 clocks even when it succeeds at once, so the next slots' barriers are looked at before this slot's
    // instructions are issued.
    const int g = warp - MMA_WARP;
    if (g < G && elect_one()) {
      const uint32_t idesc = (1u << 4) | ((BF16 ? 1u : 0u) << 7) | ((BF16 ? 1u : 0u) << 10) |
                             ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BLOCK_M >> 4) << 24);
      Ring ra{0, 0, p.sa}, rb{0, 0, p.sb};
      const uint32_t ring = a_base + g * p.sa * A_SLOT;
      bool a_ready = false, b_ready = false;
      int ab = 0, aphase = 0;
      for (int n = 0; ok; ++n) {
        const int ib = n & 1;
        if (!mbar_wait(bar(&ctl->info_full[ib]), (n >> 1) & 1, p.dev_status)) { ok = false; break; }
        const bool last = ctl->info_unit[ib] < 0;
        const uint32_t own = ctl->info_mask[ib][g];
        uint32_t rest = own | ctl->info_mask[ib][0] | ctl->info_mask[ib][1];
        mbar_arrive(bar(&ctl->info_empty[ib]));  // only the masks were needed
        if (last) break;
        // the accumulator must have been read out by the epilogue of its previous use
        if (!mbar_wait(bar(&ctl->acc_empty[ab][g]), aphase ^ 1, p.dev_status)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d = tmem_base + (uint32_t)((ab * G + g) * p.cols);
        uint32_t acc = 0;
        while (rest && ok) {
          int ku[SPAN ? KBC : 1];
          uint32_t used = 0;
          pop_offsets<SPAN ? KBC : 1>(rest, ku);
#pragma unroll
          for (int u = 0; u < (SPAN ? KBC : 1); ++u)
            if (ku[u] >= 0) used |= ((own >> ku[u]) & 1u) << u;
          for (int kb0 = 0; kb0 < (SPAN ? 1 : KB); kb0 += KBC) {
            if (!b_ready && !mbar_wait(bar(&ctl->b_full[rb.slot]), rb.phase, p.dev_status)) { ok = false; break; }
            const uint64_t bdesc = smem_desc<RB>(b_base + rb.slot * B_SLOT);
            const uint32_t b_free = bar(&ctl->b_empty[rb.slot]);
            rb.advance();
            if (!used) {  // this sub-tile has none of the slot's offsets
              mbar_arrive(b_free);
              b_ready = mbar_test(bar(&ctl->b_full[rb.slot]), rb.phase);
              continue;
            }
            if (!a_ready && !mbar_wait(bar(&ctl->a_full[g][ra.slot]), ra.phase, p.dev_status)) { ok = false; break; }
            tc_fence_after();
            const uint64_t adesc = smem_desc<RB>(ring + ra.slot * A_SLOT);
            const uint32_t a_free = bar(&ctl->a_empty[g][ra.slot]);
            ra.advance();
            a_ready = mbar_test(bar(&ctl->a_full[g][ra.slot]), ra.phase);
            b_ready = mbar_test(bar(&ctl->b_full[rb.slot]), rb.phase);
#pragma unroll
            for (int u = 0; u < KBC; ++u) {
              if (!SPAN || ((used >> u) & 1u)) {
#pragma unroll
                for (int kk = 0; kk < BK / 16; ++kk)
                  umma_f16(d, adesc + (uint64_t)(u * (A_BYTES >> 4) + kk * 2), bdesc + (uint64_t)(u * (B_BYTES >> 4) + kk * 2),
                           idesc, acc | (kk > 0 ? 1u : 0u));
                acc = 1u;
              }
            }
            umma_commit(a_free);  // the slots are free once these instructions have read them
            umma_commit(b_free);
          }
        }
        if (acc && ok) umma_commit(bar(&ctl->acc_full[ab][g]));  // the sub-tile's accumulator is complete
        else mbar_arrive(bar(&ctl->acc_full[ab][g]));
        if (++ab == NBUF) { ab = 0; aphase ^= 1; }
      }
    }
    __syncwarp();
  } else {
    // ================================================================ epilogue (warps 0..7)
    // Four warps per sub-tile; with a single sub-tile the second four take the upper half of its columns.  A load issued by
    // these warps waits its turn behind the gather's copies (2 000 to 5 000 clocks), so the residual of 64 columns is
    // requested at once, the first of them before the wait for the accumulators: one row at a time in four warps, 32
    // columns by 32, the residual of a 96-channel layer cost a quarter of its time.
    wait_for_primary();
    // (a launch that overlaps the one before it may have started before that one failed)
    const bool poison = *(volatile const int32_t*)p.dev_status == (int)WCN_ERR_WAIT_EXPIRED;
    const int half = warp >> 2, g = G == 2 ? half : 0, row = tid & (BLOCK_M - 1);
    const int middle = ((BN / 16 + 1) / 2) * 16;
    const int c_begin = G == 2 || half == 0 ? 0 : middle, c_end = G == 2 || half == 1 ? BN : middle;
    constexpr int CHUNK = RES && sizeof(TO) == 2 ? 64 : 32;   // columns per turn (whose residual is held in registers)
    constexpr int PIECE = RES ? 16 : 32;                       // columns per tensor-memory load
    int ab = 0, aphase = 0;
    const bool affine = p.scale != nullptr || p.shift != nullptr;
    for (int n = 0; ok; ++n) {
      const int ib = n & 1;
      ok = mbar_wait(bar(&ctl->info_full[ib]), (n >> 1) & 1, p.dev_status);
      if (!__all_sync(0xFFFFFFFFu, ok)) { ok = false; break; }
      const bool last = ctl->info_unit[ib] < 0;
      const bool any = ctl->info_mask[ib][g] != 0;
      // This thread's output row (-1 past the end), loaded by the index warps: another latency that is not paid here.
      const int64_t m = ctl->out_row[ib][g * BLOCK_M + row];
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(&ctl->info_empty[ib]));
      if (last) break;
      if (p.S > 1) continue;  // the slices' sums are finished behind the roles
      const bool live = m >= 0;
      const uint32_t trow = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)((ab * G + g) * p.cols);
      TO* orow = reinterpret_cast<TO*>(p.out) + m * p.out_ld + n0;
      const TO* rrow = RES && live ? reinterpret_cast<const TO*>(p.residual) + m * p.res_ld + n0 : nullptr;
      bool ready = false;
#pragma unroll 1
      for (int cb = c_begin; cb < c_end || !ready; cb += CHUNK) {  // (a half without columns waits all the same)
        __align__(32) TO res[CHUNK];
        if (rrow) {
#pragma unroll
          for (int q = 0; q < CHUNK; q += 16)
            if (cb + q < c_end) load_raw16(rrow + cb + q, res + q, p.wide_res);
        }
        if (!ready) {
          // tcgen05.ld is warp-collective, so the decision to read must be warp-uniform
          ok = mbar_wait(bar(&ctl->acc_full[ab][g]), aphase, p.dev_status);
          if (!__all_sync(0xFFFFFFFFu, ok)) { ok = false; break; }
          tc_fence_after();
          ready = true;
        }
#pragma unroll
        for (int q = 0; q < CHUNK; q += PIECE) {
          const int c0 = cb + q;
          if (c0 >= c_end) break;
          uint32_t r[PIECE / 16][16];
          if (any) {
#pragma unroll
            for (int h = 0; h < PIECE / 16; ++h)
              if (h == 0 || c0 + 16 < c_end) tmem_ld16(trow + (uint32_t)(c0 + 16 * h), r[h]);  // executed by all lanes of the warp
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int h = 0; h < PIECE / 16; ++h)
#pragma unroll
              for (int i = 0; i < 16; ++i) r[h][i] = 0u;
          }
          if (live) {
#pragma unroll
            for (int h = 0; h < PIECE / 16; ++h) {
              const int c = c0 + 16 * h;
              if (h > 0 && c >= c_end) break;
              // affine, residual, ReLU, convert, store
              float y[16];
#pragma unroll
              for (int i = 0; i < 16; ++i) y[i] = __uint_as_float(r[h][i]);
              if (affine) {
#pragma unroll
                for (int i = 0; i < 16; i += 4) {
                  const float4 s4 = *reinterpret_cast<const float4*>(&ctl->sc[c + i]);
                  const float4 h4 = *reinterpret_cast<const float4*>(&ctl->sh[c + i]);
                  y[i + 0] = fmaf(y[i + 0], s4.x, h4.x);
                  y[i + 1] = fmaf(y[i + 1], s4.y, h4.y);
                  y[i + 2] = fmaf(y[i + 2], s4.z, h4.z);
                  y[i + 3] = fmaf(y[i + 3], s4.w, h4.w);
                }
              }
              if (RES) {
#pragma unroll
                for (int i = 0; i < 16; ++i) y[i] += wcn_to_float<TO>(res[q + i]);
              }
              if (p.relu) {
#pragma unroll
                for (int i = 0; i < 16; ++i) y[i] = fmaxf(y[i], 0.f);
              }
              if (poison) {
#pragma unroll
                for (int i = 0; i < 16; ++i) y[i] = __int_as_float(0x7FC00000);
              }
              store16<TO>(orow + c, y, p.wide_out);
            }
          }
        }
      }
      if (!ok) break;
      tc_fence_before();
      mbar_arrive(bar(&ctl->acc_empty[ab][g]));   // the accumulator may be overwritten
      if (++ab == NBUF) { ab = 0; aphase ^= 1; }
    }
  }
  if (p.S > 1) {
    // ================================================================ the cluster adds its slices
    // Eight warps leave this slice's sums in shared memory, where the ring was (every slot has been consumed); then each CTA
    // finishes 1 / S of the rows.  Reading 128 x BN sums from the other CTAs is what this costs, so every CTA starts with
    // its own slice and goes round: all starting with slice 0 made one multiprocessor serve the whole cluster.  They are
    // added in slice order, whichever CTA finishes the row: the sum does not depend on where the row lies in its tile.
    __syncwarp();
    if (warp < 8) {
      bool have = __all_sync(0xFFFFFFFFu, ok);
      if (have) have = mbar_wait(bar(&ctl->acc_full[0][0]), 0, p.dev_status);
      if (__all_sync(0xFFFFFFFFu, have)) {
        tc_fence_after();
        const bool any = ctl->info_mask[0][0] != 0;
        const int q = warp & 3;
        float* prow = reinterpret_cast<float*>(gen) + (q * 32 + lane) * (BN + 4);
#pragma unroll 1
        for (int c0 = (warp >> 2) * 16; c0 < BN; c0 += 32) {
          uint32_t r[16];
          if (any) {
            tmem_ld16(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)c0, r);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) r[i] = 0u;
          }
#pragma unroll
          for (int i = 0; i < 16; i += 4) *reinterpret_cast<uint4*>(prow + c0 + i) = make_uint4(r[i], r[i + 1], r[i + 2], r[i + 3]);
        }
      }
    }
    cluster_meet();  // every slice's sums are in its CTA's shared memory
    const int32_t status = *(volatile const int32_t*)p.dev_status;
    const int64_t st = blockIdx.x / p.S;
    const int rank = (int)(blockIdx.x - st * p.S), per_row = BN / 4;
    const int r0 = rank * BLOCK_M / p.S, r1 = (rank + 1) * BLOCK_M / p.S;
    for (int i = tid; i < (r1 - r0) * per_row; i += THREADS) {
      const int r = r0 + i / per_row, c = (i % per_row) * 4;
      const int64_t slot = st * BLOCK_M + r;
      if (slot >= p.M) break;  // rows ascend with i
      const int64_t m = p.out_rows ? (int64_t)__ldg(&p.out_rows[slot]) : slot;
      const uint32_t at = base + (uint32_t)(r * (BN + 4) + c) * 4u;
      float4 v[MAX_SLICES];
#pragma unroll
      for (int s = 0; s < MAX_SLICES; ++s)
        if (s < p.S && s >= rank) v[s] = ld_cluster(at, (uint32_t)s);
#pragma unroll
      for (int s = 0; s < MAX_SLICES; ++s)
        if (s < rank) v[s] = ld_cluster(at, (uint32_t)s);
      __align__(16) TO o[4], res[4];
      if (RES) {
        const TO* rrow = reinterpret_cast<const TO*>(p.residual) + m * p.res_ld + n0 + c;
        if (sizeof(TO) == 4) *reinterpret_cast<uint4*>(res) = __ldg(reinterpret_cast<const uint4*>(rrow));
        else *reinterpret_cast<uint2*>(res) = __ldg(reinterpret_cast<const uint2*>(rrow));
      }
      float y[4] = {v[0].x, v[0].y, v[0].z, v[0].w};
#pragma unroll
      for (int s = 1; s < MAX_SLICES; ++s) {
        if (s < p.S) {
          y[0] = __fadd_rn(y[0], v[s].x); y[1] = __fadd_rn(y[1], v[s].y);
          y[2] = __fadd_rn(y[2], v[s].z); y[3] = __fadd_rn(y[3], v[s].w);
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        y[j] = fmaf(y[j], ctl->sc[c + j], ctl->sh[c + j]);  // (1 and 0 when there is no affine step)
        if (RES) y[j] += wcn_to_float<TO>(res[j]);
        if (p.relu) y[j] = fmaxf(y[j], 0.f);
        if (status == (int)WCN_ERR_WAIT_EXPIRED) y[j] = __int_as_float(0x7FC00000);
        o[j] = wcn_from_float<TO>(y[j]);
      }
      TO* dst = reinterpret_cast<TO*>(p.out) + m * p.out_ld + n0 + c;
      if (sizeof(TO) == 4) *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(o);
      else *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(o);
    }
    cluster_meet();  // no CTA leaves while another may read its sums
  }
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) tmem_dealloc(tmem_base, tmem_total < 32 ? 32u : tmem_total);
}

// weight -> packed[K][c_in/BK] tiles of [c_out][BK]: every (offset, channel slice) becomes one contiguous K-major tile
// stored as its swizzled shared-memory image (the layout of tile_offset above), so the kernel moves it with a single bulk
// copy.  A thread makes one 16-byte chunk: eight input channels of one output channel.  The source may have another
// dtype, be transposed per offset ([K, c_out, c_in]) and hold the offsets in reverse order: what a training step needs
// of its fp32 weights each time they change, without a cast or a transposed copy in between.
template <typename TS, typename TD>
__global__ void pack_weight_kernel(const TS* __restrict__ w, TD* __restrict__ packed, int K, int c_in, int c_out, int bk,
                                   int transposed, int reversed) {
  const int pad = (c_in + 31) / 32 * 32;   // channels c_in .. pad - 1 are zeros
  const int64_t total = (int64_t)K * (pad / 8) * c_out;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  // consecutive threads run along the dimension that is contiguous in the source
  int n, c8;
  int64_t r;
  if (transposed) { c8 = (int)(i % (pad / 8)); r = i / (pad / 8); n = (int)(r % c_out); r /= c_out; }
  else { n = (int)(i % c_out); r = i / c_out; c8 = (int)(r % (pad / 8)); r /= pad / 8; }
  const int k = (int)r, cin = c8 * 8;
  const int64_t ks = reversed ? K - 1 - k : k;
  __align__(16) TD v[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const int64_t at = transposed ? (ks * c_out + n) * c_in + cin + u : (ks * c_in + cin + u) * c_out + n;
    v[u] = wcn_from_float<TD>(cin + u < c_in ? wcn_to_float<TS>(w[at]) : 0.f);
  }
  const int kb = cin / bk, c = cin % bk;
  const int rb = bk * 2, chunk = c >> 3, r8 = n & 7;
  const int x = rb == 128 ? r8 : (r8 >> 1);
  const int64_t tile = ((int64_t)k * (pad / bk) + kb) * c_out * bk;  // elements
  const int64_t off_bytes = (int64_t)(n >> 3) * (8 * rb) + r8 * rb + ((chunk ^ x) << 4);
  *reinterpret_cast<uint4*>(packed + tile + off_bytes / 2) = *reinterpret_cast<const uint4*>(v);
}

inline int padded(int c_in) { return (c_in + 31) / 32 * 32; }
// (the check for channels beyond the row cost the BK = 64 form 2 % of a 256-channel layer: it has none)
inline int pick_bk(int c_in) { return c_in % 64 == 0 ? 64 : 32; }

// CTAs that can be resident at once in clusters of S (they stay inside a group of multiprocessors, whose sizes differ).
int resident_ctas(int S) {
  static std::atomic<int> known[64][MAX_SLICES + 1];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return wcn_num_sms();
  if (S == 1) return wcn_num_sms();
  int n = known[dev][S].load(std::memory_order_relaxed);
  if (n == 0) {
    auto kern = conv_tcgen05_kernel<64, 1, false, false, __half, false>;  // (one CTA per multiprocessor, like every instance)
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned)S;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)S);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = SMEM_LIMIT;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_LIMIT) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) != cudaSuccess || clusters < 1) {
      (void)cudaGetLastError();
      clusters = wcn_num_sms() / (2 * S);
    }
    n = clusters * S;
    known[dev][S].store(n, std::memory_order_relaxed);
  }
  return n;
}

// Launch geometry.  A problem with fewer 128-row tiles than multiprocessors cannot occupy the GPU with one CTA per tile:
// its kernel offsets are divided among S CTAs of a cluster and its output columns among blocks of their own (which gather
// the rows again), whichever combination of the two is expected to take least (split_k: 0 = decide here, 1 = columns only,
// >= 2 = that many slices, at most eight; < 0 = -split_k column blocks).
//
// The model: a CTA reads n_off * (A + B) bytes, A = its 128 rows, B = its columns' weights at one offset, at the ~68 KB/us
// that one multiprocessor sustains; of K offsets about 0.6 K have a neighbour in a tile; adding the slices costs 1.3 us and
// 0.0165 us per column (128 sums of every column come through the cluster's network).  Within 1.5 us of the best of all
// combinations for 128 to 9 000 rows and 32 to 256 channels.
void pick_split(const ConvTcParams& p, int64_t tiles, int split_k, int* slices, int* blocks) {
  *slices = *blocks = 1;
  double best = 1e30;
  for (int S = 1; S <= MAX_SLICES && S <= p.K; ++S) {
    if (split_k == 1 && S > 1) break;
    const int64_t fit = resident_ctas(S);
    for (int nb = 1; nb <= 8; nb *= 2) {
      if (p.c_out % (16 * nb) != 0 || (nb > 1 && p.c_out / nb < 32)) break;
      const int64_t ctas = tiles * S * nb;
      if (ctas > fit && ctas > tiles) continue;
      const double off = (p.K > 2 ? 0.6 * p.K : p.K) / S;
      const double bytes = (off < 1 ? 1 : off) * 2.0 * p.c_in * (BLOCK_M + p.c_out / nb);
      const double us = bytes / 68e3 + (S > 1 ? 1.3 + 0.0165 * (p.c_out / nb) : 0.0);
      if (us < best) { best = us; *slices = S; *blocks = nb; }
    }
  }
}

bool plan_launch(ConvTcParams& p, int bk, int split_k, size_t* smem, dim3* grid) {
  const int sms = wcn_num_sms();
  const int64_t tiles = (p.M + BLOCK_M - 1) / BLOCK_M;
  int S = 1, split = 1;
  if (split_k >= 2) {
    S = split_k < MAX_SLICES ? split_k : MAX_SLICES;
    if (S > p.K) S = p.K;
  } else if (split_k < 0) {
    split = -split_k;
    if (split > 16 || p.c_out % (16 * split) != 0) return false;
  } else if (tiles * 2 <= sms) {
    pick_split(p, tiles, split_k, &S, &split);
  }
  p.S = S;
  p.block_n = p.c_out / split;
  int cols = 32;
  while (cols < p.block_n) cols <<= 1;
  p.cols = cols;
  // Two sub-tiles per supertile (one per issuer).  Four were used for narrow outputs once, to share a weight
  // slice among more rows; narrow layers have tiny weights, and the two extra staged tables (55 KB) are worth
  // more as row slots: 3x3x3 C = 32 / 64 layers measured 11 % faster with two.
  int g = S > 1 ? 1 : 2;
  while (g > 1 && ((tiles + g - 1) / g) * split * S < 2 * (int64_t)sms) g /= 2;
  const size_t a_unit = (size_t)BLOCK_M * bk * 2, b_unit = (size_t)p.block_n * bk * 2;
  const size_t limit = SMEM_LIMIT;
  const int kb_total = p.c_in / bk;
  // Channel slices per ring slot: as many as give a 32 KiB row slot, fewer if the rings would not fit.
  // (with a single slice per offset the slot spans that many active offsets instead)
  int kbc = (int)(32 * 1024 / a_unit);
  if (kb_total > 1 && kbc > kb_total) kbc = kb_total;
  if (kb_total == 1 && kbc > p.K) kbc = p.K;
  if (kbc < 1) kbc = 1;
  while (kb_total > 1 && kb_total % kbc != 0) --kbc;
  size_t fixed = 0, a_stage = 0, b_stage = 0;
  for (;;) {  // the staged row lists and two slots of every ring must fit
    fixed = 1024 + sizeof(Control) + (size_t)g * staged_lists(p.K) * BLOCK_M * 4 + 128;
    a_stage = g * kbc * a_unit;
    b_stage = kbc * b_unit;
    if (fixed + 2 * a_stage + 2 * b_stage <= limit) break;
    if (kbc > 1) {
      do { --kbc; } while (kb_total > 1 && kb_total % kbc != 0);
      continue;
    }
    if (g == 1) return false;
    g /= 2;
  }
  p.kbc = kbc;
  p.G = g;
  p.nbuf = (g * cols * 2 <= 512) ? 2 : 1;
  p.supertiles = (tiles + g - 1) / g;
  p.units = p.supertiles * S;
  // Row slots first up to three per sub-tile, then a third weight slot (with two, the fetch of one waits for the last
  // instruction on the other), then whatever still fits.
  int sa = 2, sb = 2;
  for (;;) {
    const size_t used = fixed + sa * a_stage + sb * b_stage;
    const bool more_a = sa < MAX_RING && used + a_stage <= limit, more_b = sb < 6 && used + b_stage <= limit;
    if (more_a && (sa < 3 || (sb >= 3 && (sa < 4 || sb >= 4 || !more_b)))) ++sa;
    else if (more_b) ++sb;
    else if (more_a) ++sa;
    else break;
  }
  p.sa = sa;
  p.sb = sb;
  // the sums of a slice take the place of the rings
  if (S > 1 && sa * a_stage + sb * b_stage < (size_t)BLOCK_M * (p.block_n + 4) * 4) return false;
  *smem = fixed + sa * a_stage + sb * b_stage;
  // Where there are more units than multiprocessors one CTA per unit is launched, and the first to start claim the rest (the
  // network over 2 x 100 000 voxels 1 701 -> 1 602 us against fixed strides below four units per multiprocessor and claims
  // two ahead above).  Few units of rows in no tile order take much the same time and keep the fixed strides (2x2x2 down
  // and up of 300 000 rows 60.9 us, 61.4 with claims).  Column blocks are made of problems that fit at once; asked for on
  // larger ones, their CTAs keep the strides: a claim could return another block's.
  int64_t gx = p.units;
  const int64_t cap = sms / split > 0 ? sms / split : 1;
  p.claim = S == 1 && split == 1 && (p.out_rows ? gx > cap : gx >= 4 * cap);
  if (gx > cap && S == 1 && !p.claim) gx = cap;
  p.window = p.out_rows && S == 1 ? tile_window(p.M, wcn_overlap_launches) / (g * BLOCK_M) : 0;
  p.tail = 0;
  if (p.window > 0) {
    const int64_t whole = p.supertiles / p.window;
    p.tail = (int)(whole < TAIL_WINDOWS ? whole : TAIL_WINDOWS);
  }
  *grid = dim3((unsigned)gx, (unsigned)split);
  return true;
}

template <int BK, int KBC, bool SPAN, bool BF16, typename TO, bool RES>
int launch_kernel(const ConvTcParams& p, size_t smem, dim3 grid, cudaStream_t st) {
  auto kern = conv_tcgen05_kernel<BK, KBC, SPAN, BF16, TO, RES>;
  static bool configured[64] = {};  // per template instance and device: opt in to large shared memory once
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return WCN_ERR_INITIALIZATION;
  if (!configured[dev]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_LIMIT) != cudaSuccess) {
      (void)cudaGetLastError();  // do not leave a sticky error for the caller's next CUDA call
      return WCN_ERR_INITIALIZATION;
    }
    configured[dev] = true;
  }
  return wcn_launch(kern, grid, dim3(THREADS), smem, st, (unsigned)p.S, p);
}

template <int BK, int KBC, bool SPAN, bool BF16, typename TO>
int launch_kbc(const ConvTcParams& p, size_t smem, dim3 grid, cudaStream_t st) {
  return p.residual ? launch_kernel<BK, KBC, SPAN, BF16, TO, true>(p, smem, grid, st)
                    : launch_kernel<BK, KBC, SPAN, BF16, TO, false>(p, smem, grid, st);
}

template <int BK, bool BF16, typename TO>
int launch_tc(ConvTcParams& p, int split_k, cudaStream_t st) {
  size_t smem = 0;
  dim3 grid;
  if (!plan_launch(p, BK, split_k, &smem, &grid)) return WCN_ERR_UNSUPPORTED_CONFIG;
  // SPAN: the whole C_in is one slice and a ring slot holds KBC consecutive active offsets; otherwise a
  // slot holds KBC channel slices of one offset.  A compile-time choice, so that every role's loop
  // carries only the form it runs.  (A slot holds at most 32 KiB: two slices of 64 channels, four of 32.)
  if (p.kbc > 1 && p.c_in == BK) {
    if (p.kbc == 2) return launch_kbc<BK, 2, true, BF16, TO>(p, smem, grid, st);
    if constexpr (BK == 32) {
      if (p.kbc == 3) return launch_kbc<BK, 3, true, BF16, TO>(p, smem, grid, st);
      if (p.kbc == 4) return launch_kbc<BK, 4, true, BF16, TO>(p, smem, grid, st);
    }
    return WCN_ERR_UNSUPPORTED_CONFIG;
  }
  if (p.kbc == 1) return launch_kbc<BK, 1, false, BF16, TO>(p, smem, grid, st);
  if (p.kbc == 2) return launch_kbc<BK, 2, false, BF16, TO>(p, smem, grid, st);
  if constexpr (BK == 32) {
    if (p.kbc == 3) return launch_kbc<BK, 3, false, BF16, TO>(p, smem, grid, st);
    if (p.kbc == 4) return launch_kbc<BK, 4, false, BF16, TO>(p, smem, grid, st);
  }
  return WCN_ERR_UNSUPPORTED_CONFIG;
}

// A barrier phase that cannot complete (one arrival of two), waited for with a short limit:
// the wait has to give up, report WCN_ERR_WAIT_EXPIRED and let the kernel end normally.
__global__ void bounded_wait_probe_kernel(long long limit_cycles, int32_t* dev_status, int32_t* gave_up) {
  __shared__ uint64_t probe_bar;
  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&probe_bar), 2);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0) mbar_arrive(smem_u32(&probe_bar));
  if (threadIdx.x == 32) {
    const bool done = mbar_wait_limit(smem_u32(&probe_bar), 0, dev_status, limit_cycles);
    if (gave_up) *gave_up = done ? 0 : 1;
  }
}

}  // namespace

extern "C" int wcn_selftest_bounded_wait(int64_t limit_cycles, int32_t* dev_status, int32_t* gave_up, void* stream) {
  if (!dev_status || limit_cycles < 1000 || limit_cycles > 2000000000ll) return WCN_ERR_INVALID_PARAMETERS;
  bounded_wait_probe_kernel<<<1, 64, 0, wcn_stream(stream)>>>((long long)limit_cycles, dev_status, gave_up);
  return cudaGetLastError() == cudaSuccess ? WCN_OK : WCN_ERR_EXECUTION;
}

bool wcn_conv_tcgen05_supported(int K, int c_in, int c_out, int dtype, int out_dtype) {
  return (dtype == WCN_F16 || dtype == WCN_BF16) && (out_dtype == dtype || out_dtype == WCN_F32) && K >= 1 &&
         K <= MAX_OFFSETS && c_in >= 16 && c_in % 8 == 0 && c_out >= 16 && c_out <= 256 && c_out % 16 == 0;
}

int64_t wcn_conv_tcgen05_packed_bytes(int K, int c_in, int c_out) { return (int64_t)K * padded(c_in) * c_out * 2; }

int wcn_conv_tcgen05_pack(const void* weight, int src_dtype, int K, int c_in, int c_out, int dtype, int transposed, int reversed,
                          void* packed, cudaStream_t st) {
  const int64_t total = (int64_t)K * (padded(c_in) / 8) * c_out;
  if (total == 0) return WCN_OK;
  const unsigned grid = (unsigned)((total + 255) / 256);
#define WCN_PACK_CASE(SD, TS, DD, TD)                                                                                    \
  if (src_dtype == SD && dtype == DD) {                                                                                  \
    pack_weight_kernel<TS, TD><<<grid, 256, 0, st>>>((const TS*)weight, (TD*)packed, K, c_in, c_out, pick_bk(c_in),       \
                                                    transposed, reversed);                                               \
    return cudaGetLastError() == cudaSuccess ? WCN_OK : WCN_ERR_EXECUTION;                                               \
  }
  WCN_PACK_CASE(WCN_F32, float, WCN_F16, __half)
  WCN_PACK_CASE(WCN_F16, __half, WCN_F16, __half)
  WCN_PACK_CASE(WCN_BF16, __nv_bfloat16, WCN_F16, __half)
  WCN_PACK_CASE(WCN_F32, float, WCN_BF16, __nv_bfloat16)
  WCN_PACK_CASE(WCN_F16, __half, WCN_BF16, __nv_bfloat16)
  WCN_PACK_CASE(WCN_BF16, __nv_bfloat16, WCN_BF16, __nv_bfloat16)
#undef WCN_PACK_CASE
  return WCN_ERR_INVALID_PARAMETERS;
}

int wcn_conv_tcgen05_fwd(const void* feats, int64_t num_in, int64_t feats_ld, const void* packed, const int32_t* nbr,
                         const int32_t* out_rows, int64_t M, int K, int c_in, int c_out, int dtype,
                         const float* scale, const float* shift, const void* residual, int64_t residual_ld, int relu,
                         void* out, int64_t out_ld, int out_dtype, int split_k, int32_t* dev_status, cudaStream_t st) {
  if (!wcn_conv_tcgen05_supported(K, c_in, c_out, dtype, out_dtype)) return WCN_ERR_UNSUPPORTED_CONFIG;
  if (!dev_status || !packed || num_in <= 0 || num_in >= 0x7FFFFFFFll || M >= 0x7FFFFFFFll) return WCN_ERR_INVALID_PARAMETERS;
  const int64_t osz = out_dtype == WCN_F32 ? 4 : 2;
  if ((reinterpret_cast<uintptr_t>(feats) & 15) || (reinterpret_cast<uintptr_t>(packed) & 15) ||
      (reinterpret_cast<uintptr_t>(out) & 15) || (reinterpret_cast<uintptr_t>(residual) & 15) ||
      feats_ld < c_in || (feats_ld * 2) % 16 || out_ld < c_out || (out_ld * osz) % 16 ||
      (residual && (residual_ld < c_out || (residual_ld * osz) % 16)))
    return WCN_ERR_INVALID_PARAMETERS;
  ConvTcParams p = {};
  p.feats = (const char*)feats; p.wpacked = (const char*)packed; p.nbr = nbr; p.out_rows = out_rows;
  p.M = M; p.num_in = num_in; p.K = K; p.c_in = padded(c_in); p.row_bytes = c_in * 2; p.c_out = c_out;
  p.in_ld_bytes = feats_ld * 2; p.out_ld = out_ld; p.res_ld = residual_ld;
  p.scale = scale; p.shift = shift; p.residual = residual; p.relu = relu; p.out = out;
  p.dev_status = dev_status;
  p.wide_out = (reinterpret_cast<uintptr_t>(out) & 31) == 0 && (out_ld * osz) % 32 == 0;
  p.wide_res = residual && (reinterpret_cast<uintptr_t>(residual) & 31) == 0 && (residual_ld * osz) % 32 == 0;
  const int bk = pick_bk(c_in);
  const bool bf = dtype == WCN_BF16;
#define WCN_TC_CASE(BKV, BFV, TO) \
  if (bk == BKV && bf == BFV) return launch_tc<BKV, BFV, TO>(p, split_k, st);
  if (out_dtype == WCN_F32) {
    WCN_TC_CASE(64, false, float) WCN_TC_CASE(64, true, float) WCN_TC_CASE(32, false, float) WCN_TC_CASE(32, true, float)
  } else if (bf) {
    WCN_TC_CASE(64, true, __nv_bfloat16) WCN_TC_CASE(32, true, __nv_bfloat16)
  } else {
    WCN_TC_CASE(64, false, __half) WCN_TC_CASE(32, false, __half)
  }
#undef WCN_TC_CASE
  return WCN_ERR_UNSUPPORTED_CONFIG;
}
