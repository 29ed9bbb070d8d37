// Weight gradient of the sparse convolution on the 5th-generation tensor cores:
//
//     dW[k][ci][co] = sum over output rows m with a neighbour at offset k of
//                     X[nbr[k][m]][ci] * dY[m][co]
//
// i.e. per kernel offset a tall-skinny GEMM X_k^T (C_in x rows) times dY (rows x C_out) whose
// reduction runs over the rows.  Both operands are what the forward kernel already knows how
// to fetch: 128 gathered rows of X and 128 rows of dY, as swizzled shared-memory tiles whose
// rows are 128-byte (or 64-byte) channel slices.  Read as MN-major operands those tiles put the
// channels on the M / N side of tcgen05.mma and the rows on its K side, so a 128-row step is
// eight K = 16 instructions and nothing is transposed in memory.
//
// The M = 128 side of an instruction holds 128 / CW "units", a unit being the CW = 64 (or 32)
// channel slice of X gathered through ONE offset; consecutive units (offset-major) form a
// group: two offsets at C_in = 64, half an offset at C_in = 256.  A CTA owns every `ranges`-th
// 128-row step and as many groups as have room for their [128 x C_out] sums in tensor memory
// (512 / C_out of them): the dY tile of a step is fetched once for all of them, and a group
// none of whose offsets has a neighbour in the step costs nothing.  In the end the sums are
// added to the fp32 gradient with red.global.add.v4.f32 (the caller zeroes the gradient; the
// order of the adds is not fixed, as in any split reduction).
//
// What bounds it: the producers' instruction streams, then the gather of X (32 KB per step and group; the matrix
// instructions of one take 400 clocks at C_out = 64).  An earlier form had one group per CTA (dY read again for each, and a
// set-up and a tail for each), all eight producer warps on every tile and the neighbour indices loaded when they were
// needed.  240 000 rows of a room, 27 offsets, bf16: 96 -> 64 channels 412 -> 179 us, 64 -> 64 277 -> 110 us, 32 -> 32
// 69 us; 60 000 rows of 128 -> 128 81 us, of 256 -> 256 292 us.
//
// Roles: two teams of 4 producer warps (cp.async gathers that signal the stage's mbarrier when they
// land, and the adds at the end), 1 MMA thread.  Every wait is bounded and reports through the device
// status word.
#include "wcn_common.cuh"
#include "tcgen05_common.cuh"

namespace {

constexpr int WG_ROWS = 128;          // rows per step (K extent of 8 instructions)
constexpr int WG_MAX_STAGES = 6;
constexpr int WG_MAX_GROUPS = 16;     // 512 columns of tensor memory, 32 a group at least
constexpr int WG_PROD_THREADS = 256;  // warps 0..7, two teams of four
constexpr int WG_MMA_WARP = 8;
constexpr int WG_THREADS = 288;

struct WgradParams {
  const char* feats;     // [num_in, c_in]
  const char* gout;      // [M, c_out]
  const int32_t* nbr;    // [K][M]
  const int32_t* out_rows;     // slot -> row of gout (tiled table), or null for the identity
  const uint32_t* tile_masks;  // per 128-row step: offsets with any neighbour (null: every step is processed)
  float* gw;             // [K][c_in][c_out] fp32, accumulated into
  int64_t M, num_in;
  int K, c_in, c_out;
  int32_t* dev_status;
  int stages;            // ring depth of the X tiles (the dY ring has two)
  int groups;            // groups per CTA
  int cols;              // TMEM columns of a group (power of two >= c_out)
  int tmem;              // TMEM columns of the CTA
  bool vec;              // gw is 16-byte aligned
};

struct WgradControl {
  uint64_t full[WG_MAX_STAGES], empty[WG_MAX_STAGES];
  uint64_t dy_full[2], dy_empty[2];
  uint64_t acc_full;
  uint32_t gmask[WG_MAX_GROUPS];   // offsets that a group gathers through
  int unit_k[WG_MAX_GROUPS * 4];   // a unit's offset (-1: none) and the first byte of its channels
  int unit_at[WG_MAX_GROUPS * 4];
  uint32_t tmem_holder;
  int skip;
  uint32_t started;                // groups whose sums received at least one step
};

__device__ __forceinline__ void red_add4(float* p, const uint32_t* v) {
  asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(__uint_as_float(v[0])),
               "f"(__uint_as_float(v[1])), "f"(__uint_as_float(v[2])), "f"(__uint_as_float(v[3]))
               : "memory");
}

template <int RBA, int RBB, bool BF16>
__global__ void __launch_bounds__(WG_THREADS, 1)
conv_wgrad_tcgen05_kernel(const WgradParams p) {
  constexpr int CWA = RBA / 2;              // channels per unit
  constexpr int GU = 128 / CWA;             // units per group (the M = 128 side)
  constexpr int CHA = RBA / 16, CHB = RBB / 16;
  constexpr int A_TILE = WG_ROWS * RBA;     // one unit's tile
  constexpr int B_TILE = WG_ROWS * RBB;     // one dY channel chunk's tile
  constexpr int A_STAGE = GU * A_TILE;
  extern __shared__ uint8_t smem_raw[];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int UA = (p.c_in + CWA - 1) / CWA;               // units per offset
  const int NB = (p.c_out + RBB / 2 - 1) / (RBB / 2);    // dY channel chunks (N = c_out: what lies beyond is not read)
  const int total_units = p.K * UA;
  const int group0 = blockIdx.y * p.groups;
  const int ng = min(p.groups, (total_units + GU - 1) / GU - group0);
  const int B_STAGE = NB * B_TILE;

  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t b_base = base + p.stages * A_STAGE;
  WgradControl* ctl = reinterpret_cast<WgradControl*>(gen + (size_t)p.stages * A_STAGE + 2 * (size_t)B_STAGE);
  auto bar = [](uint64_t* b) { return smem_u32(b); };

  if (warp == 0) {
    if (lane < p.stages) { mbar_init(bar(&ctl->full[lane]), WG_PROD_THREADS / 2); mbar_init(bar(&ctl->empty[lane]), 1); }
    if (lane < 2) { mbar_init(bar(&ctl->dy_full[lane]), WG_PROD_THREADS / 2); mbar_init(bar(&ctl->dy_empty[lane]), 1); }
    if (lane == 2) mbar_init(bar(&ctl->acc_full), 2);  // the commit of the last MMAs and the issuer's own arrival
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  } else if (warp == 1) {
    if (lane == 0) ctl->skip = *(volatile int32_t*)p.dev_status;  // an earlier launch on this status word failed
  } else if (warp == 2) {
    uint32_t m = 0;
    if (lane < ng && !p.tile_masks) m = 1;  // (any number of offsets)
    if (lane < ng && p.tile_masks)
      for (int u = 0; u < GU; ++u) {
        const int unit = (group0 + lane) * GU + u;
        if (unit < total_units) m |= 1u << (unit / UA);
      }
    if (lane < WG_MAX_GROUPS) ctl->gmask[lane] = m;
  } else if (warp == 3) {
    for (int i = lane; i < ng * GU; i += 32) {
      const int unit = group0 * GU + i;
      ctl->unit_k[i] = unit < total_units ? unit / UA : -1;
      ctl->unit_at[i] = (unit % UA) * RBA;
    }
  } else if (warp == WG_MMA_WARP) {
    tmem_alloc(smem_u32(&ctl->tmem_holder), (uint32_t)p.tmem);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = ctl->tmem_holder;
  const bool run = ctl->skip != (int)WCN_ERR_WAIT_EXPIRED;

  const int64_t total_steps = (p.M + WG_ROWS - 1) / WG_ROWS, stride = gridDim.x;
  auto mask_of = [&](int64_t st) { return st >= total_steps ? 0u : p.tile_masks ? __ldg(&p.tile_masks[st]) : 0xFFFFFFFFu; };
  bool ok = run;

  if (warp < WG_MMA_WARP) {
    // ================================================================ producers
    // Two teams of four warps (32 rows of a tile each) take the items - (step, group) pairs with a neighbour - in turns, and
    // the dY tiles of the steps in turns: what an item costs is the length of a warp's instruction stream (with eight warps
    // on every item 1 900 to 2 800 clocks, with or without the copies and the matrix instructions).  The loads of an item
    // wait their turn behind the copies already issued, so they are made an item of this team early.
    constexpr int RPI = 32 / CHA;                 // tile rows per warp-wide copy instruction
    constexpr int NJ = 32 / RPI;                  // instructions per warp per unit
    const int team = warp >> 2, row0 = (warp & 3) * 32;
    const int sub_row = lane / CHA, chunk = lane % CHA;
    uint32_t aoff[NJ];
#pragma unroll
    for (int j = 0; j < NJ; ++j) aoff[j] = tile_offset<RBA>(row0 + j * RPI + sub_row, chunk);
    const int PR = p.c_out * 2 / 16;              // 16-byte pieces of a dY row
    const uint32_t mine = ctl->gmask[lane & (WG_MAX_GROUPS - 1)] & (lane < ng ? 0xFFFFFFFFu : 0u);
    const int num_in = (int)p.num_in;
    const int64_t ld = (int64_t)p.c_in * 2;
    bool bad = false;
    int64_t st = blockIdx.x;
    uint32_t rest = __ballot_sync(0xFFFFFFFFu, (mask_of(st) & mine) != 0);
    uint32_t ahead = mask_of(st + stride);
    bool fresh = true;             // no item of step `st` has been taken
    int item = 0, step = 0;        // items and steps taken
    struct Item { int group; int32_t out; bool dy; int idx[GU]; };   // dy: this team fetches the step's dY tile before it
    auto next = [&](Item& it) {
      it.dy = false;
      for (;;) {
        while (!rest && st < total_steps) {
          st += stride;
          rest = __ballot_sync(0xFFFFFFFFu, (ahead & mine) != 0);
          ahead = mask_of(st + stride);
          fresh = true;
        }
        it.group = __ffs(rest) - 1;   // -1: no more
        if (!rest) return;
        const int64_t m = st * WG_ROWS + row0 + lane;
        const bool own = (item & 1) == team;
        if (fresh) {
          fresh = false;
          if ((step++ & 1) == team) {
            it.out = m < p.M ? (p.out_rows ? __ldg(&p.out_rows[m]) : (int32_t)m) : -1;
            it.dy = true;
            if (!own) { it.group = WG_MAX_GROUPS; return; }   // the tile alone: the item is the other team's
          }
        }
        rest &= rest - 1;
        ++item;
        if (!own) continue;
#pragma unroll
        for (int u = 0; u < GU; ++u) {
          const int k = ctl->unit_k[it.group * GU + u];
          it.idx[u] = (k >= 0 && m < p.M) ? __ldg(&p.nbr[(int64_t)k * p.M + m]) : -1;
        }
        return;
      }
    };
    Item q;
    next(q);
    int slot = team, phase = 0, dslot = team, dphase = 0;   // (a team uses every other slot of either ring)
    while (ok && q.group >= 0) {
      const Item cur = q;
      next(q);
      if (cur.dy) {
        if (!mbar_wait(bar(&ctl->dy_empty[dslot]), dphase ^ 1, p.dev_status)) { ok = false; break; }
        const uint32_t dst = b_base + dslot * B_STAGE;
        for (int i = lane; i < 32 * PR; i += 32) {
          const int r = i / PR, piece = i - r * PR;
          const int32_t row = __shfl_sync(0xFFFFFFFFu, cur.out, r);
          cp_async16(dst + (piece / CHB) * B_TILE + tile_offset<RBB>(row0 + r, piece % CHB),
                     row >= 0 ? p.gout + ((int64_t)row * p.c_out) * 2 + piece * 16 : p.gout, row >= 0 ? 16u : 0u);
        }
        cp_async_arrive(bar(&ctl->dy_full[dslot]));  // hardware arrives when this thread's copies land
        dphase ^= 1;
        if (cur.group == WG_MAX_GROUPS) continue;
      }
      if (!mbar_wait(bar(&ctl->empty[slot]), phase ^ 1, p.dev_status)) { ok = false; break; }
      const uint32_t dst = base + slot * A_STAGE;
#pragma unroll
      for (int u = 0; u < GU; ++u) {
        const char* from = p.feats + ctl->unit_at[cur.group * GU + u] + chunk * 16;
        const bool over = cur.idx[u] >= num_in;   // names no feature row: counts as absent
        bad |= over;
        const int mine_row = over ? -1 : cur.idx[u];
        const bool valid = ctl->unit_at[cur.group * GU + u] + chunk * 16 < p.c_in * 2;   // (the last slice may be narrower)
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
          const int r = __shfl_sync(0xFFFFFFFFu, mine_row, j * RPI + sub_row);
          const bool have = r >= 0 && valid;
          cp_async16(dst + u * A_TILE + aoff[j], have ? from + r * ld : p.feats, have ? 16u : 0u);
        }
      }
      cp_async_arrive(bar(&ctl->full[slot]));
      slot += 2;
      if (slot >= p.stages) { slot = team; phase ^= 1; }
    }
    cp_async_drain();
    if (bad) wcn_report_bounds(p.dev_status);
    // ================================================================ the sums are added to the gradient
    __syncwarp();
    ok = __all_sync(0xFFFFFFFFu, ok);
    if (ok) ok = mbar_wait(bar(&ctl->acc_full), 0, p.dev_status);
    if (__all_sync(0xFFFFFFFFu, ok)) {
      tc_fence_after();
      const int row = (warp & 3) * 32 + lane;        // TMEM lane = position on the M side
      for (int g = warp >> 2; g < ng; g += 2) {
        if (!((ctl->started >> g) & 1u)) continue;
        const int unit = (group0 + g) * GU + row / CWA;
        const bool live = unit < total_units && (unit % UA) * CWA + row % CWA < p.c_in;
        float* dst = p.gw + ((int64_t)(unit / UA) * p.c_in + (unit % UA) * CWA + row % CWA) * p.c_out;
        const uint32_t trow = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(g * p.cols);
        for (int c0 = 0; c0 < p.c_out; c0 += 16) {
          uint32_t r[16];
          tmem_ld16(trow + (uint32_t)c0, r);  // executed by all lanes of the warp
          tmem_ld_wait();
          if (live && p.vec) {
#pragma unroll
            for (int i = 0; i < 16; i += 4) red_add4(dst + c0 + i, r + i);
          } else if (live) {
#pragma unroll
            for (int i = 0; i < 16; ++i) atomicAdd(dst + c0 + i, __uint_as_float(r[i]));
          }
        }
      }
    }
  } else {
    // ================================================================ MMA issuer
    if (elect_one()) {
      // fp32 accumulate, A and B MN-major (bits 15, 16), N = c_out, M = 128
      const uint32_t idesc = (1u << 4) | ((BF16 ? 1u : 0u) << 7) | ((BF16 ? 1u : 0u) << 10) | (1u << 15) | (1u << 16) |
                             ((uint32_t)(p.c_out >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
      int slot = 0, phase = 0, dslot = 0, dphase = 0;
      uint32_t started = 0, mask = mask_of(blockIdx.x);
      for (int64_t st = blockIdx.x; st < total_steps && ok; st += stride) {
        uint32_t rest = 0;
        for (int g = 0; g < ng; ++g) rest |= (mask & ctl->gmask[g]) ? 1u << g : 0u;
        mask = mask_of(st + stride);
        if (!rest) continue;
        if (!mbar_wait(bar(&ctl->dy_full[dslot]), dphase, p.dev_status)) { ok = false; break; }
        const uint32_t b_slot = b_base + dslot * B_STAGE;
        for (; rest; rest &= rest - 1) {
          const int g = __ffs(rest) - 1;
          if (!mbar_wait(bar(&ctl->full[slot]), phase, p.dev_status)) { ok = false; break; }
          tc_fence_after();
          const uint64_t adesc = smem_desc_mn<RBA>(base + slot * A_STAGE, (uint32_t)A_TILE);
          const uint64_t bdesc = smem_desc_mn<RBB>(b_slot, (uint32_t)B_TILE);
          const uint32_t d = tmem_base + (uint32_t)(g * p.cols), acc = (started >> g) & 1u;
#pragma unroll
          for (int ks = 0; ks < WG_ROWS / 16; ++ks)  // 16 rows = two 8-row atoms further down the tiles
            umma_f16(d, adesc + (uint64_t)(ks * RBA), bdesc + (uint64_t)(ks * RBB), idesc, acc | (ks > 0 ? 1u : 0u));
          started |= 1u << g;
          umma_commit(bar(&ctl->empty[slot]));  // the stage is free once these instructions have read it
          if (++slot == p.stages) { slot = 0; phase ^= 1; }
        }
        if (!ok) break;
        umma_commit(bar(&ctl->dy_empty[dslot]));
        dslot ^= 1;
        if (dslot == 0) dphase ^= 1;
      }
      umma_commit(bar(&ctl->acc_full));  // arrives when every MMA above has completed (at once if there were none)
      ctl->started = ok ? started : 0u;
      mbar_arrive(bar(&ctl->acc_full));  // publishes `started`
    }
    __syncwarp();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == WG_MMA_WARP) tmem_dealloc(tmem_base, (uint32_t)p.tmem);
}

template <int RBA, int RBB, bool BF16>
int launch_wgrad(WgradParams& p, cudaStream_t st) {
  constexpr int CWA = RBA / 2, GU = 128 / CWA;
  const int UA = (p.c_in + CWA - 1) / CWA, NB = (p.c_out + RBB / 2 - 1) / (RBB / 2);
  const int groups = (p.K * UA + GU - 1) / GU;
  const size_t a_stage = (size_t)GU * WG_ROWS * RBA, b_stage = (size_t)NB * WG_ROWS * RBB;
  const size_t limit = 226 * 1024, fixed = 1024 + sizeof(WgradControl) + 128;
  int stages = (int)((limit - fixed - 2 * b_stage) / a_stage);
  if (stages > WG_MAX_STAGES) stages = WG_MAX_STAGES;
  stages &= ~1;   // the two teams take turns
  if (stages < 2) return WCN_ERR_UNSUPPORTED_CONFIG;
  p.stages = stages;
  p.cols = 32;
  while (p.cols < p.c_out) p.cols <<= 1;
  // One CTA per multiprocessor.  As many groups per CTA as tensor memory holds (they share dY) while every CTA still gets
  // two steps; then as many CTAs along the rows as fit.
  const int sms = wcn_num_sms();
  const int64_t total_steps = (p.M + WG_ROWS - 1) / WG_ROWS;
  int per = 512 / p.cols;
  if (per > groups) per = groups;
  while (per > 1 && total_steps * ((groups + per - 1) / per) < 2 * (int64_t)sms) per = (per + 1) / 2;
  const int blocks = (groups + per - 1) / per;
  p.groups = (groups + blocks - 1) / blocks;   // evenly
  p.tmem = 32;
  while (p.tmem < p.groups * p.cols) p.tmem <<= 1;
  int64_t ranges = sms / blocks;
  if (ranges > (total_steps + 1) / 2) ranges = (total_steps + 1) / 2;
  if (ranges < 1) ranges = 1;

  auto kern = conv_wgrad_tcgen05_kernel<RBA, RBB, BF16>;
  static bool configured[64] = {};  // per template instance and device: opt in to large shared memory once
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return WCN_ERR_INITIALIZATION;
  if (!configured[dev]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024) != cudaSuccess) {
      (void)cudaGetLastError();
      return WCN_ERR_INITIALIZATION;
    }
    configured[dev] = true;
  }
  dim3 grid((unsigned)ranges, (unsigned)blocks);
  kern<<<grid, WG_THREADS, fixed + stages * a_stage + 2 * b_stage, st>>>(p);
  return cudaGetLastError() == cudaSuccess ? WCN_OK : WCN_ERR_EXECUTION;
}

}  // namespace

bool wcn_conv_wgrad_tcgen05_supported(int K, int c_in, int c_out, int dtype) {
  return (dtype == WCN_F16 || dtype == WCN_BF16) && K >= 1 && c_in >= 16 && c_in % 8 == 0 && c_out >= 16 &&
         c_out % 16 == 0 && c_out <= 256 && (int64_t)K * c_in <= 65535ll * 32;
}

int wcn_conv_wgrad_tcgen05(const void* feats, int64_t num_in, const void* grad_out, const int32_t* nbr,
                           const int32_t* out_rows, const uint32_t* tile_masks, int64_t M, int K, int c_in, int c_out, int dtype,
                           float* grad_weight, int32_t* dev_status, cudaStream_t st) {
  if (!wcn_conv_wgrad_tcgen05_supported(K, c_in, c_out, dtype)) return WCN_ERR_UNSUPPORTED_CONFIG;
  if (!dev_status || !grad_weight || num_in <= 0 || num_in >= 0x7FFFFFFFll) return WCN_ERR_INVALID_PARAMETERS;
  if ((reinterpret_cast<uintptr_t>(feats) & 15) || (reinterpret_cast<uintptr_t>(grad_out) & 15))
    return WCN_ERR_INVALID_PARAMETERS;
  WgradParams p;
  p.feats = (const char*)feats; p.gout = (const char*)grad_out; p.nbr = nbr; p.out_rows = out_rows; p.tile_masks = K <= 32 ? tile_masks : nullptr; p.gw = grad_weight;
  p.M = M; p.num_in = num_in; p.K = K; p.c_in = c_in; p.c_out = c_out; p.dev_status = dev_status;
  p.vec = (reinterpret_cast<uintptr_t>(grad_weight) & 15) == 0;
  const bool a128 = c_in % 64 == 0, b128 = c_out % 64 == 0, bf = dtype == WCN_BF16;
#define WCN_WG_CASE(A, B, F) if (a128 == (A == 128) && b128 == (B == 128) && bf == F) return launch_wgrad<A, B, F>(p, st);
  WCN_WG_CASE(128, 128, false) WCN_WG_CASE(128, 64, false) WCN_WG_CASE(64, 128, false) WCN_WG_CASE(64, 64, false)
  WCN_WG_CASE(128, 128, true) WCN_WG_CASE(128, 64, true) WCN_WG_CASE(64, 128, true) WCN_WG_CASE(64, 64, true)
#undef WCN_WG_CASE
  return WCN_ERR_UNSUPPORTED_CONFIG;
}
