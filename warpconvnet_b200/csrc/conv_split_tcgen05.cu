// Sparse convolution of fp32 tensors on the 5th-generation tensor cores, without giving up fp32.
//
// An fp32 number is the exact sum of three bf16 numbers (24 bits of significand, eight in each): x = h + m + l, w likewise.
// Of the nine products six are kept, h h, h m, m h, m m, h l, l h (what is left out, m l, l m and l l, is below 2^-24 of a product), each exact
// in fp32.  What the tensor core does not do as fp32 arithmetic does is add: its accumulator drops the bits below its last
// place instead of rounding them, and over the some 640 additions of a 64-channel layer that bias alone was nine times the
// error of the FMA kernel (4.1e-6 against 4.5e-7 of the result's 2-norm, 60 000 room voxels).  So an accumulator is only
// used for 32 channels of one offset, the small products first, and then added to the row's sums in registers, rounding to
// nearest: 9.7e-8 (C = 128: 1.3e-7 against 6.4e-7; 20 000 random cells, C = 32: 6.8e-8 against 1.3e-7).
//
// Two launches.  The first writes the three bf16 planes of every feature row and of the weights (as swizzled shared-memory
// images) to the caller's workspace.  A number that is infinite, NaN or above 2^39 (a product of two parts could then be
// infinite where the numbers' is not) becomes NaN there, and an output row whose sums are not finite is multiplied again on
// the FMA pipes from the numbers as they came: other rows do not notice (60 000 rows of 64 channels: 71 us, with one NaN 142,
// with one in every hundredth row 378, in every row 910; conv_fp32.cu 205.  As a second form of the whole launch, taken for
// any such number anywhere: 1 840).  The second is the convolution.  A CTA works through units of 128 output rows x BN columns, claimed
// one ahead from the hardware's queue, dense rows first:
//  * four gather warps read the unit's neighbour table (32 rows each), agree on the offsets present, and copy for every
//    (offset, 32 channels) the three planes of the listed rows into a slot of a ring (cp.async, absent rows zero-filled);
//  * one thread adds the weight planes to the slot (bulk copies), two issue the 12 tcgen05.mma of a slot in turns, each slot
//    into one of four accumulators in tensor memory;
//  * eight epilogue warps add every accumulator to the sums in their registers (two threads per row) and, after the last,
//    apply scale / shift, residual and ReLU and store the row.  No atomics, the same bits on every run.
// Few row tiles divide the offsets of a tile among the CTAs of a cluster, which add their sums through distributed shared memory.
//
// Bound by the rate at which narrow instructions are issued: 12 of M = 128, K = 16 per 128 rows, offset and 32 channels, each of
// which takes as long as A takes to be read from shared memory (57 clocks at N = 64, 61 at 96, 67 at 128; the tensor pipe itself
// is busy for 29 to 34 % of the time), and by the last tiles of a launch.  Measured (us, the
// FMA kernel of conv_fp32.cu / both launches here, L2 flushed): room voxels, 60 000: 64 -> 64 207 / 69, 128 -> 128 672 / 134,
// 100 000: 64 -> 64 320 / 105, 2 000: 64 -> 64 40 / 20; 20 000 random cells, 32 -> 32 41 / 28.  One issuing thread instead of two:
// 60 000 rows of 64 channels 75; eight gather warps of 16 rows cost the epilogue its registers; without clusters 2 000 rows of
// 64 channels 40, of 128 69 instead of 30.
#include "wcn_common.cuh"
#include "tcgen05_common.cuh"
#include "split_bf16.cuh"
#include "tile_order.cuh"
#include <atomic>

namespace {

constexpr int SP_M = 128;
constexpr int SP_BK = 32, SP_RB = SP_BK * 2;          // channels and bytes of a tile row
constexpr int SP_PLANE = SP_M * SP_RB;                // bytes of one plane of a row tile
constexpr int SP_MAX_N = 128;                         // columns of a unit (two threads per row hold its sums)
constexpr int SP_MAX_K = 27;
constexpr int SP_ACCS = 4;                            // accumulators
constexpr int SP_MAX_SLOTS = 8;
constexpr int SP_MAX_SLICES = 8;                      // CTAs of a (portable) cluster
constexpr int SP_EPI = 256, SP_GATHER = 128;          // warps 0..7 and 8..11
constexpr int SP_MMA_WARP = 12, SP_ISSUERS = 2, SP_WEIGHT_WARP = 14, SP_THREADS = 480;
constexpr size_t SP_SMEM = 226 * 1024;
constexpr int SP_PLANE_BLOCKS = 1024;                 // of the first launch at most

struct SplitParams {
  const char* planes;      // [num_in][3][cp] bf16
  const char* wplanes;     // [K][cp / 32][3] images of [c_out][32] bf16
  const float* feats;
  const float* weight;     // (the two as they came, for rows with numbers that cannot be split)
  const int32_t* nbr;
  const int32_t* out_rows;
  int64_t M, in_ld, out_ld, res_ld;
  int K, c_in, cp, c_out, num_in;
  int block_n, blocks;     // columns of a unit (of the last column block: what is left), column blocks
  int tiles, window, tail; // row tiles; see tile_of
  int S;                   // CTAs of a cluster that divide the offsets of a unit: slice s has those with k % S == s
  int slots;
  const float* scale;
  const float* shift;
  const float* residual;
  int relu;
  float* out;
  int32_t* dev_status;
};

struct SplitControl {
  uint64_t full[SP_MAX_SLOTS], empty[SP_MAX_SLOTS];
  uint64_t acc_full[SP_ACCS], acc_empty[SP_ACCS];
  uint64_t info_full[2], info_empty[2];
  uint64_t meet, claim_full;
  __align__(16) uint64_t claim[2];
  int32_t info_unit[2];        // < 0: no more units
  uint32_t info_mask[2];       // offsets that any row of the unit has
  uint32_t mask_acc[3];
  uint32_t tmem;
  int32_t out_row[2][SP_M];    // -1 past the end
  int32_t lists[4][SP_MAX_K][32];   // input rows of a gather warp's 32 rows at every offset
};

// Row tile that comes `turn`-th: dense rows first, as conv_tcgen05.cu orders its supertiles.
__device__ __forceinline__ int tile_of(const SplitParams& p, int turn) {
  if (p.window == 0) return turn;
  const int head = p.tiles - p.tail * p.window;
  if (turn < head) return p.tiles - 1 - turn;
  const int j = turn - head, place = j / p.tail, w = j - place * p.tail;
  return w * p.window + (p.window - 1 - place);
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

__device__ __forceinline__ float finish(const SplitParams& p, float y, int64_t m, int n) {
  y = wcn_affine(y, p.scale, p.shift, n);
  if (p.residual) y = __fadd_rn(y, __ldg(p.residual + m * p.res_ld + n));
  return p.relu ? fmaxf(y, 0.f) : y;
}

// Whether any of `cols` sums is infinite or NaN (0 times it is no zero).  0.4 us a unit of a narrow layer: 32 -> 48, 95 702 outdoor voxels
// 57.2 us without, 60.4 with it.  A branch for sixteen columns, or two numbers an instruction, take as long.
__device__ __forceinline__ bool not_finite(const float (&sum)[64], int cols) {
  float t[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int c = 0; c < 64; ++c)
    if (c < cols) t[c & 3] = fmaf(sum[c], 0.f, t[c & 3]);
  return !((t[0] + t[1]) + (t[2] + t[3]) == 0.f);
}

// Four columns of a table row on the FMA pipes, offsets and channels in order: what a number without three parts (its first
// part is NaN) or a sum past the end of fp32 asks for.
__device__ __forceinline__ void fma_four(const SplitParams& p, int64_t slot, int n, float (&y)[4]) {
  y[0] = y[1] = y[2] = y[3] = 0.f;
  int next = __ldg(&p.nbr[slot]);
  for (int k = 0; k < p.K; ++k) {
    const int r = next;
    if (k + 1 < p.K) next = __ldg(&p.nbr[(int64_t)(k + 1) * p.M + slot]);
    if (r < 0 || r >= p.num_in) continue;   // (reported by the gather warps)
    const float* x = p.feats + (int64_t)r * p.in_ld;
    const float* w = p.weight + (int64_t)k * p.c_in * p.c_out + n;
#pragma unroll 4   // (loads in flight are what this takes its time for)
    for (int c = 0; c < p.c_in; c += 4) {
      const float4 a = __ldg(reinterpret_cast<const float4*>(x + c));
      const float v[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float4 b = __ldg(reinterpret_cast<const float4*>(w + (int64_t)(c + u) * p.c_out));
        y[0] = fmaf(v[u], b.x, y[0]);
        y[1] = fmaf(v[u], b.y, y[1]);
        y[2] = fmaf(v[u], b.z, y[2]);
        y[3] = fmaf(v[u], b.w, y[3]);
      }
    }
  }
}

// ------------------------------------------------------------------ planes

// Bound by memory (4 bytes in, 6 out per channel): a thread makes eight channels of a row, or of a column of the weights.
__global__ void __launch_bounds__(256)
split_planes_kernel(const float* __restrict__ feats, int64_t num_in, int64_t in_ld, const float* __restrict__ weight, int K, int c_in,
                    int cp, int c_out, char* __restrict__ planes, char* __restrict__ wplanes) {
  launch_dependents();
  const int per_row = cp / 8;
  const int64_t rows = num_in * per_row, total = rows + (int64_t)K * per_row * c_out;
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < total; i += (int64_t)gridDim.x * 256) {
    float v[8];
    char* dst;
    int64_t apart;
    if (i < rows) {
      const int64_t r = i / per_row;
      const int c = (int)(i - r * per_row) * 8;
      load_eight(feats + r * in_ld, c, c_in, v);
      apart = (int64_t)cp * 2;
      dst = planes + r * 3 * apart + c * 2;
    } else {
      int64_t q = i - rows;
      const int n = (int)(q % c_out);
      q /= c_out;
      const int c = (int)(q % per_row) * 8, k = (int)(q / per_row);
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = c + u < c_in ? __ldg(&weight[((int64_t)k * c_in + c + u) * c_out + n]) : 0.f;
      apart = (int64_t)c_out * SP_RB;
      dst = wplanes + ((int64_t)k * (cp / SP_BK) + c / SP_BK) * 3 * apart + tile_offset<SP_RB>(n, (c % SP_BK) / 8);
    }
    store_parts(v, dst, apart);
  }
}

// ------------------------------------------------------------------ convolution

__global__ void __launch_bounds__(SP_THREADS, 1)
conv_split_kernel(const SplitParams p) {
  extern __shared__ uint8_t smem_raw[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int BN = p.block_n, KB = p.cp / SP_BK;
  const int b_bytes = BN * SP_RB, slot_bytes = 3 * (SP_PLANE + b_bytes);
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  SplitControl* ctl = reinterpret_cast<SplitControl*>(smem_raw + (base - smem_u32(smem_raw)) + p.slots * slot_bytes);
  auto bar = [](uint64_t* b) { return smem_u32(b); };
  const int units = p.tiles * p.blocks;
  auto columns_of = [&](int unit) { return min(BN, p.c_out - unit % p.blocks * BN); };
  const int first = p.S > 1 ? (int)blockIdx.x / p.S : (int)blockIdx.x, rank = p.S > 1 ? (int)blockIdx.x % p.S : 0;

  if (warp == 0) {
    if (lane < p.slots) { mbar_init(bar(&ctl->full[lane]), SP_GATHER + 1); mbar_init(bar(&ctl->empty[lane]), 1); }
    if (lane < SP_ACCS) { mbar_init(bar(&ctl->acc_full[lane]), 1); mbar_init(bar(&ctl->acc_empty[lane]), SP_EPI / 32); }
    if (lane < 2) { mbar_init(bar(&ctl->info_full[lane]), SP_GATHER); mbar_init(bar(&ctl->info_empty[lane]), SP_EPI / 32 + SP_ISSUERS + 1); }
    if (lane == 2) mbar_init(bar(&ctl->meet), SP_GATHER);
    if (lane == 3) mbar_init(bar(&ctl->claim_full), 1);
    if (lane < 3) ctl->mask_acc[lane] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == SP_MMA_WARP) tmem_alloc(smem_u32(&ctl->tmem), 512);
  // (everything above runs while the planes are written; tables, weights and rows are older than that launch)
  wait_for_primary();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = ctl->tmem;
  bool ok = true;

  if (warp >= 8 && warp < SP_MMA_WARP) {
    // ================================================================ gather
    const int g = warp - 8, gtid = tid - SP_EPI;
    const int sub = lane >> 2, chunk = lane & 3;      // a copy instruction covers eight rows of 64 bytes
    const uint32_t at0 = tile_offset<SP_RB>(g * 32 + sub, chunk);
    const char* from = p.planes + chunk * 16;
    const int64_t row_bytes = (int64_t)p.cp * 6;
    int unit = first, slot = 0, phase = 0, acc = 0, meet_phase = 0, claim_phase = 0;
    uint32_t slice = 0;   // this CTA's offsets
    for (int k = rank; k < p.K; k += p.S) slice |= 1u << k;
    bool bad = false;
    for (int n = 0; ok; ++n) {
      const int ib = n & 1;
      const int64_t m = (int64_t)tile_of(p, unit / p.blocks) * SP_M + g * 32 + lane;
      int r[SP_MAX_K];
#pragma unroll
      for (int k = 0; k < SP_MAX_K; ++k) r[k] = ((slice >> k) & 1u) && m < p.M ? __ldg(&p.nbr[(int64_t)k * p.M + m]) : -1;
      const int32_t out_row = m < p.M ? (p.out_rows ? __ldg(&p.out_rows[m]) : (int32_t)m) : -1;
      if (!mbar_wait(bar(&ctl->info_empty[ib]), ((n >> 1) & 1) ^ 1, p.dev_status)) { ok = false; break; }
      __syncwarp();   // (the lists of the unit before have been read)
      uint32_t has = 0;
#pragma unroll
      for (int k = 0; k < SP_MAX_K; ++k) {
        if (r[k] >= p.num_in) { r[k] = -1; bad = true; }
        has |= r[k] >= 0 ? 1u << k : 0u;
        ctl->lists[g][k][lane] = r[k];
      }
      has = __reduce_or_sync(0xFFFFFFFFu, has);
      ctl->out_row[ib][g * 32 + lane] = out_row;
      if (lane == 0 && has) atomicOr(&ctl->mask_acc[acc], has);
      mbar_arrive(bar(&ctl->meet));
      if (!mbar_wait(bar(&ctl->meet), meet_phase, p.dev_status)) { ok = false; break; }
      meet_phase ^= 1;
      const uint32_t mask = ctl->mask_acc[acc];
      // (scratch in turns of three: what is cleared here was read before this rendezvous and is next added to after the next)
      acc = acc == 2 ? 0 : acc + 1;
      if (gtid == 0) {
        ctl->mask_acc[acc == 2 ? 0 : acc + 1] = 0;
        ctl->info_unit[ib] = unit;
        ctl->info_mask[ib] = mask;
      }
      __syncwarp();
      mbar_arrive(bar(&ctl->info_full[ib]));
      for (uint32_t rest = mask; rest && ok; rest &= rest - 1) {
        const int k = __ffs(rest) - 1;
        const char* src[4];
        uint32_t bytes[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int q = ctl->lists[g][k][8 * j + sub];
          src[j] = from + (int64_t)max(q, 0) * row_bytes;
          bytes[j] = q >= 0 ? 16u : 0u;
        }
        for (int kb = 0; kb < KB; ++kb) {
          if (!mbar_wait(bar(&ctl->empty[slot]), phase ^ 1, p.dev_status)) { ok = false; break; }
          const uint32_t dst = base + slot * slot_bytes + at0;
#pragma unroll
          for (int s = 0; s < 3; ++s)
#pragma unroll
            for (int j = 0; j < 4; ++j) cp_async16(dst + s * SP_PLANE + j * (8 * SP_RB), src[j] + s * p.cp * 2 + kb * SP_RB, bytes[j]);
          cp_async_arrive(bar(&ctl->full[slot]));
          if (++slot == p.slots) { slot = 0; phase ^= 1; }
        }
      }
      // The next unit is claimed when this one's copies have been issued: a multiprocessor with a long unit leaves those that are
      // left to others (asked for before the copies, by whoever started first: 20 000 / 25 000 / 60 000 room voxels, 128 -> 128, 128,
      // 96 channels 93 / 98 / 116 us, now 69 / 72 / 111; 20 000 cells, 32 -> 32 25.0 / 22.8).
      if (p.S == 1 && gtid == 0) {
        // (every gather thread has read the last claim: they met since)
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_expect_tx(bar(&ctl->claim_full), 16u);
        asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(
                         smem_u32(&ctl->claim[0])), "r"(bar(&ctl->claim_full))
                     : "memory");
      }
      // (on failure the claim still has to arrive: it writes shared memory)
      uint32_t got = 0, x = 0;
      if (p.S == 1) {
        if (!mbar_wait(bar(&ctl->claim_full), claim_phase, p.dev_status)) {
          (void)mbar_wait(bar(&ctl->claim_full), claim_phase, p.dev_status);
          ok = false;
          break;
        }
        claim_phase ^= 1;
        asm volatile(
            "{\n\t.reg .b128 h;\n\t.reg .pred p;\n\tmov.b128 h, {%2, %3};\n\t"
            "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\n\tselp.u32 %0, 1, 0, p;\n\tmov.u32 %1, 0;\n\t"
            "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %1, h;\n\t}"
            : "=r"(got), "=r"(x)
            : "l"(*(volatile const uint64_t*)&ctl->claim[0]), "l"(*(volatile const uint64_t*)&ctl->claim[1])
            : "memory");
        __syncwarp();
      }
      if (!got || (int)x >= units) {
        const int nb = (n + 1) & 1;
        if (!mbar_wait(bar(&ctl->info_empty[nb]), (((n + 1) >> 1) & 1) ^ 1, p.dev_status)) { ok = false; break; }
        if (gtid == 0) ctl->info_unit[nb] = -1;
        __syncwarp();
        mbar_arrive(bar(&ctl->info_full[nb]));
        break;
      }
      unit = (int)x;
    }
    cp_async_drain();
    if (bad) wcn_report_bounds(p.dev_status);
  } else if (warp == SP_WEIGHT_WARP) {
    // ================================================================ weights
    if (elect_one()) {
      int slot = 0, phase = 0;
      for (int n = 0; ok; ++n) {
        const int ib = n & 1;
        if (!mbar_wait(bar(&ctl->info_full[ib]), (n >> 1) & 1, p.dev_status)) { ok = false; break; }
        const int unit = ctl->info_unit[ib];
        uint32_t rest = ctl->info_mask[ib];
        mbar_arrive(bar(&ctl->info_empty[ib]));
        if (unit < 0) break;
        const int n0 = (unit % p.blocks) * BN;
        const uint32_t bytes = (uint32_t)(columns_of(unit) * SP_RB);
        for (; rest && ok; rest &= rest - 1) {
          const char* src = p.wplanes + ((int64_t)(__ffs(rest) - 1) * KB * 3 * p.c_out + n0) * SP_RB;
          for (int kb = 0; kb < KB; ++kb) {
            if (!mbar_wait(bar(&ctl->empty[slot]), phase ^ 1, p.dev_status)) { ok = false; break; }
            const uint32_t dst = base + slot * slot_bytes + 3 * SP_PLANE, full = bar(&ctl->full[slot]);
            mbar_expect_tx(full, 3 * bytes);
#pragma unroll
            for (int s = 0; s < 3; ++s)
              bulk_copy_g2s(dst + s * b_bytes, src + (int64_t)(kb * 3 + s) * p.c_out * SP_RB, bytes, full);
            if (++slot == p.slots) { slot = 0; phase ^= 1; }
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == SP_MMA_WARP || warp == SP_MMA_WARP + 1) {
    // ================================================================ tensor-core instructions
    // Two threads take the slots in turns: what one of them waits and signals between its instructions (some 250 clocks a
    // slot, of 690) the other's fill.
    if (elect_one()) {
      const uint32_t idesc0 = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(SP_M >> 4) << 24);
      const int mine = warp - SP_MMA_WARP;
      int slot = 0, phase = 0, ab = 0, aphase = 0, turn = 0;
      for (int n = 0; ok; ++n) {
        const int ib = n & 1;
        if (!mbar_wait(bar(&ctl->info_full[ib]), (n >> 1) & 1, p.dev_status)) { ok = false; break; }
        const int unit = ctl->info_unit[ib];
        const int steps = __popc(ctl->info_mask[ib]) * KB;
        mbar_arrive(bar(&ctl->info_empty[ib]));
        if (unit < 0) break;
        const uint32_t idesc = idesc0 | ((uint32_t)(columns_of(unit) >> 3) << 17);
        for (int i = 0; i < steps; ++i) {
          if (turn == mine) {
            if (!mbar_wait(bar(&ctl->acc_empty[ab]), aphase ^ 1, p.dev_status) ||
                !mbar_wait(bar(&ctl->full[slot]), phase, p.dev_status)) { ok = false; break; }
            tc_fence_after();
            const uint64_t a = smem_desc<SP_RB>(base + slot * slot_bytes), b = smem_desc<SP_RB>(base + slot * slot_bytes + 3 * SP_PLANE);
            const uint32_t d = tmem + ab * SP_MAX_N;
#pragma unroll
            for (int q = 0; q < 6; ++q)
#pragma unroll
              for (int kk = 0; kk < SP_BK / 16; ++kk)
                umma_f16(d, a + (uint64_t)(split_a(q) * (SP_PLANE >> 4) + kk * 2), b + (uint64_t)(split_b(q) * (b_bytes >> 4) + kk * 2), idesc,
                         q + kk > 0 ? 1u : 0u);
            umma_commit(bar(&ctl->empty[slot]));
            umma_commit(bar(&ctl->acc_full[ab]));
          }
          turn ^= 1;
          if (++slot == p.slots) { slot = 0; phase ^= 1; }
          if (++ab == SP_ACCS) { ab = 0; aphase ^= 1; }
        }
      }
    }
    __syncwarp();
  } else {
    // ================================================================ sums and epilogue
    const int half = warp >> 2, row = tid & (SP_M - 1);
    int ab = 0, aphase = 0;
    for (int n = 0; ok; ++n) {
      const int ib = n & 1;
      ok = mbar_wait(bar(&ctl->info_full[ib]), (n >> 1) & 1, p.dev_status);
      if (!__all_sync(0xFFFFFFFFu, ok)) { ok = false; break; }
      const int unit = ctl->info_unit[ib];
      const int steps = unit < 0 ? 0 : __popc(ctl->info_mask[ib]) * KB;
      const int64_t m = unit < 0 ? -1 : ctl->out_row[ib][row];
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(&ctl->info_empty[ib]));
      if (unit < 0) break;
      const int bn = columns_of(unit), middle = ((bn / 16 + 1) / 2) * 16;
      const int c_begin = half ? middle : 0, cols = half ? bn - middle : middle;   // at most 64 columns a thread
      float sum[64];
#pragma unroll
      for (int i = 0; i < 64; ++i) sum[i] = 0.f;
      for (int i = 0; i < steps; ++i) {
        ok = mbar_wait(bar(&ctl->acc_full[ab]), aphase, p.dev_status);
        if (!__all_sync(0xFFFFFFFFu, ok)) { ok = false; break; }
        tc_fence_after();
        const uint32_t at = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(ab * SP_MAX_N + c_begin);
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
        if (++ab == SP_ACCS) { ab = 0; aphase ^= 1; }
      }
      if (!ok) break;
      if (p.S > 1) {   // the slices' sums are added behind the roles; every slot of the ring has been read by now
        float* dst = reinterpret_cast<float*>(smem_raw + (base - smem_u32(smem_raw))) + row * (BN + 4) + c_begin;
#pragma unroll
        for (int c = 0; c < 64; c += 4)
          if (c < cols) *reinterpret_cast<float4*>(dst + c) = make_float4(sum[c], sum[c + 1], sum[c + 2], sum[c + 3]);
      } else {
        const bool poison = *(volatile const int32_t*)p.dev_status == (int)WCN_ERR_WAIT_EXPIRED;
        const int n0 = (unit % p.blocks) * BN + c_begin;
        const bool again = m >= 0 && !poison && not_finite(sum, cols);
        if (m >= 0 && !again) {
          float* dst = p.out + m * p.out_ld + n0;
#pragma unroll
          for (int c = 0; c < 64; c += 4) {
            if (c < cols) {
              float y[4];
#pragma unroll
              for (int j = 0; j < 4; ++j) y[j] = poison ? __int_as_float(0x7FC00000) : finish(p, sum[c + j] * kSumScale, m, n0 + c + j);
              *reinterpret_cast<float4*>(dst + c) = make_float4(y[0], y[1], y[2], y[3]);
            }
          }
        }
        // rows with such sums: four columns a lane, as many rows at once as the warp has room for
        for (uint32_t rest = __ballot_sync(0xFFFFFFFFu, again); rest;) {
          const int per = cols >> 2, at_once = 32 / per, turn = lane / per, c = (lane - turn * per) * 4;
          int r = -1;
          for (int i = 0; i < at_once && rest; ++i, rest &= rest - 1)
            if (i == turn) r = __ffs(rest) - 1;
          if (r >= 0) {
            const int64_t slot = (int64_t)tile_of(p, unit / p.blocks) * SP_M + (warp & 3) * 32 + r;
            const int64_t at = p.out_rows ? (int64_t)__ldg(&p.out_rows[slot]) : slot;
            float y[4];
            fma_four(p, slot, n0 + c, y);
#pragma unroll
            for (int j = 0; j < 4; ++j) y[j] = finish(p, y[j], at, n0 + c + j);
            *reinterpret_cast<float4*>(p.out + at * p.out_ld + n0 + c) = make_float4(y[0], y[1], y[2], y[3]);
          }
          __syncwarp();
        }
      }
    }
  }
  if (p.S > 1) {
    // Each CTA finishes 1 / S of the rows, reading the slices' sums through distributed shared memory, added in slice order.
    __syncwarp();
    cluster_meet();
    const bool poison = *(volatile const int32_t*)p.dev_status == (int)WCN_ERR_WAIT_EXPIRED;
    const int64_t m0 = (int64_t)tile_of(p, first / p.blocks) * SP_M;
    const int n0 = (first % p.blocks) * BN, per_row = columns_of(first) / 4;
    const int r0 = rank * SP_M / p.S, r1 = (rank + 1) * SP_M / p.S;
    for (int i = tid; i < (r1 - r0) * per_row; i += SP_THREADS) {
      const int r = r0 + i / per_row, c = (i % per_row) * 4;
      if (m0 + r >= p.M) break;   // rows ascend with i
      const uint32_t at = base + (uint32_t)(r * (BN + 4) + c) * 4u;
      float4 v[SP_MAX_SLICES];
#pragma unroll
      for (int q = 0; q < SP_MAX_SLICES; ++q)
        if (q < p.S) v[q] = ld_cluster(at, (uint32_t)q);
#pragma unroll
      for (int q = 1; q < SP_MAX_SLICES; ++q)
        if (q < p.S) { v[0].x += v[q].x; v[0].y += v[q].y; v[0].z += v[q].z; v[0].w += v[q].w; }
      const int64_t m = p.out_rows ? (int64_t)__ldg(&p.out_rows[m0 + r]) : m0 + r;
      float y[4] = {v[0].x * kSumScale, v[0].y * kSumScale, v[0].z * kSumScale, v[0].w * kSumScale};
      if (!poison && !(fmaf(v[0].x, 0.f, v[0].y * 0.f) + fmaf(v[0].z, 0.f, v[0].w * 0.f) == 0.f)) fma_four(p, m0 + r, n0 + c, y);
      float o[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) o[j] = poison ? __int_as_float(0x7FC00000) : finish(p, y[j], m, n0 + c + j);
      *reinterpret_cast<float4*>(p.out + m * p.out_ld + n0 + c) = make_float4(o[0], o[1], o[2], o[3]);
    }
    cluster_meet();   // no CTA leaves while another may read its sums
  }
  tc_fence_before();
  __syncthreads();
  if (warp == SP_MMA_WARP) tmem_dealloc(tmem, 512);
}

struct SplitPlan {
  int cp, block_n, blocks;
  size_t weights, rows;   // bytes of the parts of the workspace
};

SplitPlan plan_split(int64_t num_in, int K, int c_in, int c_out) {
  SplitPlan q;
  q.cp = (c_in + SP_BK - 1) / SP_BK * SP_BK;
  // As few column blocks as there can be (each gathers all rows again), about equally wide; c_out is a multiple of 16.  (Blocks
  // of one width: 64 -> 208 columns were thirteen, 100 000 room / outdoor voxels 632 / 644 us, two take 206 / 198.)
  q.blocks = (c_out + SP_MAX_N - 1) / SP_MAX_N;
  q.block_n = (c_out / 16 + q.blocks - 1) / q.blocks * 16;
  q.blocks = (c_out + q.block_n - 1) / q.block_n;
  q.weights = (size_t)K * q.cp * c_out * 6;
  q.rows = (size_t)num_in * q.cp * 6;
  return q;
}

// CTAs that can be resident at once in clusters of S (they stay inside a group of multiprocessors, whose sizes differ).
int resident_split_ctas(int S) {
  static std::atomic<int> known[64][SP_MAX_SLICES + 1];
  int dev = 0;
  if (S == 1 || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return wcn_num_sms();
  int n = known[dev][S].load(std::memory_order_relaxed);
  if (n == 0) {
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned)S;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)S); cfg.blockDim = dim3(SP_THREADS); cfg.dynamicSmemBytes = SP_SMEM;
    cfg.attrs = &attr; cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, conv_split_kernel, &cfg) != cudaSuccess || clusters < 1) {
      (void)cudaGetLastError();
      clusters = wcn_num_sms() / (2 * S);
    }
    n = clusters * S;
    known[dev][S].store(n, std::memory_order_relaxed);
  }
  return n;
}

}  // namespace

bool wcn_conv_split_supported(int K, int c_in, int c_out) {
  return K >= 1 && K <= SP_MAX_K && c_in >= 16 && c_in % 4 == 0 && c_out >= 16 && c_out % 16 == 0 && c_in <= 4096 && c_out <= 4096;
}

int64_t wcn_conv_split_workspace(int64_t num_in, int K, int c_in, int c_out) {
  const SplitPlan q = plan_split(num_in, K, c_in, c_out);
  return (int64_t)(q.weights + q.rows);
}

// (rows and weights that wcn_conv_fp32_supported takes; `workspace` on a 16-byte boundary)
int wcn_conv_split_fwd(const void* feats, int64_t num_in, int64_t feats_ld, const void* weight, const int32_t* nbr,
                       const int32_t* out_rows, int64_t M, int K, int c_in, int c_out, const float* scale, const float* shift,
                       const void* residual, int64_t residual_ld, int relu, void* out, int64_t out_ld, int split_k, void* workspace,
                       int32_t* dev_status, cudaStream_t st) {
  static bool configured[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return WCN_ERR_INITIALIZATION;
  if (!configured[dev]) {
    if (cudaFuncSetAttribute(conv_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SP_SMEM) != cudaSuccess) {
      (void)cudaGetLastError();
      return WCN_ERR_INITIALIZATION;
    }
    configured[dev] = true;
  }
  const SplitPlan q = plan_split(num_in, K, c_in, c_out);
  char* ws = (char*)workspace;
  SplitParams p = {};
  p.wplanes = ws; p.planes = ws + q.weights;
  p.feats = (const float*)feats; p.weight = (const float*)weight; p.nbr = nbr; p.out_rows = out_rows;
  p.M = M; p.in_ld = feats_ld; p.out_ld = out_ld; p.res_ld = residual_ld;
  p.K = K; p.c_in = c_in; p.cp = q.cp; p.c_out = c_out; p.num_in = (int)num_in;
  p.block_n = q.block_n; p.blocks = q.blocks;
  p.scale = scale; p.shift = shift; p.residual = (const float*)residual; p.relu = relu; p.out = (float*)out;
  p.dev_status = dev_status;
  const int64_t tiles = (M + SP_M - 1) / SP_M;
  if (tiles * q.blocks * SP_MAX_SLICES > 0x7FFFFFFFll) return WCN_ERR_UNSUPPORTED_CONFIG;
  p.tiles = (int)tiles;
  // Units that leave multiprocessors idle divide their offsets among the CTAs of a cluster.  The model: 0.4 us a slot, of K
  // offsets about 0.6 K in a tile, and what the slices' sums cost (see conv_tcgen05.cu).
  p.S = 1;
  double best = 1e30;
  for (int S = 1; S <= SP_MAX_SLICES && S <= K; ++S) {
    if (split_k > 0 && S != (split_k < SP_MAX_SLICES ? split_k < K ? split_k : K : SP_MAX_SLICES < K ? SP_MAX_SLICES : K)) continue;
    if (split_k <= 0 && S > 1 && tiles * q.blocks * S > resident_split_ctas(S)) continue;
    const double off = (K > 2 ? 0.6 * K : K) / S;
    const double us = 0.4 * (off < 1 ? 1 : off) * (q.cp / SP_BK) + (S > 1 ? 1.3 + 0.0165 * q.block_n : 0.0);
    if (us < best) { best = us; p.S = S; }
  }
  p.window = out_rows && p.S == 1 ? tile_window(M, false) / SP_M : 0;
  if (p.window) p.tail = (int)(tiles / p.window < 12 ? tiles / p.window : 12);
  const size_t slot = 3 * ((size_t)SP_PLANE + (size_t)q.block_n * SP_RB), fixed = 1024 + sizeof(SplitControl) + 64;
  p.slots = (int)((SP_SMEM - fixed) / slot);
  if (p.slots > SP_MAX_SLOTS) p.slots = SP_MAX_SLOTS;
  if (p.slots < 2) return WCN_ERR_UNSUPPORTED_CONFIG;
  const int64_t items = (num_in + (int64_t)K * c_out) * (q.cp / 8);
  int64_t blocks = (items + 511) / 512;
  if (blocks > SP_PLANE_BLOCKS) blocks = SP_PLANE_BLOCKS;
  split_planes_kernel<<<(unsigned)blocks, 256, 0, st>>>(p.feats, num_in, feats_ld, p.weight, K, c_in, q.cp, c_out, ws + q.weights, ws);
  WCN_CHECK_LAUNCH();
  cudaLaunchAttribute attr[2] = {};
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)p.S;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(tiles * q.blocks * p.S)); cfg.blockDim = dim3(SP_THREADS);
  cfg.dynamicSmemBytes = fixed + p.slots * slot;
  cfg.stream = st; cfg.attrs = attr; cfg.numAttrs = p.S > 1 ? 2 : 1;
  if (cudaLaunchKernelEx(&cfg, conv_split_kernel, p) != cudaSuccess) {
    (void)cudaGetLastError();
    return WCN_ERR_EXECUTION;
  }
  return WCN_OK;
}
