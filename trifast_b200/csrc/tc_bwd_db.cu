// Bias gradient db[j, k] = sum over pair rows i of dS[i, j, k] on the tensor cores.
//
// A work item is a 128 x 128 (j, k) tile of one (b, h) and one block of pair rows
// (a "row split"); every CTA works on exactly one item (blockIdx.x).  Per row of its item the CTA
// recomputes
//     S  = Q_i K_i^T,   dP = dO_i V_i^T        (two SS MMAs, 128 x 128 each)
//     P  = exp2(S * c + bias * log2e - lse_i * log2e),   dS = P * (dP - delta_i)
// and sums dS in fp32 registers: thread = (query row j, 32-key quarter), 32
// accumulators.  The partial of every row split is written as fp32 and the splits
// are added in split order afterwards, so the result is deterministic: no atomics.
//
// A row without an open key has P = 1/n throughout, so it needs no S and no weights (d <= 64): its dP is
// added as it is, less its delta, before the other rows, while the sums are small (n = 512, h = 4, with
// the prepare step, all rows without: 264 us walked like others, 147 so).  Summed over the rows by the
// MMAs and added once it took 118 us, and 217 in place of 221 with 15 % of the rows padded, but the
// accumulator cuts off where an fp32 addition rounds: relative error of such sums against float64 1.9e-6
// to 4e-6, row by row 1.6e-7.
//
// Warps 0-15: four elementwise warpgroups, one per 32-key quarter of the tile, so
// that four warps per scheduler cover each other's barrier, TMEM-load and MUFU
// latencies; warp 16 TMA producer (Q, dO, K, V tiles and the -lse*log2e / delta
// vectors per row, NS-deep ring); warp 17 MMA issuer; warps 18-19 idle.  TMEM: two buffers of S [0,128) and
// dP [128,256), so the MMAs of row i+1 overlap the elementwise work of row i.
//
// What bounds it: the exponential unit (1024 cycles per row and tile) and the issue slots, and the waits
// between them (n = 1024, d = 32, 148 rows: 6.1 instructions a score, issue slots 56 %, exponential unit
// 74 %); at large n the card's power limit.  The next row's
// barriers are tested under this row's sums and its mask words come with the stage (two waits and two
// global loads at the top of every row: n = 1024 1.87 ms against 1.50).  The elementwise warps walk a
// count of rows with running stages and phases: with the prepare step, h = 4, d = 32, bf16, n = 384
// 120 -> 114 us, n = 733 680 -> 630 us, n = 1024 1.50 -> 1.49 ms (each row found in the bitmap, its stage and
// phases made from its number).  Bias kept as fp32 times log2(e) in place of 16-bit pairs, columns
// in eights for the registers: 1.62 ms.
//
// Stands in for `_bwd_b` of the reference (src/trifast/triton.py:388-501), which
// loops over all rows with 16-32 wide tiles.

#include <math.h>

#include <type_traits>

#include "kernels.h"
#include "tc_common.cuh"

namespace trifast {
namespace {
using namespace tc;

constexpr float kLog2e = 1.4426950408889634f;
// Register hand-over (setmaxnreg): 640 threads launch with 96 registers each; what
// the math warpgroups gain must not exceed what the issue warpgroup releases (the
// registers a CTA did not get at launch are not part of the pool), or the request
// blocks forever.
constexpr int kRegsLaunch = 96, kRegsIssue = 32, kRegsMath = 112;
static_assert(512 * kRegsMath + 128 * kRegsIssue <= 640 * kRegsLaunch, "setmaxnreg pool");
constexpr int kTmaWarp = 16, kMmaWarp = 17;

// D = 128: a row of a tile is two 128-byte swizzle spans, and a stage holds one 64-element half
// of the four tiles (KS = 2 stages per pair row, accumulated by the MMAs).
template <int D, int NS>
struct DbCfg {
  static constexpr int KS = D > 64 ? 2 : 1;
  static constexpr int DS = D / KS;                       // head-dim elements per stage
  static constexpr int kRowBytes = DS * 2;
  static constexpr int kTileBytes = 128 * kRowBytes;
  static constexpr int kVecBytes = 128 * 4;
  static constexpr int kStageBytes = 4 * kTileBytes + 2 * kVecBytes;   // multiple of 1024
  static constexpr int kThreads = 640;
  static constexpr uint64_t kSwz = RowSwizzle<DS>::kDesc;
  static constexpr int kSbo = 8 * kRowBytes;
  static constexpr int kLiveBytes = 8192;   // one bit per row of the split (n_rows <= 65535)
  static constexpr bool kMaskedApart = KS == 1;           // rows without an open key: see above
  static constexpr int kBitBytes = (kMaskedApart ? 2 : 1) * kLiveBytes;
  static int smem_bytes() { return 1024 + 1024 + NS * kStageBytes + kBitBytes; }
  // Row splits summed inside a cluster: every CTA leaves its 128 x 128 partial in its own
  // shared memory (over the stages; rows padded by 4 floats against bank conflicts).
  static constexpr int kPartPitch = 132;
  static_assert(128 * kPartPitch * 4 <= NS * kStageBytes, "cluster partial");
};

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 ld_cluster4(uint32_t local_addr, uint32_t cta) {
  uint32_t addr;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(local_addr), "r"(cta));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr)
               : "memory");
  return v;
}

// kCluster: the CTAs of a cluster are the row splits of one tile; their partials are summed in
// split order through distributed shared memory and `out` gets the sum, so that neither
// partials in global memory nor a reduce kernel are needed.
template <typename T, int D, int NS, bool kCluster>
__global__ void __launch_bounds__(640, 1)
tc_db_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_do,
             const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
             const __grid_constant__ CUtensorMap map_nlse, const __grid_constant__ CUtensorMap map_delta,
             View4 bias, const uint8_t* __restrict__ rowfull, const uint32_t* __restrict__ maskbits,
             int mask_words, const uint32_t* __restrict__ rowrange, float* __restrict__ out,
             int splits, Dims dm, unsigned int* status) {
  using Cfg = DbCfg<D, NS>;
  constexpr int FULL = 0, EMPTY = FULL + NS, S_FULL = EMPTY + NS, S_FREE = S_FULL + 2,
                NBARS = S_FREE + 2;
  static_assert(NBARS * 8 <= 256, "barrier area");
  static_assert(Cfg::kStageBytes % 1024 == 0, "stage alignment");

  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* gbase = smem_raw + (base - raw);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gbase + 256);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gbase + 260);
  // per stage: the row's key-mask words of this key tile (four, bit set = dropped) and, where rows
  // without an open key are not kept apart, its flag
  volatile uint32_t* info = reinterpret_cast<volatile uint32_t*>(gbase + 320);   // [NS][8]

  const int n = dm.n;
  constexpr uint32_t tiles_off = 1024;
  auto bar = [&](int i) -> uint32_t { return base + 8u * i; };
  auto stage_off = [&](int s) -> uint32_t { return tiles_off + s * Cfg::kStageBytes; };
  auto q_tile = [&](int s) -> uint32_t { return base + stage_off(s); };
  auto do_tile = [&](int s) -> uint32_t { return base + stage_off(s) + Cfg::kTileBytes; };
  auto k_tile = [&](int s) -> uint32_t { return base + stage_off(s) + 2 * Cfg::kTileBytes; };
  auto v_tile = [&](int s) -> uint32_t { return base + stage_off(s) + 3 * Cfg::kTileBytes; };
  auto nlse_off = [&](int s) -> uint32_t { return stage_off(s) + 4 * Cfg::kTileBytes; };
  auto delta_off = [&](int s) -> uint32_t { return nlse_off(s) + Cfg::kVecBytes; };

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&map_q);
    tma_prefetch_desc(&map_do);
    tma_prefetch_desc(&map_k);
    tma_prefetch_desc(&map_v);
    tma_prefetch_desc(&map_nlse);
    tma_prefetch_desc(&map_delta);
  }
  after_previous();

  // (a cluster's CTAs must all reach its barriers: they skip the rows instead)
  if (!kCluster && *reinterpret_cast<volatile unsigned int*>(status) != 0u) return;
  volatile int* skip = reinterpret_cast<volatile int*>(gbase + 264);

  const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;
  const int tiles_k = (n + 127) / 128;
  const int tiles = tiles_k * tiles_k;
  // Rows of a split: every splits-th one, the same for every tile (a batch's padded rows lie
  // together: as one block they would be one split's lot).
  struct Item {
    int jt, kt, split, bh, b, h, nrows;
  };
  // item order: tile fastest, then split, then (b, h): the CTAs running together work
  // on the same rows of the same (b, h), so the Q/dO/K/V row tiles are shared in L2
  // (split fastest with clusters, whose CTAs are consecutive)
  auto decode = [&](int w) {
    Item im;
    const int tile = kCluster ? (w / splits) % tiles : w % tiles;
    const int rest = w / tiles;
    im.jt = tile / tiles_k;
    im.kt = tile % tiles_k;
    im.split = kCluster ? w % splits : rest % splits;
    im.bh = rest / splits;
    im.b = im.bh / dm.heads;
    im.h = im.bh % dm.heads;
    im.nrows = (dm.n_rows - im.split + splits - 1) / splits;
    return im;
  };

  if (tid == 0) {
    for (int s = 0; s < NS; ++s) {
      mbar_init(bar(FULL + s), 1);
      mbar_init(bar(EMPTY + s), 1 + 16);  // MMA commit + 16 elementwise warps (vectors read)
    }
    for (int u = 0; u < 2; ++u) {
      mbar_init(bar(S_FULL + u), 1);
      mbar_init(bar(S_FREE + u), 16);
    }
    *abort_flag = 0;
    if (kCluster) *skip = *reinterpret_cast<volatile unsigned int*>(status) != 0u;
    mbar_fence_init();
  }
  if (warp == kMmaWarp) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  // Rows of this split whose live key-tile range holds this item's key tile, one bit per
  // row: the others weigh all 128 keys of the tile zero and add nothing to db, so no role
  // touches them.  (A fully masked row's range is every tile.)
  uint32_t* live = reinterpret_cast<uint32_t*>(gbase + tiles_off + NS * Cfg::kStageBytes);
  uint32_t* masked = live + Cfg::kLiveBytes / 4;   // (kMaskedApart) rows without an open key
  {
    const Item im = decode(blockIdx.x);
    for (int w0 = warp * 32; w0 < im.nrows; w0 += 32 * (Cfg::kThreads / 32)) {
      const int g = w0 + lane;
      bool on = false, none = false;
      if (g < im.nrows) {
        const int row = im.b * dm.n_rows + im.split + g * splits;
        const uint32_t v = rowrange ? __ldg(rowrange + row) : 0xffff0000u;
        on = (uint32_t)im.kt >= (v & 0xffffu) && (uint32_t)im.kt < (v >> 16);
        if (Cfg::kMaskedApart) {
          none = rowfull[row] != 0;
          on = on && !none;
        }
      }
      const uint32_t bits = __ballot_sync(0xffffffffu, on);
      const uint32_t apart = __ballot_sync(0xffffffffu, none);
      if (lane == 0) {
        live[w0 >> 5] = bits;
        if (Cfg::kMaskedApart) masked[w0 >> 5] = apart;
      }
    }
  }
  // (the roles walk the set bits word by word: one shared-memory read per 32 rows, nothing
  // per row)
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = uniform(*tmem_slot);
  const bool skipped = kCluster && *skip != 0;

  if (warp >= kTmaWarp) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsIssue));
    if (warp == kTmaWarp) {
      // ---------------------------------------------------------- TMA producer
      // (The whole warp runs the loop: its first lanes bring what info holds, which travels with
      // the stage.)
      constexpr int kInfo = Cfg::kMaskedApart ? 4 : 5;
      const Item im = decode(blockIdx.x);
      int g = 0;
      bool ok = !skipped;
      if constexpr (Cfg::kMaskedApart) {
        for (int r0 = 0; r0 < im.nrows && ok; r0 += 32) {
          for (uint32_t bits = uniform(masked[r0 >> 5]); bits != 0u && ok; bits &= bits - 1u, ++g) {
            const int i = im.split + (r0 + __ffs(bits) - 1) * splits, s = g % NS;
            if (g >= NS) ok = __all_sync(0xffffffffu, mbar_wait(bar(EMPTY + s), ((g / NS) - 1) & 1, abort_flag));
            if (!ok) break;
            if (elect_one()) {
              mbar_arrive_expect_tx(bar(FULL + s), 2 * Cfg::kTileBytes + Cfg::kVecBytes);
              tma_load_5d(do_tile(s), &map_do, bar(FULL + s), 0, im.jt * 128, i, im.h, im.b);
              tma_load_5d(v_tile(s), &map_v, bar(FULL + s), 0, im.kt * 128, i, im.h, im.b);
              tma_load_4d(base + delta_off(s), &map_delta, bar(FULL + s), im.jt * 128, i, im.h, im.b);
            }
            __syncwarp();
          }
        }
      }
      for (int r0 = 0; r0 < im.nrows && ok; r0 += 32) {
        for (uint32_t bits = uniform(live[r0 >> 5]); bits != 0u && ok; bits &= bits - 1u) {
          const int i = im.split + (r0 + __ffs(bits) - 1) * splits;
          const int64_t row = (int64_t)im.b * dm.n_rows + i;
          uint32_t word = 0u;
          if (lane < 4) word = __ldg(maskbits + row * mask_words + im.kt * 4 + lane);
          if (!Cfg::kMaskedApart && lane == 4) word = rowfull[row];
          for (int c = 0; c < Cfg::KS; ++c, ++g) {
            const int s = g % NS;
            if (g >= NS) ok = __all_sync(0xffffffffu, mbar_wait(bar(EMPTY + s), ((g / NS) - 1) & 1, abort_flag));
            if (!ok) break;
            if (c == Cfg::KS - 1 && lane < kInfo) info[s * 8 + lane] = word;
            __syncwarp();
            if (elect_one()) {
              const int c0 = c * Cfg::DS;
              mbar_arrive_expect_tx(bar(FULL + s), Cfg::kStageBytes);
              tma_load_5d(q_tile(s), &map_q, bar(FULL + s), c0, im.jt * 128, i, im.h, im.b);
              tma_load_5d(do_tile(s), &map_do, bar(FULL + s), c0, im.jt * 128, i, im.h, im.b);
              tma_load_5d(k_tile(s), &map_k, bar(FULL + s), c0, im.kt * 128, i, im.h, im.b);
              tma_load_5d(v_tile(s), &map_v, bar(FULL + s), c0, im.kt * 128, i, im.h, im.b);
              tma_load_4d(base + nlse_off(s), &map_nlse, bar(FULL + s), im.jt * 128, i, im.h, im.b);
              tma_load_4d(base + delta_off(s), &map_delta, bar(FULL + s), im.jt * 128, i, im.h, im.b);
            }
            __syncwarp();
          }
        }
      }
    } else if (warp == kMmaWarp) {
      // ---------------------------------------------------------- MMA issuer
      {
        constexpr bool kBf16 = std::is_same<T, __nv_bfloat16>::value;
        constexpr uint32_t idesc = make_idesc(128, 128, kBf16, false, false);
        bool ok = !skipped;
        {
          const int nrows = decode(blockIdx.x).nrows;
          int g = 0;
          if constexpr (Cfg::kMaskedApart) {   // rows without an open key: dP alone
            for (int r0 = 0; r0 < nrows && ok; r0 += 32) {
              for (uint32_t bits = uniform(masked[r0 >> 5]); bits != 0u; bits &= bits - 1u, ++g) {
                const int s = g % NS, u = g & 1;
                ok = (g < 2 || mbar_wait(bar(S_FREE + u), ((g >> 1) - 1) & 1, abort_flag)) &&
                     mbar_wait(bar(FULL + s), (g / NS) & 1, abort_flag);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                tc_fence_after();
                const uint64_t ag = make_smem_desc(do_tile(s), 16, Cfg::kSbo, Cfg::kSwz);
                const uint64_t bv = make_smem_desc(v_tile(s), 16, Cfg::kSbo, Cfg::kSwz);
                if (elect_one()) {
#pragma unroll
                  for (int kk = 0; kk < Cfg::DS / 16; ++kk)
                    umma_ss(tmem_base + u * 256 + 128, ag + 2 * kk, bv + 2 * kk, idesc, kk > 0);
                  umma_commit(bar(S_FULL + u));
                  umma_commit(bar(EMPTY + s));
                }
                __syncwarp();
              }
            }
          }
          for (int r0 = 0; r0 < nrows && ok; r0 += 32) {
          for (uint32_t bits = uniform(live[r0 >> 5]); bits != 0u && ok; bits &= bits - 1u) {
            const int u = g & 1;
            if (g >= 2) ok = mbar_wait(bar(S_FREE + u), ((g >> 1) - 1) & 1, abort_flag);
            for (int c = 0; c < Cfg::KS; ++c) {
              const int sg = g * Cfg::KS + c, s = sg % NS;
              ok = __all_sync(0xffffffffu, ok && mbar_wait(bar(FULL + s), (sg / NS) & 1, abort_flag));
              if (!ok) break;
              tc_fence_after();
              const uint64_t aq = make_smem_desc(q_tile(s), 16, Cfg::kSbo, Cfg::kSwz);
              const uint64_t bk = make_smem_desc(k_tile(s), 16, Cfg::kSbo, Cfg::kSwz);
              const uint64_t ag = make_smem_desc(do_tile(s), 16, Cfg::kSbo, Cfg::kSwz);
              const uint64_t bv = make_smem_desc(v_tile(s), 16, Cfg::kSbo, Cfg::kSwz);
              if (elect_one()) {   // (a K slice of 16 elements is 32 bytes further along the row)
#pragma unroll
                for (int kk = 0; kk < Cfg::DS / 16; ++kk)
                  umma_ss(tmem_base + u * 256, aq + 2 * kk, bk + 2 * kk, idesc, c > 0 || kk > 0);
#pragma unroll
                for (int kk = 0; kk < Cfg::DS / 16; ++kk)
                  umma_ss(tmem_base + u * 256 + 128, ag + 2 * kk, bv + 2 * kk, idesc, c > 0 || kk > 0);
                if (c == Cfg::KS - 1) umma_commit(bar(S_FULL + u));
                umma_commit(bar(EMPTY + s));
              }
              __syncwarp();
            }
            if (!ok) break;
            ++g;
          }
          }
        }
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsMath));
    // ------------------------------------------------------------ elementwise warpgroups
    const int quarter = warp >> 2, wq = warp & 3, row = tid & 127;
    const uint32_t lane_base = (uint32_t)(wq * 32) << 16;
    const float c1 = in_register(dm.scale * kLog2e), log2e = in_register(kLog2e);
    const float p_full = 1.f / (float)n;

    bool ok = !skipped;
    {
      const Item im = decode(blockIdx.x);
      const int b = im.b, h = im.h, kt = im.kt;
      const int j = im.jt * 128 + row;
      const int key0 = kt * 128 + quarter * 32;

      // where this thread's 32 sums go, settled now so that the item's indices need not
      // stay live through the row loop
      float* const dst =
          out + (((int64_t)im.split * dm.batch * dm.heads + im.bh) * n + min(j, n - 1)) * n + key0;
      const int n_store = (j < n) ? min(32, n - key0) : 0;  // <= 0: nothing to store

      float acc[32];
      uint32_t bp[16];  // this thread's 32 bias values, kept as 16-bit pairs
      {
        const T* brow = reinterpret_cast<const T*>(bias.p) + b * bias.sb + h * bias.sh +
                        (int64_t)min(j, n - 1) * bias.sj + key0;
#pragma unroll
        for (int c = 0; c < 32; ++c) acc[c] = 0.f;
        if (key0 + 32 <= n && (reinterpret_cast<uintptr_t>(brow) & 15) == 0) {
          // four 16-byte loads: a lane reads its own row, so every load instruction
          // touches 32 lines; 2-byte loads would take 32 such instructions
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const uint4 u = __ldg(reinterpret_cast<const uint4*>(brow) + c);
            bp[4 * c + 0] = u.x;
            bp[4 * c + 1] = u.y;
            bp[4 * c + 2] = u.z;
            bp[4 * c + 3] = u.w;
          }
        } else {
#pragma unroll
          for (int c = 0; c < 32; c += 2) {
            const float b0 = (key0 + c < n) ? to_f32<T>(brow[c]) : 0.f;
            const float b1 = (key0 + c + 1 < n) ? to_f32<T>(brow[c + 1]) : 0.f;
            bp[c >> 1] = pack2<T>(b0, b1);  // exact: the values are 16-bit already
          }
        }
      }
      // live rows of the item (which ones they are is the producer's business)
      int count = 0;
      for (int w0 = lane; w0 * 32 < im.nrows; w0 += 32) count += __popc(live[w0]);
      count = __reduce_add_sync(0xffffffffu, count);
      // stage and phases kept as such: made from the row's number they cost twenty instructions a row
      int s = 0, g = 0;
      uint32_t ring = 0u, u = 0u, turn = 0u;
      auto next_stage = [&]() {
        if (++s == NS) {
          s = 0;
          ring ^= 1u;
        }
      };
      if constexpr (Cfg::kMaskedApart) {
        int without = 0;   // rows without an open key
        for (int w0 = lane; w0 * 32 < im.nrows; w0 += 32) without += __popc(masked[w0]);
        without = __reduce_add_sync(0xffffffffu, without);
        for (int e = 0; e < without; ++e) {
          ok = mbar_wait(bar(FULL + s), ring, abort_flag) && mbar_wait(bar(S_FULL + u), turn, abort_flag);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tc_fence_after();
          const float dl = reinterpret_cast<const float*>(gbase + delta_off(s))[row];
          float gd[32];
          tmem_ld32(tmem_base + lane_base + u * 256 + 128 + quarter * 32, reinterpret_cast<uint32_t*>(gd));
          tmem_wait_ld();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) {
            mbar_arrive(bar(S_FREE + u));
            mbar_arrive(bar(EMPTY + s));
          }
          next_stage();
          turn ^= u;
          u ^= 1u;
#pragma unroll
          for (int c = 0; c < 32; ++c) acc[c] = fmaf(p_full, gd[c] - dl, acc[c]);
        }
      }
      bool there = false;   // the next row's barriers, tested while this one's sums are made
      for (; ok && g < count; ++g) {
        // (with KS stages per row the vectors are read from the last one; the earlier ones are
        // released as they come, untouched)
        if (Cfg::KS > 1) {
          ok = __all_sync(0xffffffffu, mbar_wait(bar(FULL + s), ring, abort_flag));
          if (!ok) break;
          if (lane == 0) mbar_arrive(bar(EMPTY + s));
          next_stage();
        }
        if (!__all_sync(0xffffffffu, there)) {
          ok = mbar_wait(bar(FULL + s), ring, abort_flag) && mbar_wait(bar(S_FULL + u), turn, abort_flag);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
        }
        tc_fence_after();
        const float nl = reinterpret_cast<const float*>(gbase + nlse_off(s))[row];
        const float dl = reinterpret_cast<const float*>(gbase + delta_off(s))[row];
        const uint32_t mw = info[s * 8 + quarter];
        bool row_full = false;
        if constexpr (!Cfg::kMaskedApart) row_full = info[s * 8 + 4] != 0u;
        const float ndl = -dl;
        const uint32_t tS = tmem_base + lane_base + u * 256 + quarter * 32;
        const uint32_t tDP = tS + 128;
#pragma unroll
        for (int hc = 0; hc < 2; ++hc) {
          float x[16], gd[16];
          tmem_ld16(tS + hc * 16, reinterpret_cast<uint32_t*>(x));
          tmem_ld16(tDP + hc * 16, reinterpret_cast<uint32_t*>(gd));
          tmem_wait_ld();
          if (hc == 1) {  // everything this warp needs from the buffer is in registers
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
              mbar_arrive(bar(S_FREE + u));
              mbar_arrive(bar(EMPTY + s));   // (the vectors and the mask, read above)
            }
            next_stage();
            turn ^= u;
            u ^= 1u;
            if constexpr (Cfg::KS == 1)
              there = mbar_test_wait(bar(FULL + s), ring) && mbar_test_wait(bar(S_FULL + u), turn);
          }
          const uint32_t mh = (mw >> (hc * 16)) & 0xffffu;
          if (row_full) {
#pragma unroll
            for (int c = 0; c < 16; ++c) {
              const float p = ((mh >> c) & 1u) ? 0.f : p_full;
              acc[hc * 16 + c] = fmaf(p, gd[c] - dl, acc[hc * 16 + c]);
            }
          } else if (mh == 0u) {  // no dropped key: a straight block the compiler can overlap
#pragma unroll
            for (int c = 0; c < 16; c += 2) {  // packed fp32 pairs: two scores per FMA instruction
              float b0, b1, t0, t1, a0, a1, s0, s1;
              unpack2<T>(bp[(hc * 16 + c) >> 1], b0, b1);
              ffma2(t0, t1, b0, b1, log2e, log2e, nl, nl);
              ffma2(a0, a1, x[c], x[c + 1], c1, c1, t0, t1);
              const float p0 = ex2(a0), p1 = ex2(a1);
              fadd2(s0, s1, gd[c], gd[c + 1], ndl, ndl);
              ffma2(acc[hc * 16 + c], acc[hc * 16 + c + 1], p0, p1, s0, s1, acc[hc * 16 + c],
                    acc[hc * 16 + c + 1]);
            }
          } else {
#pragma unroll
            for (int c = 0; c < 16; c += 2) {
              float b0, b1, t0, t1, a0, a1, s0, s1;
              unpack2<T>(bp[(hc * 16 + c) >> 1], b0, b1);
              ffma2(t0, t1, b0, b1, log2e, log2e, nl, nl);
              ffma2(a0, a1, x[c], x[c + 1], c1, c1, t0, t1);
              float p0 = ex2(a0), p1 = ex2(a1);
              p0 = ((mh >> c) & 1u) ? 0.f : p0;
              p1 = ((mh >> (c + 1)) & 1u) ? 0.f : p1;
              fadd2(s0, s1, gd[c], gd[c + 1], ndl, ndl);
              ffma2(acc[hc * 16 + c], acc[hc * 16 + c + 1], p0, p1, s0, s1, acc[hc * 16 + c],
                    acc[hc * 16 + c + 1]);
            }
          }
        }
      }
      if (kCluster) {
        // the last row's S_FULL has completed every load and MMA that used the stages, for all
        // warps alike once the cluster barrier below is passed; here a named barrier of the
        // elementwise warps orders their last reads of the vectors before the partials
        asm volatile("bar.sync 1, 512;" ::: "memory");
        float* part = reinterpret_cast<float*>(gbase + tiles_off) + row * Cfg::kPartPitch + quarter * 32;
#pragma unroll
        for (int c = 0; c < 32; c += 4)
          *reinterpret_cast<float4*>(part + c) = make_float4(acc[c], acc[c + 1], acc[c + 2], acc[c + 3]);
      } else if (ok && n_store > 0) {
        if (n_store == 32 && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
#pragma unroll
          for (int c = 0; c < 32; c += 4)
            *reinterpret_cast<float4*>(dst + c) = make_float4(acc[c], acc[c + 1], acc[c + 2], acc[c + 3]);
        } else {
#pragma unroll
          for (int c = 0; c < 32; ++c)
            if (c < n_store) dst[c] = acc[c];
        }
      }
    }
  }

  if (kCluster) {
    // each CTA sums its share of the tile's rows over the cluster, in split order; the second
    // barrier keeps a CTA's shared memory alive until its readers are done
    __syncwarp();
    cluster_sync();
    const Item im = decode(blockIdx.x);
    const int share = 128 / splits, r0 = im.split * share;
    if (!skipped && *abort_flag == 0) {
      for (int idx = tid; idx < share * 32; idx += Cfg::kThreads) {
        const int r = r0 + (idx >> 5), c = (idx & 31) * 4;
        const uint32_t at = base + tiles_off + (r * Cfg::kPartPitch + c) * 4;
        float4 sum = ld_cluster4(at, 0);
        for (int k = 1; k < splits; ++k) {
          const float4 v = ld_cluster4(at, k);
          sum.x += v.x;
          sum.y += v.y;
          sum.z += v.z;
          sum.w += v.w;
        }
        const int j = im.jt * 128 + r, key = im.kt * 128 + c;
        if (j < n && key < n) {
          float* dst = out + ((int64_t)im.bh * n + j) * n + key;
          if (key + 4 <= n && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
            *reinterpret_cast<float4*>(dst) = sum;
          } else {
            const float e[4] = {sum.x, sum.y, sum.z, sum.w};
            for (int k = 0; k < 4 && key + k < n; ++k) dst[k] = e[k];
          }
        }
      }
    }
    cluster_sync();
  }

  // ---------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    const long long t0 = clock64();
    while (clock64() - t0 < 4000000LL) {
    }
    if (tid == 0) set_status(status, kStatusTimeoutBwdDb);
    __syncthreads();
  }
  if (warp == kMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

template <typename T, int D, int NS, bool kCluster = false>
cudaError_t launch_db(const BwdArgs& a, cudaStream_t stream) {
  using Cfg = DbCfg<D, NS>;
  const Dims& dm = a.dm;
  const bool bf16 = std::is_same<T, __nv_bfloat16>::value;
  const uint64_t eb = 2;
  CUtensorMap mq, mdo, mk, mv, mnl, mdl;
  const uint64_t dims5[5] = {(uint64_t)D, (uint64_t)dm.n, (uint64_t)dm.n_rows, (uint64_t)dm.heads,
                             (uint64_t)dm.batch};
  const uint32_t box[5] = {(uint32_t)Cfg::DS, 128, 1, 1, 1};
  const CUtensorMapSwizzle swz = (CUtensorMapSwizzle)RowSwizzle<Cfg::DS>::kTma;
  auto map5 = [&](CUtensorMap* m, const View5& v) {
    const uint64_t st[4] = {(uint64_t)v.sj * eb, (uint64_t)v.si * eb, (uint64_t)v.sh * eb,
                            (uint64_t)v.sb * eb};
    return make_tensor_map(m, bf16, 5, v.p, dims5, st, box, swz);
  };
  if (!map5(&mq, a.q) || !map5(&mdo, a.d_o) || !map5(&mk, a.k) || !map5(&mv, a.v))
    return cudaErrorInvalidValue;
  {
    const uint64_t n = dm.n, np = dm.n_pad, rows = dm.n_rows;
    const uint64_t dims4[4] = {n, rows, (uint64_t)dm.heads, (uint64_t)dm.batch};
    const uint64_t st[3] = {np * 4, np * rows * 4, np * rows * dm.heads * 4};
    const uint32_t box4[4] = {128, 1, 1, 1};
    if (!make_tensor_map_f32(&mnl, 4, a.neg_lse2, dims4, st, box4) ||
        !make_tensor_map_f32(&mdl, 4, a.delta, dims4, st, box4))
      return cudaErrorInvalidValue;
  }
  const int smem = Cfg::smem_bytes();
  constexpr auto kern = tc_db_kernel<T, D, NS, kCluster>;
  cudaError_t e = opt_in_smem<kern>(smem);
  if (e != cudaSuccess) return e;
  const int t = (dm.n + 127) / 128;
  const int total = t * t * a.splits * dm.batch * dm.heads;
  const int grid = total;  // one item per CTA
  float* out = a.splits > 1 && !kCluster ? a.db_partials : a.db_f32;
  View4 bias = a.bias;
  if (a.bias_pad) {  // the copy with a 16-byte row pitch: its rows can be read 16 bytes at a time
    bias.p = (char*)a.bias_pad;
    bias.sj = dm.n_pad;
    bias.sh = (int64_t)dm.n * dm.n_pad;
    bias.sb = bias.sh * dm.heads;
    bias.sk = 1;
  }
  if (kCluster) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = a.splits;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // (as launch_early)
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(Cfg::kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, kern, mq, mdo, mk, mv, mnl, mdl, bias, (const uint8_t*)a.rowfull,
                              (const uint32_t*)a.maskbits_lin, a.mask_words, (const uint32_t*)a.rowrange,
                              out, a.splits, dm, a.status);
  }
  return launch_early(kern, grid, Cfg::kThreads, smem, stream, mq, mdo, mk, mv, mnl, mdl, bias, a.rowfull,
                                              a.maskbits_lin, a.mask_words, a.rowrange, out, a.splits,
                                              dm, a.status);
}

}  // namespace

// Row splits of a tile when a cluster sums them (a power of two up to 8, the portable cluster
// size): the count whose rounds of CTAs over the SMs, each lasting a split's rows and about
// six rows' time of prologue and exchange, end first.
int tc_db_cluster_splits(int64_t tiles, int n_rows, int sms) {
  int best = 1;
  int64_t best_cost = INT64_MAX;
  for (int s = 1; s <= 8 && n_rows / s >= 8; s *= 2) {
    const int64_t cost = ((tiles * s + sms - 1) / sms) * ((n_rows + s - 1) / s + 6);
    if (cost < best_cost) {
      best_cost = cost;
      best = s;
    }
  }
  return best;
}

// Row splits of a tile whose partials go through global memory (d <= 64), up to `most`: the same
// estimate with the 9 rows' time (8 us) that a CTA's start and end measure there, and the
// partials' way to memory and back at 5 TB/s, a row taking 0.85 us (by now about 0.75; the picks below are the same).
// The constants were fitted at d = 32; timed with this kernel against every count up to `most` at d = 16,
// 32 and 64 (h = 4, n = 97, 128, 192, 256, 384, 512, 733, 1024), the pick was the fastest each time, and
// so with 15 % of rows and keys padded, which the host does not know of, but for n = 1024, where 3 splits
// in place of 4 take 4 % less (d = 32 1271 against 1323 us).  Against clusters of
// 2 to 8 at n = 97 to 1024 (d = 32): faster everywhere but at n = 512 (equal), since clusters leave
// SMs idle.
int tc_db_splits(int64_t tiles, int n_rows, int sms, int64_t partial_bytes, int most) {
  int best = 1;
  double best_cost = 1e30;
  for (int s = 1; s <= most; ++s) {
    const double cost = (double)((tiles * s + sms - 1) / sms) * ((n_rows + s - 1) / s + 9) +
                        (s > 1 ? s * (2.0 * partial_bytes / 5e6) / 0.85 : 0.0);
    if (cost < best_cost) {
      best_cost = cost;
      best = s;
    }
  }
  return best;
}

cudaError_t tc_bwd_db(const BwdArgs& a, cudaStream_t s) {
  const bool bf16 = a.dtype == TRIFAST_BF16;
  if (!a.neg_lse2 || !a.maskbits_lin) return cudaErrorInvalidValue;
  switch (a.dm.d) {
    case 16: return bf16 ? launch_db<__nv_bfloat16, 16, 4>(a, s) : launch_db<__half, 16, 4>(a, s);
    case 32: return bf16 ? launch_db<__nv_bfloat16, 32, 4>(a, s) : launch_db<__half, 32, 4>(a, s);
    case 64: return bf16 ? launch_db<__nv_bfloat16, 64, 3>(a, s) : launch_db<__half, 64, 3>(a, s);
    default: return bf16 ? launch_db<__nv_bfloat16, 128, 3, true>(a, s) : launch_db<__half, 128, 3, true>(a, s);
  }
}

}  // namespace trifast
