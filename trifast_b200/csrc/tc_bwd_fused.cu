// dq, dk and dv of triangle attention in ONE pass over the scores (bf16 / fp16).
//
// A work item is one pair row i of one (b, h): the CTA walks the row's key tiles
// (128 keys, outer loop) and, per key tile, its queries in steps of 64 (inner loop),
// and evaluates every score exactly once.  Everything is computed transposed, keys
// on the TMEM lanes:
//     S^T  = K Q^T,  dP^T = V dO^T                      (SS MMAs, 128 keys x 64 queries)
//     P^T  = exp2(S^T * c + bias^T * log2e - lse_j * log2e),  dS^T = P^T * (dP^T - delta_j)
//     dV  += P^T dO,  dK += dS^T Q                      (A = P^T / dS^T from TMEM)
//     dQ  += dS K                                       (A = dS from shared memory)
// dK and dV of the current key tile and dQ of the WHOLE row stay in TMEM: dK / dV
// are written out after each key tile, dQ once per row.  dS is needed in both
// orientations; the elementwise threads (one key each) write their dS^T rows to TMEM
// for dK and, as 16-bit, to a shared-memory tile whose rows are keys and whose columns
// are queries; read as an MN-major A operand that tile is dS.  One dQ MMA (128 queries
// x D, K = 128 keys) is issued per pair of steps.
//
// The reference computes dq and dk/dv in two kernels that each recompute S, P and
// dS (src/trifast/triton.py:268-383 _bwd_q, :137-263 _bwd_kv); this kernel replaces
// both with one exponential per score.
//
// Warps 0-15: elementwise, two groups of eight that take the steps in turn; 16 TMA producer;
// 17 issues the S and dP MMAs (and owns the TMEM allocation), 18 the dV / dK MMAs (and, with two S
// buffers, S), 19 the dQ MMAs; 20-23 write dK, dV and dQ.  TMEM columns: SB buffers of S^T (64 each,
// overwritten by the step's P^T and dS^T as 16-bit pairs), PB buffers of dP^T (64), AB pairs of dK and
// dV (D each), dQ with D columns per 128-query tile.  The dQ of eight tiles (d = 32: n = 1024) or
// three (d = 64: n = 384) fits beside the fewest buffers.  Longer rows are walked in query chunks of
// equal length: per chunk all key tiles are swept again (S, P, dS of a chunk's queries are still evaluated
// once), dQ of the chunk leaves at its end, and dK / dV of a key tile are completed over the chunks:
// the partial of the earlier chunks waits as fp32 in a per-CTA scratch (written and read by the same
// thread, L2-resident).
//
// What bounds it: the chain of a step, S^T -> registers -> P^T, dS^T -> accumulating MMAs -> the
// next S^T in that place, which takes about 3400 cycles, of which a group's arithmetic takes
// 1800 (the exponential unit 512 cycles a step, the tensor pipe 560; n = 1024, d = 32, 148 rows, two S buffers:
// 12.2 instructions a score, issue slots 53 %, exponential unit 35 %).  With
// three S buffers (as far as six tiles of dQ) a step is started every 1250 cycles, with two every
// 1550.  Time at h = 4, bf16, before and after (one group of eight warps that also wrote the results, S and P
// in places of their own): d = 32, n = 256 86 -> 61 us, n = 512 (15 % padding) 456 -> 333, n = 733 1354 -> 977,
// n = 1024 3.20 -> 2.83 ms, n = 2048 (10 %) 26.4 -> 21.3 ms; d = 64, n = 1024 8.90 -> 5.7 ms.  n = 1024 in two chunks with
// three S buffers takes 2.47 ms, but sums dk and dv in another order and needs the scratch.
// At d = 64 the third S buffer would leave dQ two tiles instead of three: 7.80 ms.
//
// Masked keys weigh exactly zero; rows whose keys are all masked use P = 1/n over
// the n keys (the PyTorch semantics, src/trifast/equiv.py:42-69).

#include <math.h>

#include <type_traits>

#include "kernels.h"
#include "tc_common.cuh"

namespace trifast {
namespace {
using namespace tc;

constexpr int kBKeys = 128, kBJ = 64;
constexpr float kLog2e = 1.4426950408889634f;
constexpr int kSmemLimit = 232448;
constexpr int kFusedMaxCtas = 160;  // grid cap: the per-CTA dK / dV scratch is sized by it
// Register hand-over (setmaxnreg): 768 threads launch with 80 registers each; what the
// math warpgroups gain must not exceed what the other two release, or the request
// blocks forever.
constexpr int kRegsLaunch = 80, kRegsIssue = 40, kRegsOut = 56, kRegsMath = 96;
static_assert(512 * kRegsMath + 128 * (kRegsIssue + kRegsOut) <= 768 * kRegsLaunch, "setmaxnreg pool");
constexpr int kTmaWarp = 16, kOutWarp = 20;
// Stages of the ring.
template <int D> constexpr int kFusedStages = D == 64 ? 3 : 5;

template <int D, int NS, int SB, int PB, int AB>
struct FusedCfg {
  static constexpr int kRowBytes = D * 2;
  static constexpr int kKVBytes = 128 * kRowBytes;       // resident K or V tile
  static constexpr int kQBytes = kBJ * kRowBytes;        // streamed Q or dO tile
  static constexpr int kBiasBytes = 128 * kBJ * 2;       // bias^T tile: 128 keys x 64 queries
  static constexpr int kVecBytes = kBJ * 4;              // -lse*log2e or delta of 64 queries
  static constexpr int kStageBytes = 2 * kQBytes + kBiasBytes;   // (the vectors lie in the header)
  static constexpr int kHalfBytes = 128 * kBJ * 2;       // dS of one step: 128 keys x 64 queries
  static constexpr int kPairBytes = 2 * kHalfBytes;      // dS of a pair of steps: 128 x 128
  static constexpr int kTilesBytes = 4 * kKVBytes + NS * kStageBytes + 2 * kPairBytes;
  static constexpr int kThreads = 768;
  static constexpr uint64_t kSwz = RowSwizzle<D>::kDesc;
  static constexpr int kSbo = 8 * kRowBytes;
  // TMEM columns: SB buffers of S^T (64 each, overwritten by P^T and dS^T), PB buffers of dP^T (64
  // each), AB pairs of dK, dV (D each) and dQ, D columns per 128-query tile
  // (an accumulator of D = 16 columns still starts on a multiple of 32 columns)
  static constexpr int kAcc = D < 32 ? 32 : D;
  static constexpr int kDpCol = SB * 64, kDkCol = kDpCol + PB * 64, kDvCol = kDkCol + kAcc;
  static constexpr int kDqCol = kDkCol + AB * 2 * kAcc;     // first dQ column
  static constexpr int kMaxJTiles = (512 - kDqCol) / kAcc;  // 128-query tiles whose dQ fits
  static constexpr bool kChunks = AB == 1;                  // rows may be walked in several query chunks
  static constexpr int kVecOff = 1024, kHeader = (kVecOff + NS * 2 * kVecBytes + 1023) / 1024 * 1024;
  static constexpr int kSmemBytes = kHeader + kTilesBytes;   // (the base is aligned to 1024 bytes)
};

struct FusedGrid {
  int total;     // work items = batch * heads * n_rows
  int nkt;       // key tiles of 128
  int njs;       // query steps of 64
  int njt;       // query tiles of 128 (dQ tiles)
  int nch;       // query chunks: a row whose dQ does not fit TMEM is walked chunk by chunk
  int jsc;       // query steps per full chunk (even)
};

__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

template <typename T, int D, int NS, int SB, int PB, int AB>
__global__ void __launch_bounds__(768, 1)
tc_dqkv_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
               const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_do,
               const __grid_constant__ CUtensorMap map_bt, const __grid_constant__ CUtensorMap map_lse,
               const __grid_constant__ CUtensorMap map_delta, View5 dq, View5 dk, View5 dv,
               const uint8_t* __restrict__ rowfull, const uint32_t* __restrict__ maskbits_lin,
               int mask_words, const uint32_t* __restrict__ rowrange, Dims dm, FusedGrid grid,
               float* __restrict__ kv_scratch, unsigned int* status) {
  using Cfg = FusedCfg<D, NS, SB, PB, AB>;
  // Barriers of step g: S_FULL, ACC_DONE g % SB; DP_FULL, DP_FREE g & 1; P_READY g & 3; FULL, EMPTY
  // g % NS; DQ_PAIR by the parity of its pair.  A wait names a phase by its parity, so a waiter must be
  // neither a phase early nor two late.  Late: what would complete the phase after comes behind the
  // waiter's own arrive (step g + 4 of P_READY: the elementwise warps wait for the dQ of the pair
  // two before, which the dQ issuer commits after its waits for that pair's steps).  Early:
  // a role that waits for every step in turn cannot be.  An elementwise group sees every other step,
  // and where a barrier's successive steps are not all its own (SB, NS odd) the phase between has
  // completed because of what the group has waited for: S_FULL (SB = 3) by DP_FULL of the same step,
  // whose commit follows those of S up to this step; FULL by the S of its own step before,
  // issued after those of all earlier steps; DQ_PAIR by that of an earlier pair, all committed in order.
  constexpr int KV_FULL = 0, KV_EMPTY = 2, FULL = 4, EMPTY = FULL + NS, S_FULL = EMPTY + NS,
                DP_FULL = S_FULL + SB, DP_FREE = DP_FULL + 2, P_READY = DP_FREE + 2, ACC_DONE = P_READY + 4, DQ_PAIR = ACC_DONE + SB,
                ACC_FREE = DQ_PAIR + 2, TILE_DONE = ACC_FREE + AB, DQ_DONE = TILE_DONE + AB,
                DQ_FREE = DQ_DONE + 1, NBARS = DQ_FREE + Cfg::kMaxJTiles;
  // With two S^T buffers the next S^T is what a step waits for: it is issued behind the MMAs that
  // free its place (n = 1024, h = 4, d = 32: 2.83 ms; by the dP issuer behind their commit 2.93 ms).  With
  // three it is not urgent, and out of the way of the next step's accumulation (n = 512 372 -> 350 us).
  constexpr bool kBehind = SB == 2;
  static_assert(NBARS * 8 <= 512, "barrier area");
  static_assert(Cfg::kDqCol + Cfg::kMaxJTiles * Cfg::kAcc <= 512, "TMEM columns");

  extern __shared__ __align__(1024) uint8_t smem_raw[];   // (see opt_in_smem)
  const uint32_t base = smem_u32(smem_raw);
  uint8_t* gbase = smem_raw;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gbase + 512);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gbase + 516);

  const int n = dm.n;
  const int nkt = grid.nkt, njs = grid.njs, njt = grid.njt, nch = grid.nch, jsc = grid.jsc;
  constexpr uint32_t tiles_off = Cfg::kHeader;
  constexpr uint32_t stages_off = tiles_off + 4 * Cfg::kKVBytes;
  constexpr uint32_t pairs_off = stages_off + NS * Cfg::kStageBytes;
  auto bar = [&](int i) -> uint32_t { return base + 8u * i; };
  auto k_tile = [&](int kvb) -> uint32_t { return base + tiles_off + (2 * kvb) * Cfg::kKVBytes; };
  auto v_tile = [&](int kvb) -> uint32_t { return base + tiles_off + (2 * kvb + 1) * Cfg::kKVBytes; };
  auto stage_off = [&](int s) -> uint32_t { return stages_off + s * Cfg::kStageBytes; };
  auto q_tile = [&](int s) -> uint32_t { return base + stage_off(s); };
  auto do_tile = [&](int s) -> uint32_t { return base + stage_off(s) + Cfg::kQBytes; };
  auto bias_off = [&](int s) -> uint32_t { return stage_off(s) + 2 * Cfg::kQBytes; };
  auto lse_off = [&](int s) -> uint32_t { return Cfg::kVecOff + s * 2 * Cfg::kVecBytes; };
  auto delta_off = [&](int s) -> uint32_t { return lse_off(s) + Cfg::kVecBytes; };
  auto pair_off = [&](int pb) -> uint32_t { return pairs_off + pb * Cfg::kPairBytes; };
  // item -> (row, head, batch): consecutive CTAs work on neighbouring rows of one
  // (b, h) and sweep the same bias tiles at about the same time (L2 hits)
  struct Item {
    int i, h, b;
  };
  auto decode = [&](int w) -> Item {
    Item it;
    it.i = w % dm.n_rows;
    const int bh = w / dm.n_rows;
    it.h = bh % dm.heads;
    it.b = bh / dm.heads;
    return it;
  };
  // Key tiles [lo, hi) of the item's row that hold an open key, as lo | hi << 16: the roles
  // walk only those (dK, dV of the others are zero-filled, dQ gets nothing from them).
  // Fetched one item ahead.
  auto item_range = [&](int w) -> uint32_t {
    if (rowrange == nullptr || w >= grid.total) return (uint32_t)nkt << 16;
    const Item it = decode(w);
    return uniform(__ldg(rowrange + it.b * dm.n_rows + it.i));
  };

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&map_k);
    tma_prefetch_desc(&map_v);
    tma_prefetch_desc(&map_q);
    tma_prefetch_desc(&map_do);
    tma_prefetch_desc(&map_bt);
    tma_prefetch_desc(&map_lse);
    tma_prefetch_desc(&map_delta);
  }
  after_previous();

  if (*reinterpret_cast<volatile unsigned int*>(status) != 0u) return;

  // (what every lane of a warp shares goes through uniform(), so that the compiler keeps it, and the
  // descriptors made of it, in uniform registers, where the MMAs want them)
  const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;

  if (tid == 0) {
    for (int u = 0; u < 2; ++u) {
      mbar_init(bar(KV_FULL + u), 1);
      mbar_init(bar(KV_EMPTY + u), 1);
      mbar_init(bar(DP_FULL + u), 1);
      mbar_init(bar(DP_FREE + u), 8);
      mbar_init(bar(DQ_PAIR + u), 1);
    }
    for (int u = 0; u < SB; ++u) {
      mbar_init(bar(S_FULL + u), 1);
      mbar_init(bar(ACC_DONE + u), 1);
    }
    for (int u = 0; u < 4; ++u) mbar_init(bar(P_READY + u), 8);
    for (int s = 0; s < NS; ++s) {
      mbar_init(bar(FULL + s), 1);
      mbar_init(bar(EMPTY + s), 9);  // the dV / dK commit + the 8 elementwise warps of the step
    }
    for (int u = 0; u < AB; ++u) {
      mbar_init(bar(ACC_FREE + u), 4);
      mbar_init(bar(TILE_DONE + u), 1);
    }
    mbar_init(bar(DQ_DONE), 1);
    for (int u = 0; u < Cfg::kMaxJTiles; ++u) mbar_init(bar(DQ_FREE + u), 4);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == kTmaWarp + 1) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = uniform(*tmem_slot);

  if (warp >= kTmaWarp && warp < kOutWarp) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsIssue));
    if (warp == kTmaWarp) {
      // ------------------------------------------------------------ TMA producer
      // (Every lane of an issuing warp runs the loop, so that addresses, coordinates
      // and descriptors are warp-uniform values; one lane issues.)
      int g = 0, ktg = 0;  // running step and key-tile counters (barrier phases)
      bool ok = true;
      uint32_t rng_next = item_range(blockIdx.x);
      for (int w = blockIdx.x; w < grid.total && ok; w += gridDim.x) {
        const Item im = decode(w);
        const int kt_lo = rng_next & 0xffffu, kt_hi = rng_next >> 16;
        rng_next = item_range(w + gridDim.x);
        for (int c = 0; c < nch && ok; ++c) {
        const int js0 = c * jsc, js1 = min(njs, js0 + jsc);
        for (int kt = kt_lo; kt < kt_hi && ok; ++kt, ++ktg) {
          const int kvb = ktg & 1;
          if (ktg >= 2)
            ok = __all_sync(0xffffffffu,
                            mbar_wait(bar(KV_EMPTY + kvb), ((ktg >> 1) - 1) & 1, abort_flag));
          if (!ok) break;
          if (elect_one()) {
            mbar_arrive_expect_tx(bar(KV_FULL + kvb), 2 * Cfg::kKVBytes);
            tma_load_5d(k_tile(kvb), &map_k, bar(KV_FULL + kvb), 0, kt * kBKeys, im.i, im.h, im.b);
            tma_load_5d(v_tile(kvb), &map_v, bar(KV_FULL + kvb), 0, kt * kBKeys, im.i, im.h, im.b);
          }
          for (int js = js0; js < js1; ++js, ++g) {
            const int s = g % NS;
            if (g >= NS)
              ok = __all_sync(0xffffffffu,
                              mbar_wait(bar(EMPTY + s), ((g / NS) - 1) & 1, abort_flag));
            if (!ok) break;
            if (elect_one()) {
              mbar_arrive_expect_tx(bar(FULL + s),
                                    2 * Cfg::kQBytes + Cfg::kBiasBytes + 2 * Cfg::kVecBytes);
              tma_load_5d(q_tile(s), &map_q, bar(FULL + s), 0, js * kBJ, im.i, im.h, im.b);
              tma_load_5d(do_tile(s), &map_do, bar(FULL + s), 0, js * kBJ, im.i, im.h, im.b);
              tma_load_4d(base + bias_off(s), &map_bt, bar(FULL + s), js * kBJ, kt * kBKeys, im.h, im.b);
              tma_load_4d(base + lse_off(s), &map_lse, bar(FULL + s), js * kBJ, im.i, im.h, im.b);
              tma_load_4d(base + delta_off(s), &map_delta, bar(FULL + s), js * kBJ, im.i, im.h, im.b);
            }
            __syncwarp();
          }
        }
        }
      }
    } else if (warp == kTmaWarp + 1) {
      // ------------------------------------------------------------ S^T / dP^T issuer
      constexpr bool kBf16 = std::is_same<T, __nv_bfloat16>::value;
      constexpr uint32_t idesc_s = make_idesc(128, kBJ, kBf16, false, false);
      int g = 0, ktg = 0;
      bool ok = true;
      uint32_t rng_next = item_range(blockIdx.x);
      for (int w = blockIdx.x; w < grid.total && ok; w += gridDim.x) {
        const int kt_lo = rng_next & 0xffffu, kt_hi = rng_next >> 16;
        rng_next = item_range(w + gridDim.x);
        for (int c = 0; c < nch && ok; ++c) {
        const int js0 = c * jsc, js1 = min(njs, js0 + jsc);
        for (int kt = kt_lo; kt < kt_hi && ok; ++kt, ++ktg) {
          const int kvb = ktg & 1;
          for (int js = js0; js < js1; ++js, ++g) {
            const int s = g % NS, sb = g % SB;
            // S^T: its buffer held P^T, dS^T of step g - SB, which the dV / dK MMAs have read
            ok = (js > js0 || mbar_wait(bar(KV_FULL + kvb), (ktg >> 1) & 1, abort_flag)) &&
                 mbar_wait(bar(FULL + s), (g / NS) & 1, abort_flag) &&
                 (kBehind || g < SB || mbar_wait(bar(ACC_DONE + sb), (g / SB - 1) & 1, abort_flag));
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            const uint64_t ak = make_smem_desc(k_tile(kvb), 16, Cfg::kSbo, Cfg::kSwz);
            const uint64_t bq = make_smem_desc(q_tile(s), 16, Cfg::kSbo, Cfg::kSwz);
            const uint64_t av = make_smem_desc(v_tile(kvb), 16, Cfg::kSbo, Cfg::kSwz);
            const uint64_t bg = make_smem_desc(do_tile(s), 16, Cfg::kSbo, Cfg::kSwz);
            const uint32_t t_s = tmem_base + sb * 64, t_dp = tmem_base + Cfg::kDpCol + (g % PB) * 64;
            if (!kBehind && elect_one()) {
              // a K slice of 16 elements is 32 bytes further along the row: + 2 in the
              // descriptor's address field (16-byte units)
#pragma unroll
              for (int kk = 0; kk < D / 16; ++kk)
                umma_ss(t_s, ak + 2 * kk, bq + 2 * kk, idesc_s, kk > 0);
              umma_commit(bar(S_FULL + sb));
            }
            __syncwarp();
            const int gp = g - PB;   // dP^T: its buffer was last read at step g - PB
            if (gp >= 0) {
              ok = __all_sync(0xffffffffu, mbar_wait(bar(DP_FREE + (gp & 1)), (gp >> 1) & 1, abort_flag));
              if (!ok) break;
              tc_fence_after();
            }
            if (elect_one()) {
#pragma unroll
              for (int kk = 0; kk < D / 16; ++kk)
                umma_ss(t_dp, av + 2 * kk, bg + 2 * kk, idesc_s, kk > 0);
              umma_commit(bar(DP_FULL + (g & 1)));
            }
            __syncwarp();
          }
        }
        }
      }
    } else if (warp == kTmaWarp + 2) {
      // ------------------------------------------------------------ dV / dK issuer
      // kBehind: after the dV / dK MMAs of step g come the S^T MMAs of step g + SB, whose result
      // overwrites the P^T and dS^T those read, with no wait in between.  This counts on the tensor
      // core taking one thread's MMAs in the order of their issue; the PTX documentation says so
      // for MMAs of one accumulator and shape, and these differ in both.  What bears it are
      // results equal to the two-kernel path's bit for bit (tests/test_one_pass_steps_gpu.py);
      // with three S buffers ACC_DONE stands between, the documented way.
      constexpr bool kBf16 = std::is_same<T, __nv_bfloat16>::value;
      constexpr uint32_t idesc_s = make_idesc(128, kBJ, kBf16, false, false);
      constexpr uint32_t idesc_acc = make_idesc(128, D, kBf16, false, true);
      // 16 rows of an MN-major tile are this many 16-byte units further on
      constexpr uint32_t kStep16Rows = (16 * Cfg::kRowBytes) >> 4;
      bool ok = true;
      // the step whose S^T is next: item, its range of key tiles, chunk, key tile, query step
      struct {
        int w, lo, hi, c, kt, js, js1, ktg, g;
        uint32_t rng;
      } nx;
      nx.w = blockIdx.x;
      nx.rng = item_range(nx.w);
      nx.c = nx.ktg = nx.g = nx.js = 0;
      nx.js1 = min(njs, jsc);
      nx.lo = nx.kt = nx.rng & 0xffffu;
      nx.hi = nx.rng >> 16;
      nx.rng = item_range(nx.w + gridDim.x);
      auto issue_s = [&]() {
        if (nx.w >= grid.total) return;
        const int js0 = nx.c * jsc, s = nx.g % NS, kvb = nx.ktg & 1;
        ok = (nx.js > js0 || mbar_wait(bar(KV_FULL + kvb), (nx.ktg >> 1) & 1, abort_flag)) &&
             mbar_wait(bar(FULL + s), (nx.g / NS) & 1, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) return;
        tc_fence_after();
        const uint64_t ak = make_smem_desc(k_tile(kvb), 16, Cfg::kSbo, Cfg::kSwz);
        const uint64_t bq = make_smem_desc(q_tile(s), 16, Cfg::kSbo, Cfg::kSwz);
        const uint32_t t_s = tmem_base + (nx.g % SB) * 64;
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) umma_ss(t_s, ak + 2 * kk, bq + 2 * kk, idesc_s, kk > 0);
          umma_commit(bar(S_FULL + nx.g % SB));
        }
        __syncwarp();
        ++nx.g;
        ++nx.js;
        if (nx.js < nx.js1) return;
        ++nx.ktg;
        ++nx.kt;
        if (nx.kt == nx.hi) {
          nx.kt = nx.lo;
          ++nx.c;
          if (nx.c == nch) {
            nx.c = 0;
            nx.w += gridDim.x;
            nx.lo = nx.kt = nx.rng & 0xffffu;
            nx.hi = nx.rng >> 16;
            nx.rng = item_range(nx.w + gridDim.x);
          }
        }
        nx.js = nx.c * jsc;
        nx.js1 = min(njs, nx.js + jsc);
      };
      if constexpr (kBehind)
        for (int u = 0; u < SB && ok; ++u) issue_s();
      int g = 0, ktg = 0;
      uint32_t rng_next = item_range(blockIdx.x);
      for (int w = blockIdx.x; w < grid.total && ok; w += gridDim.x) {
        const int kt_lo = rng_next & 0xffffu, kt_hi = rng_next >> 16;
        rng_next = item_range(w + gridDim.x);
        for (int c = 0; c < nch && ok; ++c) {
        const int js0 = c * jsc, js1 = min(njs, js0 + jsc);
        for (int kt = kt_lo; kt < kt_hi && ok; ++kt, ++ktg) {
          const int ab = ktg % AB;
          for (int js = js0; js < js1 && ok; ++js, ++g) {
            const int s = g % NS;
            // the first accumulating MMAs of a key tile overwrite dK, dV: the output warps
            // must have read those of the key tile AB before
            ok = mbar_wait(bar(P_READY + (g & 3)), (g >> 2) & 1, abort_flag) &&
                 (js > js0 || ktg < AB || mbar_wait(bar(ACC_FREE + ab), (ktg / AB - 1) & 1, abort_flag));
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            const uint32_t acc = (js > js0) ? 1u : 0u;
            const uint64_t b_do = make_smem_desc(do_tile(s), Cfg::kSbo, Cfg::kSbo, Cfg::kSwz);
            const uint64_t b_q = make_smem_desc(q_tile(s), Cfg::kSbo, Cfg::kSbo, Cfg::kSwz);
            // (P^T and dS^T of 16 queries lie side by side, 8 columns each, where their S^T was)
            const uint32_t t_p = tmem_base + (g % SB) * 64, t_acc = tmem_base + ab * 2 * Cfg::kAcc;
            if (elect_one()) {
#pragma unroll
              for (int ks = 0; ks < kBJ / 16; ++ks) {  // dV += P^T dO, dK += dS^T Q, interleaved
                umma_ts(t_acc + Cfg::kDvCol, t_p + ks * 16, b_do + ks * kStep16Rows, idesc_acc,
                        (ks > 0) ? 1u : acc);
                umma_ts(t_acc + Cfg::kDkCol, t_p + ks * 16 + 8, b_q + ks * kStep16Rows, idesc_acc,
                        (ks > 0) ? 1u : acc);
              }
              if (!kBehind) umma_commit(bar(ACC_DONE + g % SB));
              umma_commit(bar(EMPTY + s));
              if (js == js1 - 1) umma_commit(bar(TILE_DONE + ab));
            }
            __syncwarp();
            if constexpr (kBehind) issue_s();
          }
        }
        }
      }
    } else {
      // ------------------------------------------------------------ dQ issuer
      constexpr bool kBf16 = std::is_same<T, __nv_bfloat16>::value;
      constexpr uint32_t idesc_dq = make_idesc(128, D, kBf16, true, true);
      constexpr uint32_t kStep16Rows = (16 * Cfg::kRowBytes) >> 4;
      int g = 0, ktg = 0, pgc = 0, chg = 0;  // chg: running chunk counter (DQ_FREE phases)
      bool ok = true;
      uint32_t rng_next = item_range(blockIdx.x);
      for (int w = blockIdx.x; w < grid.total && ok; w += gridDim.x) {
        const int kt_lo = rng_next & 0xffffu, kt_hi = rng_next >> 16;
        rng_next = item_range(w + gridDim.x);
        for (int c = 0; c < nch && ok; ++c, ++chg) {
        const int js0 = c * jsc, js1 = min(njs, js0 + jsc);
        for (int kt = kt_lo; kt < kt_hi && ok; ++kt, ++ktg) {
          const int kvb = ktg & 1;
          for (int js = js0; js < js1; ++js, ++g) {
            const bool with_dq = ((js - js0) & 1) || js == js1 - 1;
            const int pr = (js - js0) >> 1, pb = (pgc + pr) & 1;
            // the first dQ MMA of a 128-query tile in a chunk overwrites it: the output warps
            // must have read the previous chunk's
            ok = mbar_wait(bar(P_READY + (g & 3)), (g >> 2) & 1, abort_flag) &&
                 (!with_dq || kt > kt_lo || chg == 0 || mbar_wait(bar(DQ_FREE + pr), (chg - 1) & 1, abort_flag));
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            if (!with_dq) continue;
            tc_fence_after();
            // dS tile of the pair (rows = keys, 128-byte rows of 64 queries, two halves):
            // read as an MN-major A operand it is dS (queries x keys)
            const uint64_t a_ds = make_smem_desc(base + pair_off(pb), Cfg::kHalfBytes, 1024, kSwizzle128);
            const uint64_t b_k = make_smem_desc(k_tile(kvb), Cfg::kSbo, Cfg::kSbo, Cfg::kSwz);
            if (elect_one()) {
              // dQ of the 128-query tile js / 2: both halves of its dS tile are written
              // (an odd last step leaves the second half stale: those queries lie
              // beyond n and their dQ rows are never stored)
#pragma unroll
              for (int ks = 0; ks < kBKeys / 16; ++ks)
                umma_ss(tmem_base + Cfg::kDqCol + pr * Cfg::kAcc, a_ds + ks * ((16 * 128) >> 4),
                        b_k + ks * kStep16Rows, idesc_dq, (kt > kt_lo || ks > 0) ? 1u : 0u);
              umma_commit(bar(DQ_PAIR + pb));
              if (js == js1 - 1) {
                umma_commit(bar(KV_EMPTY + kvb));  // last read of this K, V
                if (kt == kt_hi - 1) umma_commit(bar(DQ_DONE));
              }
            }
            __syncwarp();
          }
          pgc += (js1 - js0 + 1) >> 1;
        }
        }
      }
    }
  } else if (warp >= kOutWarp) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsOut));
    // ------------------------------------------------------------ output warps
    // dK and dV of a key tile (thread = key), dQ of a chunk (thread = query of each tile).
    const int t = tid & 127;
    const uint32_t t_out = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
    constexpr int kCols = 16;   // columns of a piece
    auto row_of = [&](const View5& v, const Item& im, int j) -> T* {
      return reinterpret_cast<T*>(v.p) + im.b * v.sb + im.h * v.sh + (int64_t)im.i * v.si + (int64_t)j * v.sj;
    };
    auto store = [&](T* dst, const uint32_t* acc, float sc) {
#pragma unroll
      for (int e = 0; e < kCols; e += 8) {
        uint4 u;
        u.x = pack2<T>(__uint_as_float(acc[e + 0]) * sc, __uint_as_float(acc[e + 1]) * sc);
        u.y = pack2<T>(__uint_as_float(acc[e + 2]) * sc, __uint_as_float(acc[e + 3]) * sc);
        u.z = pack2<T>(__uint_as_float(acc[e + 4]) * sc, __uint_as_float(acc[e + 5]) * sc);
        u.w = pack2<T>(__uint_as_float(acc[e + 6]) * sc, __uint_as_float(acc[e + 7]) * sc);
        *reinterpret_cast<uint4*>(dst + e) = u;
      }
    };
    int ktg = 0, chg = 0;
    bool ok = true;
    uint32_t rng_next = item_range(blockIdx.x);
    for (int w = blockIdx.x; w < grid.total && ok; w += gridDim.x) {
      const Item im = decode(w);
      const int kt_lo = rng_next & 0xffffu, kt_hi = rng_next >> 16;
      rng_next = item_range(w + gridDim.x);
      // dK, dV of the key tiles nobody walks: zero
      for (int kt = 0; kt < nkt; ++kt) {
        const int key = kt * kBKeys + t;
        if ((kt < kt_lo || kt >= kt_hi) && key < n) {
          T* dst_k = row_of(dk, im, key);
          T* dst_v = row_of(dv, im, key);
#pragma unroll
          for (int e = 0; e < D; e += 8) {
            *reinterpret_cast<uint4*>(dst_k + e) = make_uint4(0u, 0u, 0u, 0u);
            *reinterpret_cast<uint4*>(dst_v + e) = make_uint4(0u, 0u, 0u, 0u);
          }
        }
      }
      for (int c = 0; c < nch && ok; ++c, ++chg) {
        for (int kt = kt_lo; kt < kt_hi && ok; ++kt, ++ktg) {
          const int key = kt * kBKeys + t;
          // A row walked in several query chunks: dK / dV of a key tile are sums over the
          // chunks.  The partial of the earlier chunks waits, as fp32, in this CTA's own
          // scratch (the same thread writes and reads a given element; it stays in L2).
          // (Four columns of neighbouring keys lie side by side.)
          float4* part = nullptr;
          if (Cfg::kChunks && nch > 1)
            part = reinterpret_cast<float4*>(kv_scratch) +
                   ((size_t)blockIdx.x * nkt + kt) * (kBKeys * 2 * D / 4) + t;
          const bool carry_in = Cfg::kChunks && c > 0, carry_out = Cfg::kChunks && c + 1 < nch;
          // a piece's partial is fetched one piece ahead (the first before the tile is done)
          float4 ahead[kCols / 4];
          auto fetch = [&](int piece) {
#pragma unroll
            for (int e = 0; e < kCols / 4; ++e) ahead[e] = __ldcg(part + (piece * (kCols / 4) + e) * kBKeys);
          };
          if (carry_in) fetch(0);
          const int ab = ktg % AB;
          ok = __all_sync(0xffffffffu, mbar_wait(bar(TILE_DONE + ab), (ktg / AB) & 1, abort_flag));
          if (!ok) break;
          tc_fence_after();
#pragma unroll
          for (int p = 0; p < 2 * D / kCols; ++p) {   // pieces of dK, then of dV
            uint32_t acc[kCols];
            const bool is_v = p * kCols >= D;
            const int e0 = p * kCols - (is_v ? D : 0);
            tmem_ld_cols<kCols>(t_out + ab * 2 * Cfg::kAcc + (is_v ? Cfg::kDvCol : Cfg::kDkCol) + e0, acc);
            tmem_wait_ld();
            if (p == 2 * D / kCols - 1) {
              tc_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive(bar(ACC_FREE + ab));  // a later key tile may overwrite dK, dV
            }
            if (carry_in) {
#pragma unroll
              for (int e = 0; e < kCols; e += 4) {
                const float4 pv = ahead[e >> 2];
                acc[e + 0] = __float_as_uint(__uint_as_float(acc[e + 0]) + pv.x);
                acc[e + 1] = __float_as_uint(__uint_as_float(acc[e + 1]) + pv.y);
                acc[e + 2] = __float_as_uint(__uint_as_float(acc[e + 2]) + pv.z);
                acc[e + 3] = __float_as_uint(__uint_as_float(acc[e + 3]) + pv.w);
              }
              if (p + 1 < 2 * D / kCols) fetch(p + 1);
            }
            if (carry_out) {
#pragma unroll
              for (int e = 0; e < kCols; e += 4)
                __stcg(part + (p * (kCols / 4) + (e >> 2)) * kBKeys,
                       make_float4(__uint_as_float(acc[e + 0]), __uint_as_float(acc[e + 1]),
                                   __uint_as_float(acc[e + 2]), __uint_as_float(acc[e + 3])));
            } else if (key < n) {
              store(row_of(is_v ? dv : dk, im, key) + e0, acc, is_v ? 1.f : dm.scale);
            }
          }
        }
        if (!ok) break;
        ok = __all_sync(0xffffffffu, mbar_wait(bar(DQ_DONE), chg & 1, abort_flag));
        if (!ok) break;
        tc_fence_after();
        // (every tile's barrier once per chunk, also those a short last chunk does not have)
        const int jt0 = c * (jsc >> 1);
        for (int jl = 0; jl < Cfg::kMaxJTiles; ++jl) {
          const int j = (jt0 + jl) * 128 + t;
          if (jl < (jsc >> 1) && jt0 + jl < njt) {
#pragma unroll
            for (int e0 = 0; e0 < D; e0 += kCols) {
              uint32_t acc[kCols];
              tmem_ld_cols<kCols>(t_out + Cfg::kDqCol + jl * Cfg::kAcc + e0, acc);
              tmem_wait_ld();
              if (e0 + kCols == D) {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar(DQ_FREE + jl));  // the next chunk may overwrite the tile
              }
              if (j < n) store(row_of(dq, im, j) + e0, acc, dm.scale);
            }
          } else if (lane == 0) {
            mbar_arrive(bar(DQ_FREE + jl));
          }
        }
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsMath));
    {
      // ------------------------------------------------------------ elementwise warps
      // Thread = one key (TMEM lane).  Two groups of eight warps take the steps in turn, so that
      // one group's waits, loads and stores lie under the other's arithmetic; in a group, warps w
      // and w + 4 share the lanes and take 32 of the step's 64 queries each.
      const int group = warp >> 3, half = (warp >> 2) & 1, wq = warp & 3, t = tid & 127;
      const uint32_t lane_base = (uint32_t)(wq * 32) << 16;
      const uint32_t tS0 = tmem_base + lane_base + half * 32;
      const uint32_t tDP0 = tmem_base + lane_base + Cfg::kDpCol + half * 32;
      const float c1 = in_register(dm.scale * kLog2e), log2e = in_register(kLog2e), minus = in_register(-1.f);
      const float p_full = 1.f / (float)n;

      int g = 0, pgc = 0;
      bool ok = true;
      // Key mask of the row in key order (bit set = key dropped or beyond n; on a fully
      // masked row only the keys beyond n): word kt * 4 + wq covers this warp's 32 keys of key
      // tile kt.  The next key tile's word and the next row's range and flag are fetched one
      // key tile or row ahead: a global load costs as much as half a step.
      auto mask_row = [&](int w) -> int64_t {
        const Item im = decode(w);
        return (int64_t)im.b * dm.n_rows + im.i;
      };
      uint32_t rng_next = item_range(blockIdx.x), mword_next = 0u;
      uint8_t full_next = 0;
      int64_t row_next = 0;
      if ((int)blockIdx.x < grid.total) {
        row_next = mask_row(blockIdx.x);
        full_next = __ldg(rowfull + row_next);
        mword_next = __ldg(maskbits_lin + row_next * mask_words + (rng_next & 0xffffu) * 4 + wq);
      }
      for (int w = blockIdx.x; w < grid.total && ok; w += gridDim.x) {
        const int kt_lo = rng_next & 0xffffu, kt_hi = rng_next >> 16;
        const bool row_full = full_next != 0;
        const uint32_t* mrow = maskbits_lin + row_next * mask_words;
        const bool more = w + (int)gridDim.x < grid.total;
        if (more) {
          rng_next = item_range(w + gridDim.x);
          row_next = mask_row(w + gridDim.x);
          full_next = __ldg(rowfull + row_next);
        }
        for (int c = 0; c < nch && ok; ++c) {
        const int js0 = c * jsc, js1 = min(njs, js0 + jsc);

        for (int kt = kt_lo; kt < kt_hi && ok; ++kt) {
          const uint32_t mword = mword_next;
          if (kt + 1 < kt_hi)
            mword_next = __ldg(mrow + (kt + 1) * 4 + wq);
          else if (c + 1 < nch)
            mword_next = __ldg(mrow + kt_lo * 4 + wq);
          else if (more)
            mword_next = __ldg(maskbits_lin + row_next * mask_words + (rng_next & 0xffffu) * 4 + wq);
          const bool dropped = ((mword >> lane) & 1u) != 0u;
          // The key weight pattern is fixed for the whole query loop of a key tile, so
          // the loop is instantiated per pattern of this warp: 0 = every key kept (no
          // selects), 1 = mixed, 2 = every key dropped (no exponentials), 3 = fully
          // masked row.
          const int mode = row_full ? 3
                           : __all_sync(0xffffffffu, !dropped) ? 0
                           : __all_sync(0xffffffffu, dropped)  ? 2
                                                               : 1;
          const int g0 = g;
          auto query_loop = [&](auto mode_tag) {
            constexpr int kMode = decltype(mode_tag)::value;
            for (int js = js0 + ((g0 ^ group) & 1); js < js1; js += 2) {
              const int gg = g0 + (js - js0);
              const int s = gg % NS;
              // S^T and dP^T of this step and its bias / lse / delta stage; the dS tile that the
              // step's pair writes was last read by the dQ MMAs two pairs ago
              const int pair = pgc + ((js - js0) >> 1);
              ok = mbar_wait(bar(FULL + s), (gg / NS) & 1, abort_flag) &&
                   mbar_wait(bar(DP_FULL + group), (gg >> 1) & 1, abort_flag) &&
                   (pair < 2 || mbar_wait(bar(DQ_PAIR + (pair & 1)), ((pair >> 1) - 1) & 1, abort_flag)) &&
                   mbar_wait(bar(S_FULL + gg % SB), (gg / SB) & 1, abort_flag);
              ok = __all_sync(0xffffffffu, ok);
              if (!ok) break;
              tc_fence_after();
              const uint32_t tS = tS0 + (gg % SB) * 64, tDP = tDP0 + (gg % PB) * 64;
              // (dP^T leaves TMEM at once, for the next step's; S^T in two halves)
              float x[16], g_[32];
              tmem_ld32(tDP, reinterpret_cast<uint32_t*>(g_));
              tmem_ld16(tS, reinterpret_cast<uint32_t*>(x));
              tmem_wait_ld();
              tc_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive(bar(DP_FREE + group));

              // One fused pass per 8 queries: bias^T / lse / delta loads, unpack, FMAs, the
              // exponential, dS and both 16-bit packs, which overwrite this thread's own S^T;
              // the dS chunk also goes to the shared-memory tile (row = key, 128-byte rows,
              // 16-byte chunks swizzled by the row as the 128B TMA / UMMA swizzle does).
              const uint8_t* brow = gbase + bias_off(s) + t * 128;
              const float4* lse4 = reinterpret_cast<const float4*>(gbase + lse_off(s)) + half * 8;
              const float4* del4 = reinterpret_cast<const float4*>(gbase + delta_off(s)) + half * 8;
              uint8_t* srow = gbase + pair_off(pair & 1) +
                              ((js - js0) & 1) * Cfg::kHalfBytes + t * 128;
#pragma unroll
              for (int hq = 0; hq < 2; ++hq) {
                if (hq == 1) {
                  tmem_ld16(tS + 16, reinterpret_cast<uint32_t*>(x));
                  tmem_wait_ld();
                }
                uint32_t pp[8], pd[8];
#pragma unroll
                for (int q8 = 0; q8 < 2; ++q8) {
                  const int at = hq * 2 + q8;   // this warp's 8 queries
                  const int chunk = (((half * 4 + at) ^ (t & 7)) << 4);
                  const float4 da = del4[at * 2];
                  const float4 db = del4[at * 2 + 1];
                  const float dl[8] = {da.x, da.y, da.z, da.w, db.x, db.y, db.z, db.w};
                  float p[8];
                  if (kMode == 2) {
#pragma unroll
                    for (int e = 0; e < 8; ++e) p[e] = 0.f;
                  } else if (kMode == 3) {
#pragma unroll
                    for (int e = 0; e < 8; ++e) p[e] = p_full;
                  } else {
                    const uint4 u = *reinterpret_cast<const uint4*>(brow + chunk);
                    const float4 la = lse4[at * 2];
                    const float4 lb = lse4[at * 2 + 1];
                    const float nl[8] = {la.x, la.y, la.z, la.w, lb.x, lb.y, lb.z, lb.w};
                    float bv[8];
                    unpack2<T>(u.x, bv[0], bv[1]);
                    unpack2<T>(u.y, bv[2], bv[3]);
                    unpack2<T>(u.z, bv[4], bv[5]);
                    unpack2<T>(u.w, bv[6], bv[7]);
                    // packed fp32 pairs: two scores per FMA instruction
#pragma unroll
                    for (int e = 0; e < 8; e += 2) {
                      float t0, t1, a0, a1;
                      ffma2(t0, t1, bv[e], bv[e + 1], log2e, log2e, nl[e], nl[e + 1]);
                      ffma2(a0, a1, x[q8 * 8 + e], x[q8 * 8 + e + 1], c1, c1, t0, t1);
                      p[e] = ex2(a0);
                      p[e + 1] = ex2(a1);
                    }
                  }
#pragma unroll
                  for (int e = 0; e < 8; e += 2) {
                    const int col = q8 * 8 + e;
                    float s0, s1, d0, d1;
                    ffma2(s0, s1, dl[e], dl[e + 1], minus, minus, g_[hq * 16 + col], g_[hq * 16 + col + 1]);   // dP - delta
                    fmul2(d0, d1, p[e], p[e + 1], s0, s1);
                    uint32_t wp = pack2<T>(p[e], p[e + 1]);
                    uint32_t wd = pack2<T>(d0, d1);
                    if (kMode == 1 || kMode == 3) {  // dropped keys weigh exactly zero
                      wp = dropped ? 0u : wp;
                      wd = dropped ? 0u : wd;
                    }
                    pp[col >> 1] = wp;
                    pd[col >> 1] = wd;
                  }
                  *reinterpret_cast<uint4*>(srow + chunk) =
                      make_uint4(pd[q8 * 4 + 0], pd[q8 * 4 + 1], pd[q8 * 4 + 2], pd[q8 * 4 + 3]);
                }
                tmem_st8(tS + hq * 16, pp);
                tmem_st8(tS + hq * 16 + 8, pd);
              }
              tmem_wait_st();
              tc_fence_before();
              fence_proxy_async_smem();  // the dS rows in shared memory are read by an MMA
              __syncwarp();
              if (lane == 0) {
                mbar_arrive(bar(P_READY + (gg & 3)));
                mbar_arrive(bar(EMPTY + s));  // bias^T, lse, delta consumed by this warp
              }
            }
          };
          switch (mode) {
            case 0: query_loop(std::integral_constant<int, 0>{}); break;
            case 1: query_loop(std::integral_constant<int, 1>{}); break;
            case 2: query_loop(std::integral_constant<int, 2>{}); break;
            default: query_loop(std::integral_constant<int, 3>{}); break;
          }
          if (!ok) break;
          g = g0 + (js1 - js0);
          pgc += (js1 - js0 + 1) >> 1;

        }
        }
      }
    }
  }

  // ---------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    const long long t0 = clock64();
    while (clock64() - t0 < 4000000LL) {
    }
    if (tid == 0) set_status(status, kStatusTimeoutBwdFused);
    __syncthreads();
  }
  if (warp == kTmaWarp + 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

template <typename T, int D, int NS, int SB, int PB, int AB>
cudaError_t launch_fused(const BwdArgs& a, cudaStream_t stream) {
  using Cfg = FusedCfg<D, NS, SB, PB, AB>;
  static_assert(Cfg::kSmemBytes <= kSmemLimit, "shared memory");
  const Dims& dm = a.dm;
  const bool bf16 = std::is_same<T, __nv_bfloat16>::value;
  const uint64_t eb = 2;
  CUtensorMap mk, mv, mq, mdo, mbt, mlse, mdelta;
  const uint64_t dims5[5] = {(uint64_t)D, (uint64_t)dm.n, (uint64_t)dm.n_rows, (uint64_t)dm.heads,
                             (uint64_t)dm.batch};
  const uint32_t box_kv[5] = {(uint32_t)D, 128, 1, 1, 1};
  const uint32_t box_q[5] = {(uint32_t)D, (uint32_t)kBJ, 1, 1, 1};
  const CUtensorMapSwizzle swz = (CUtensorMapSwizzle)RowSwizzle<D>::kTma;
  auto map5 = [&](CUtensorMap* m, const View5& v, const uint32_t* box) {
    const uint64_t st[4] = {(uint64_t)v.sj * eb, (uint64_t)v.si * eb, (uint64_t)v.sh * eb,
                            (uint64_t)v.sb * eb};
    return make_tensor_map(m, bf16, 5, v.p, dims5, st, box, swz);
  };
  if (!map5(&mk, a.k, box_kv) || !map5(&mv, a.v, box_kv) || !map5(&mq, a.q, box_q) ||
      !map5(&mdo, a.d_o, box_q))
    return cudaErrorInvalidValue;
  {  // transposed bias copy: (b, h, k, j) with row pitch n_pad
    const uint64_t n = dm.n, np = dm.n_pad;
    const uint64_t dims4[4] = {n, n, (uint64_t)dm.heads, (uint64_t)dm.batch};
    const uint64_t st[3] = {np * eb, n * np * eb, n * np * dm.heads * eb};
    const uint32_t box4[4] = {(uint32_t)kBJ, 128, 1, 1};
    if (!make_tensor_map(&mbt, bf16, 4, a.bias_t, dims4, st, box4, CU_TENSOR_MAP_SWIZZLE_128B))
      return cudaErrorInvalidValue;
  }
  {  // -lse * log2(e) and delta: (b, h, rows, n_pad) fp32, made by the prepare step
    const uint64_t n = dm.n, np = dm.n_pad, rows = dm.n_rows;
    const uint64_t dims4[4] = {n, rows, (uint64_t)dm.heads, (uint64_t)dm.batch};
    const uint64_t st[3] = {np * 4, np * rows * 4, np * rows * dm.heads * 4};
    const uint32_t box4[4] = {(uint32_t)kBJ, 1, 1, 1};
    if (!make_tensor_map_f32(&mlse, 4, a.neg_lse2, dims4, st, box4) ||
        !make_tensor_map_f32(&mdelta, 4, a.delta, dims4, st, box4))
      return cudaErrorInvalidValue;
  }
  const int smem = Cfg::kSmemBytes;
  constexpr auto kern = tc_dqkv_kernel<T, D, NS, SB, PB, AB>;
  cudaError_t e = opt_in_smem<kern, true>(smem);
  if (e != cudaSuccess) return e;
  FusedGrid grid;
  grid.total = dm.batch * dm.heads * dm.n_rows;
  grid.nkt = (dm.n + kBKeys - 1) / kBKeys;
  grid.njs = (dm.n + kBJ - 1) / kBJ;
  grid.njt = (dm.n + 127) / 128;
  grid.nch = tc_bwd_fused_chunks(dm.n, D);
  grid.jsc = 2 * ((grid.njt + grid.nch - 1) / grid.nch);
  if (grid.nch > 1 && !a.kv_scratch) return cudaErrorInvalidValue;
  int sms = sm_count();
  if (sms > kFusedMaxCtas) sms = kFusedMaxCtas;  // the dK / dV scratch is sized for this many CTAs
  int ctas = grid.total < sms ? grid.total : sms;
  if (a.reserve_sms > 0) {
    // A collective runs beside this kernel: leave it SMs.  Every CTA walks its items one
    // after the other, so the kernel lasts ceil(items / CTAs) items: keep at least
    // `reserve_sms` SMs free, then drop every further CTA that does not shorten that.
    // (Measured on 4 GPUs, n = 1024: with 8 SMs free the kernel takes 8 rounds instead of 7,
    // +0.11 ms, and the all-reduce stays hidden; with 1 SM free it keeps 7 rounds but the
    // all-reduce crawls and 0.20 ms of it show after the kernel.)
    const int keep = sms - a.reserve_sms > 0 ? sms - a.reserve_sms : 1;
    const int waves = (grid.total + keep - 1) / keep;
    ctas = (grid.total + waves - 1) / waves;
  }
  return launch_early(kern, ctas, Cfg::kThreads, smem, stream, mk, mv, mq, mdo, mbt, mlse, mdelta, a.dq, a.dk, a.dv,
                                              a.rowfull, a.maskbits_lin, a.mask_words, a.rowrange, dm,
                                              grid, a.kv_scratch, a.status);
}

// The number of chunks follows from the fewest buffers; then the most buffers that the dQ of a chunk
// leaves room for are taken: a third S (d <= 32), a second dP, and, for rows walked at once, a second
// pair of dK, dV.
template <typename T, int D>
cudaError_t launch_d(const BwdArgs& a, cudaStream_t s) {
  constexpr int NS = kFusedStages<D>, SB = D == 64 ? 2 : 3;
  const int njt = (a.dm.n + 127) / 128, nch = tc_bwd_fused_chunks(a.dm.n, D), per = (njt + nch - 1) / nch;
  if constexpr (FusedCfg<D, NS, SB, 2, 2>::kMaxJTiles > 0) {
    if (nch == 1 && per <= FusedCfg<D, NS, SB, 2, 2>::kMaxJTiles) return launch_fused<T, D, NS, SB, 2, 2>(a, s);
  }
  if (per <= FusedCfg<D, NS, SB, 2, 1>::kMaxJTiles) return launch_fused<T, D, NS, SB, 2, 1>(a, s);
  if constexpr (SB == 3) {
    if (per <= FusedCfg<D, NS, SB, 1, 1>::kMaxJTiles) return launch_fused<T, D, NS, SB, 1, 1>(a, s);
  }
  return launch_fused<T, D, NS, 2, 1, 1>(a, s);
}
template <typename T>
cudaError_t launch_for(const BwdArgs& a, cudaStream_t s) {
  switch (a.dm.d) {
    case 16: return launch_d<T, 16>(a, s);
    case 32: return launch_d<T, 32>(a, s);
    default: return launch_d<T, 64>(a, s);
  }
}

}  // namespace

bool tc_bwd_fused_supported(const BwdArgs& a) {
  const int d = a.dm.d;
  if (d != 16 && d != 32 && d != 64) return false;
  if (!a.bias_t || !a.neg_lse2 || !a.maskbits_lin) return false;
  return tc_bwd_fused_chunks(a.dm.n, d) == 1 || a.kv_scratch != nullptr;
}

int tc_bwd_fused_chunks(int n, int d) {
  const int njt = (n + 127) / 128;
  const int max_tiles = (d == 16)   ? FusedCfg<16, kFusedStages<16>, 2, 1, 1>::kMaxJTiles
                        : (d == 32) ? FusedCfg<32, kFusedStages<32>, 2, 1, 1>::kMaxJTiles
                                    : FusedCfg<64, kFusedStages<64>, 2, 1, 1>::kMaxJTiles;
  return (njt + max_tiles - 1) / max_tiles;
}

size_t tc_bwd_fused_scratch_bytes(int n, int d) {
  if (tc_bwd_fused_chunks(n, d) <= 1) return 0;
  const size_t nkt = (n + kBKeys - 1) / kBKeys;
  return (size_t)kFusedMaxCtas * nkt * kBKeys * 2 * d * sizeof(float);
}

cudaError_t tc_bwd_dqkv_fused(const BwdArgs& a, cudaStream_t s) {
  const bool bf16 = a.dtype == TRIFAST_BF16;
  if (!tc_bwd_fused_supported(a)) return cudaErrorInvalidValue;
  return bf16 ? launch_for<__nv_bfloat16>(a, s) : launch_for<__half>(a, s);
}

}  // namespace trifast
