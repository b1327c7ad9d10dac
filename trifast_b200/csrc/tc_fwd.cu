// Forward triangle attention on the 5th-generation tensor cores (bf16 / fp16).
//
// Work item = one 128-query tile (h, j-tile) of R = 4 consecutive pair rows i
// ("slots"), walked over the keys in steps of 64.  The slots share every bias
// tile, the dominant shared-memory stream, and cover each other's waits: a slot's
// step is a chain (S -> weights -> O += P V -> the next S), and four of them on an SM are what
// keeps the exponential unit fed.  CTAs are persistent: one per SM, each looping over work
// items, so that the loads and the first MMA of the next item overlap the tail of the current
// one.
//
//   warps 0 .. 15   : softmax warpgroups, one per slot; thread t owns query row t:
//                     S (TMEM) -> registers, + bias (shared memory), mask, online
//                     softmax in fp32, P -> TMEM as 16-bit pairs over S, O rescale when
//                     the row maximum moves, final O / l and lse
//   warp 16         : TMA producer: Q per item, then K, V (per slot) and the bias tile per
//                     key step through an NS-deep ring; it also finds the items (those whose rows
//                     all have no open key are left out) and hands them to the other roles
//   warps 17, 18    : MMA issuers, two slots each: O += P V (A = P from TMEM, B = V as
//                     an MN-major tile), then the slot's next S = Q K^T (SS, both operands
//                     K-major), whose result overwrites that P with no wait in between, and a
//                     step's S is complete only when the O += P V before it is.  This counts on
//                     the tensor core taking one thread's MMAs in the order of their issue; the
//                     PTX documentation says so for MMAs of one accumulator and shape, and these
//                     differ in both.  What bears it are results that repeat bit for bit and
//                     agree with float64 (tests/test_forward_steps_gpu.py)
//   warp 19         : idle; it completes the warpgroup whose registers are handed over
//
// What bounds it: a slot's step takes about 3400 cycles, two thirds of them in its own arithmetic
// beside the other slots', the rest on the way to the MMAs and back (n = 1024, d = 32, 148 rows: 7.4
// instructions a score, issue slots 58 %, exponential unit 64 %).  Time at h = 4 by the C ABI, back to back,
// before (two slots of eight warps, steps of 128 keys, P beside S) and after: d = 32 bf16 n = 64 10.3 -> 5.7 us, n = 512
// (15 % padding) 271 -> 207 us, n = 1024 1.94 -> 1.55 ms, n = 2048 (10 % padding) 14.1 -> 10.5 ms; d = 64 fp16
// n = 1024 2.33 -> 2.03 ms.
// Measured and left (n = 1024, d = 32): P beside S, the next S issued as soon as this one is read, 1.67 ms,
// all slots then keep in step; the same with two pairs of slots taking turns in the exponentials
// 1.62 ms.
//
// TMEM columns per slot r (base r * 128): S [0,64) fp32, P over it [0,32) packed 16-bit pairs,
// O [64, 64 + D) fp32.
//
// Semantics follow the PyTorch path of the reference (src/trifast/equiv.py:42-69):
// masked keys weigh exactly zero; rows whose keys are all masked get the mean of all n
// values and lse = finfo(dtype).min (written by the prepare kernel where it runs).  The
// kernel stands in for `_fwd` of the reference (src/trifast/triton.py:14-132); unlike it, the
// scale d^-0.5 is applied to the fp32 accumulator, not to Q in 16 bits.

#include <math.h>

#include <mutex>

#include "kernels.h"
#include "tc_common.cuh"

namespace trifast {
namespace {
using namespace tc;

// Register hand-over (setmaxnreg): 640 threads launch with 96 registers each; what the
// softmax warpgroups gain must not exceed what the issue warpgroup releases, or the request
// blocks forever.
constexpr int kRegsLaunch = 96, kRegsIssue = 32, kRegsMath = 112;
static_assert(512 * kRegsMath + 128 * kRegsIssue <= 640 * kRegsLaunch, "setmaxnreg pool");

constexpr int kR = kFwdRows;      // slots: pair rows of an item
constexpr int kBJ = 128, kBK = 64;
constexpr int kTmaWarp = 16;
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;
constexpr float kMaxInit = -1e30f;
// A step moves the running maximum only when it exceeds it by more than the lazy threshold
// (natural-log units).  0 = always track the exact maximum: the largest weight of a
// row is then exactly 1 before rounding to 16 bits, which keeps the error of peaked
// rows lowest; a positive value (FlashAttention-style lazy rescale) trades that for
// fewer rescales of O, 64 columns at d = 64.  There (n = 300, fp16, relative 2-norm error of o against
// float64; forward of n = 512, h = 8, one session): 0 2.50e-4, 547 us; 2 2.74e-4, 537 us; 5.5 2.83e-4, 523 us, and
// 2.75e-4 before the steps were 64 keys long.  1.5 against 0, in turn: n = 512, h = 8, fp16 2.73e-4, 527 us
// and 2.54e-4, 531 us (bf16 2.18e-3, 544 and 2.03e-3, 551); n = 1024, h = 4, 5 % random mask 2.76e-4, 2.09 to
// 2.14 ms and 2.58e-4, 2.15 to 2.17 ms.
template <int D> constexpr float lazy_tau() { return D >= 64 ? 1.5f : 0.f; }
constexpr int kSmemLimit = 232448;  // 227 KiB opt-in limit per CTA
constexpr int kHeaderBytes = 1024;

template <int D> struct FwdCfg {
  static constexpr int NS = tc_forward_stages(D);           // stages of the ring
  static constexpr int kRowBytes = D * 2;
  static constexpr int kQBytes = kBJ * kRowBytes;           // Q tile of a slot
  static constexpr int kKVBytes = kBK * kRowBytes;          // K or V tile of a slot
  static constexpr int kBiasBytes = kBJ * kBK * 2;
  static constexpr int kStageBytes = 2 * kR * kKVBytes + kBiasBytes;
  static constexpr int kSmemBytes = kHeaderBytes + kR * kQBytes + NS * kStageBytes;
  static constexpr int kThreads = 640;
  static constexpr uint64_t kSwz = RowSwizzle<D>::kDesc;
  static constexpr int kSbo = 8 * kRowBytes;                // pitch of 8-row groups
  static_assert(kSmemBytes <= kSmemLimit, "shared memory");
};

// Work items in launch order: j-tile fastest, then row group, then (b, h): the CTAs
// running at one time share bias strips and K/V rows in L2.
// The first `full` row groups' items have kR rows; those after it are halves of two rows each, so
// that a last round that would fill at most half of the CTAs fills them all and ends earlier
// (a half item takes about 0.6 of a whole one).
struct ItemGrid {
  int njt, nrg, full, total;
};

// The key mask: the prepare step's packed words, or the caller's bytes; kAlone: bytes, and no prepare
// step has run (at most 128 keys: the mask of a row is one word a lane, and the ranges are all keys).
enum Masks { kWords, kBytes, kAlone };
template <typename T, int D, Masks M>
__global__ void __launch_bounds__(640, 1)
tc_fwd_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
              const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_b,
              View5 o, float* __restrict__ lse, MaskView mask,
              const uint32_t* __restrict__ ws_maskbits, int ws_mask_words,
              const uint32_t* __restrict__ ws_rowrange, Dims dm, ItemGrid items,
              unsigned int* status) {
  using Cfg = FwdCfg<D>;
  constexpr int NS = Cfg::NS;
  constexpr int ITEM = 0, Q_FULL = 4, Q_EMPTY = 5, FULL = 6, EMPTY = FULL + NS, S_FULL = EMPTY + NS,
                P_READY = S_FULL + kR, O_DONE = P_READY + kR, O_FREE = O_DONE + kR, NBARS = O_FREE + kR;
  static_assert(NBARS * 8 <= 512, "barrier area");

  extern __shared__ __align__(1024) uint8_t smem_raw[];   // (see opt_in_smem)
  const uint32_t base = smem_u32(smem_raw);
  uint8_t* gbase = smem_raw;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gbase + 512);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gbase + 516);

  const int n = dm.n;
  constexpr uint32_t tiles_off = kHeaderBytes;
  constexpr uint32_t stages_off = tiles_off + kR * Cfg::kQBytes;
  auto bar = [&](int i) -> uint32_t { return base + 8u * i; };
  auto q_tile = [&](int r) -> uint32_t { return base + tiles_off + r * Cfg::kQBytes; };
  auto k_tile = [&](int s, int r) -> uint32_t { return base + stages_off + s * Cfg::kStageBytes + r * Cfg::kKVBytes; };
  auto v_tile = [&](int s, int r) -> uint32_t { return k_tile(s, kR + r); };
  auto bias_off = [&](int s) -> uint32_t { return stages_off + s * Cfg::kStageBytes + 2 * kR * Cfg::kKVBytes; };
  // item -> (j tile, first row, head, batch); a slot beyond the last row re-does the
  // last row (its loads stay in range, its results are not stored)
  struct Item {
    int jt, i0, h, b;
  };
  auto decode = [&](int w) -> Item {
    Item it;
    const int half = w - items.full;
    if (half >= 0) w = items.full + (half >> 1);
    it.jt = w % items.njt;
    const int rest = w / items.njt;
    it.i0 = (rest % items.nrg) * kR + (half >= 0 ? 2 * (half & 1) : 0);
    const int bh = rest / items.nrg;
    it.h = bh % dm.heads;
    it.b = bh / dm.heads;
    return it;
  };
  auto slot_row = [&](const Item& it, int r) -> int { return min(it.i0 + r, dm.n_rows - 1); };
  // The producer hands an item to the other roles through a ring of four records and barriers: number
  // (-1 at the end), its key steps [lo, hi) as lo | hi << 16 (twice the 15 bits of a row's key tiles),
  // first query, first row, head, batch.  It is never more than two items ahead of a reader: an
  // item's Q is loaded behind Q_EMPTY of the one before, whose MMAs are issued behind P_READY of
  // the one before that.
  volatile int* records = reinterpret_cast<volatile int*>(gbase + 544);   // [4][8]

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&map_q);
    tma_prefetch_desc(&map_k);
    tma_prefetch_desc(&map_v);
    tma_prefetch_desc(&map_b);
  }
  after_previous();

  // A wait that gave up in an earlier CTA or launch leaves the status word set:
  // stop doing work until the host has read and cleared it.
  if (*reinterpret_cast<volatile unsigned int*>(status) != 0u) {
    if (threadIdx.x == 0) repeat_status(status);   // (no prepare kernel runs before small problems)
    return;
  }

  // (what every lane of a warp shares goes through uniform(), so that the compiler keeps it, and the
  // descriptors made of it, in uniform registers, where the MMAs want them)
  const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;

  if (tid == 0) {
    for (int u = 0; u < 4; ++u) mbar_init(bar(ITEM + u), 1);
    mbar_init(bar(Q_FULL), 1);
    mbar_init(bar(Q_EMPTY), kR);
    for (int s = 0; s < NS; ++s) {
      mbar_init(bar(FULL + s), 1);
      mbar_init(bar(EMPTY + s), kR * 5);  // per slot: 1 MMA commit + 4 softmax warps
    }
    for (int r = 0; r < kR; ++r) {
      mbar_init(bar(S_FULL + r), 1);
      mbar_init(bar(P_READY + r), 4);
      mbar_init(bar(O_DONE + r), 1);
      mbar_init(bar(O_FREE + r), 4);
    }
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

  if (warp >= kTmaWarp) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsIssue));
  // (The whole warp runs the loops of the producer and the issuers; elect_one() issues, which
  // tells the compiler that one thread does: under a lane test it wraps every MMA and TMA
  // load in code for several, 130 cycles an MMA instead of 50.)
  if (warp == kTmaWarp) {
    // ------------------------------------------------------------ TMA producer
    // key steps an item walks: the union of the live ranges of its rows (in 128-key tiles; a row
    // without an open key has none), fetched one item ahead; none for the second half of a group
    // of one or two rows
    auto item_range = [&](int w) -> uint32_t {
      const uint32_t steps = (uint32_t)(n + kBK - 1) / kBK;
      if (w >= items.total) return 0u;
      const Item it = decode(w);
      if (it.i0 >= dm.n_rows) return 0u;
      if (M == kAlone) return steps << 16;
      uint32_t lo = 0xffffu, hi = 0u;
      for (int r = 0; r < (w < items.full ? kR : 2); ++r) {
        const uint32_t u = __ldg(ws_rowrange + it.b * dm.n_rows + slot_row(it, r));
        lo = min(lo, u & 0xffffu);
        hi = max(hi, (u >> 16) & 0x7fffu);
      }
      return uniform(lo >= hi ? 0u : 2 * lo | min(2 * hi, steps) << 16);
    };
    int g = 0, it = 0;  // running key-step and item counters (barrier phases)
    bool ok = true;
    uint32_t rng_next = item_range(blockIdx.x);
    for (int w = blockIdx.x; w < items.total && ok; w += gridDim.x) {
      const uint32_t rng = rng_next;
      const int lo = rng & 0xffffu, hi = rng >> 16;
      rng_next = item_range(w + gridDim.x);
      if (lo >= hi) continue;
      const Item im = decode(w);
      const int slots = w < items.full ? kR : 2;
      if (it > 0) ok = __all_sync(0xffffffffu, mbar_wait(bar(Q_EMPTY), (it - 1) & 1, abort_flag));
      if (!ok) break;
      if (elect_one()) {
        volatile int* rec = records + (it & 3) * 8;
        rec[0] = w;
        rec[1] = (int)rng;
        rec[2] = im.jt * kBJ;
        rec[3] = im.i0;
        rec[4] = im.h;
        rec[5] = im.b;
        mbar_arrive(bar(ITEM + (it & 3)));
        mbar_arrive_expect_tx(bar(Q_FULL), slots * Cfg::kQBytes);
        for (int r = 0; r < slots; ++r)
          tma_load_5d(q_tile(r), &map_q, bar(Q_FULL), 0, im.jt * kBJ, slot_row(im, r), im.h, im.b);
      }
      __syncwarp();
      ++it;
      for (int st = lo; st < hi; ++st, ++g) {
        const int s = g % NS;
        if (g >= NS)
          ok = __all_sync(0xffffffffu, mbar_wait(bar(EMPTY + s), ((g / NS) - 1) & 1, abort_flag));
        if (!ok) break;
        if (elect_one()) {
          mbar_arrive_expect_tx(bar(FULL + s), 2 * slots * Cfg::kKVBytes + Cfg::kBiasBytes);
          for (int r = 0; r < slots; ++r) {
            tma_load_5d(k_tile(s, r), &map_k, bar(FULL + s), 0, st * kBK, slot_row(im, r), im.h, im.b);
            tma_load_5d(v_tile(s, r), &map_v, bar(FULL + s), 0, st * kBK, slot_row(im, r), im.h, im.b);
          }
          tma_load_4d(base + bias_off(s), &map_b, bar(FULL + s), st * kBK, im.jt * kBJ, im.h, im.b);
        }
        __syncwarp();
      }
    }
    if (ok && elect_one()) {
      records[(it & 3) * 8] = -1;
      mbar_arrive(bar(ITEM + (it & 3)));
    }
    __syncwarp();
  } else if (warp < kTmaWarp + 3) {
    // ------------------------------------------------------------ MMA issuers (two slots each)
    const int r0 = (warp - kTmaWarp - 1) * 2;
    constexpr bool kBf16 = std::is_same<T, __nv_bfloat16>::value;
    constexpr uint32_t idesc_qk = make_idesc(128, kBK, kBf16, false, false);
    constexpr uint32_t idesc_pv = make_idesc(128, D, kBf16, false, true);
    // (a K slice of 16 elements is 32 bytes further along the row; 16 rows of the MN-major V tile
    // are kStep16Rows units of 16 bytes further on)
    constexpr uint32_t kStep16Rows = (16 * Cfg::kRowBytes) >> 4;
    auto qk = [&](int r, int s, bool last_q) {   // in the elected lane
      const uint64_t ad = make_smem_desc(q_tile(r), 16, Cfg::kSbo, Cfg::kSwz);
      const uint64_t bd = make_smem_desc(k_tile(s, r), 16, Cfg::kSbo, Cfg::kSwz);
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk)
        umma_ss(tmem_base + r * 128, ad + 2 * kk, bd + 2 * kk, idesc_qk, kk > 0);
      umma_commit(bar(S_FULL + r));
      if (last_q) umma_commit(bar(Q_EMPTY));   // last read of this item's Q tile
    };
    int g = 0, gs = 0;   // running key steps of all items (ring) and of those this warp's slots walk
    int its = 0;         // running items of this warp's slots
    bool ok = true;
    for (int it = 0; ok; ++it) {
      ok = __all_sync(0xffffffffu, mbar_wait(bar(ITEM + (it & 3)), (it >> 2) & 1, abort_flag));
      if (!ok) break;
      const int w = uniform(records[(it & 3) * 8]);
      if (w < 0) break;
      const uint32_t rng = uniform(records[(it & 3) * 8 + 1]);
      const int steps = (rng >> 16) - (rng & 0xffffu);
      ok = mbar_wait(bar(Q_FULL), it & 1, abort_flag) &&
           mbar_wait(bar(FULL + g % NS), (g / NS) & 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      if (w >= items.full && r0 > 0) {   // half an item: these slots' share of the arrivals
        if (lane == 0) mbar_arrive_n(bar(Q_EMPTY), 2);
        for (int st = 0; st < steps && ok; ++st, ++g) {
          ok = __all_sync(0xffffffffu, mbar_wait(bar(FULL + g % NS), (g / NS) & 1, abort_flag));
          if (ok && lane == 0) mbar_arrive_n(bar(EMPTY + g % NS), 2 * 5);
        }
        continue;
      }
      // S of the first step (the P under it is read by MMAs issued before)
      tc_fence_after();
      if (elect_one()) {
        qk(r0, g % NS, steps == 1);
        qk(r0 + 1, g % NS, steps == 1);
      }
      __syncwarp();
      for (int st = 0; st < steps && ok; ++st, ++g, ++gs) {
        const int s = g % NS, ns = (g + 1) % NS;
        const bool more = st + 1 < steps;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int r = r0 + u;
          // the first PV of an item overwrites O: the previous item's epilogue must have read it
          ok = ok && mbar_wait(bar(P_READY + r), gs & 1, abort_flag) &&
               (st > 0 || its == 0 || mbar_wait(bar(O_FREE + r), (its - 1) & 1, abort_flag));
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tc_fence_after();
          const uint64_t bd = make_smem_desc(v_tile(s, r), Cfg::kSbo, Cfg::kSbo, Cfg::kSwz);
          const uint32_t t_r = tmem_base + r * 128, acc = st > 0 ? 1u : 0u;
          if (elect_one()) {
#pragma unroll
            for (int ks = 0; ks < kBK / 16; ++ks)
              umma_ts(t_r + 64, t_r + ks * 8, bd + ks * kStep16Rows, idesc_pv, ks > 0 ? 1u : acc);
            if (!more) umma_commit(bar(O_DONE + r));
            umma_commit(bar(EMPTY + s));
          }
          __syncwarp();
          if (more) {   // (the next stage may still be on its way: only this slot waits for it)
            ok = __all_sync(0xffffffffu, mbar_wait(bar(FULL + ns), ((g + 1) / NS) & 1, abort_flag));
            if (!ok) break;
            tc_fence_after();
            if (elect_one()) qk(r, ns, st + 2 == steps);
            __syncwarp();
          }
        }
      }
      ++its;
    }
  }
  } else {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsMath));
  {
    // ------------------------------------------------------------ softmax warpgroups
    const int r = warp >> 2, wq = warp & 3, t = tid & 127;
    const uint32_t lane_base = (uint32_t)(wq * 32) << 16;
    const uint32_t tS = tmem_base + lane_base + r * 128, tP = tS, tO = tS + 64;

    const float log2e = in_register(kLog2e), scale = in_register(dm.scale);
    // (as the issuers count, but with the ring's stage and phase and the slot's phase kept as such:
    // made from running counters they cost some forty instructions a step)
    int s = 0;
    uint32_t ring = 0u, turn = 0u;   // phase of the stage, of the slot's barriers
    bool ok = true;
    struct {
      int w, j0, i0, h, b;
      uint32_t rng, own;   // key steps of the item; the row's word of ws_rowrange
    } im, nx;
    auto next_item = [&](int it) {
      ok = __all_sync(0xffffffffu, mbar_wait(bar(ITEM + (it & 3)), (it >> 2) & 1, abort_flag));
      const volatile int* rec = records + (it & 3) * 8;
      nx.w = ok ? uniform(rec[0]) : -1;
      nx.rng = uniform((uint32_t)rec[1]);
      nx.j0 = rec[2];
      nx.i0 = rec[3];
      nx.h = rec[4];
      nx.b = rec[5];
      if (M != kAlone && nx.w >= 0) nx.own = __ldg(ws_rowrange + nx.b * dm.n_rows + min(nx.i0 + r, dm.n_rows - 1));
    };
    next_item(0);
    for (int it = 0; ok && nx.w >= 0; ++it) {
      im = nx;
      if (im.w >= items.full && r >= 2) break;   // half an item: the last one
      const int i = min(im.i0 + r, dm.n_rows - 1), b = im.b, h = im.h;
      // the row's own steps [lo, hi) within the item's [from, to): none for a row without an open key
      const int from = im.rng & 0xffffu, to = im.rng >> 16;
      const uint32_t own = M == kAlone ? 0u : uniform(im.own);
      const int lo = M == kAlone ? from : min(2 * (int)(own & 0xffffu), to);
      const int hi = M == kAlone ? to : max(lo, min(2 * (int)((own >> 16) & 0x7fffu), to));

      // Key mask of a step, fetched one step ahead.  Bytes: lane l < 16 reads keys 4l .. 4l + 3 as
      // one word.  Words: those of the 128-key chunk, of which the step is one half.
      const uint8_t* mrow = mask.p + b * mask.sb + (int64_t)i * mask.si;
      const uint32_t* mwords = ws_maskbits + ((int64_t)b * dm.n_rows + i) * ws_mask_words;
      // A row without an open key is left to the prepare kernel, which marks it with an empty range.
      // Where none runs (at most 128 keys, one word a lane: the mask of both steps) it is found here
      // and every score is 0: its weights are 1 and O / l the mean.
      bool row_full = hi == lo;
      uint32_t both = 0x01010101u;
      if (M == kAlone) {
        if (4 * lane < n) both = __ldg(reinterpret_cast<const uint32_t*>(mrow + 4 * lane));
        row_full = __all_sync(0xffffffffu, __vcmpeq4(both, 0u) == 0u);
        if (row_full && 4 * lane < n) both = 0u;
      }
      uint4 m_next;
      auto fetch_mask = [&](int st) {
        if constexpr (M == kWords) {
          m_next = __ldg(reinterpret_cast<const uint4*>(mwords + (st >> 1) * 4));
        } else if constexpr (M == kAlone) {
          m_next.x = __shfl_sync(0xffffffffu, both, st * 16 + (lane & 15));
          if (lane >= 16) m_next.x = 0u;
        } else {
          const int key4 = st * kBK + 4 * lane;
          m_next.x = lane >= 16 ? 0u : key4 < n ? __ldg(reinterpret_cast<const uint32_t*>(mrow + key4)) : 0x01010101u;
        }
      };
      // (a row without a dropped key needs its mask for the step at the row's end alone)
      const int masked_from = own >> 31 ? n / kBK : lo;
      if (masked_from <= lo && lo < hi) fetch_mask(lo);

      // Steps of the item's other rows: weights of zero, as a walk would give, and nothing else moves.
      auto pass_steps = [&](int count) {
        for (; count > 0; --count) {
          ok = mbar_wait(bar(FULL + s), ring, abort_flag) && mbar_wait(bar(S_FULL + r), turn, abort_flag);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tc_fence_after();
          uint32_t zero[16];
#pragma unroll
          for (int e = 0; e < 16; ++e) zero[e] = 0u;
          tmem_st16(tP, zero);
          tmem_st16(tP + 16, zero);
          tmem_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) {
            mbar_arrive(bar(EMPTY + s));
            mbar_arrive(bar(P_READY + r));
          }
          turn ^= 1u;
          if (++s == NS) {
            s = 0;
            ring ^= 1u;
          }
        }
      };
      if (M != kAlone) pass_steps(lo - from);
      if (!ok) break;

      float m_run = kMaxInit, l_run = 0.f;
      for (int st = lo; st < hi; ++st) {
        // mask words of this step (uniform over the warp): key c of the step is bit c >> 2 of word c & 3
        uint32_t mw[4] = {0u, 0u, 0u, 0u};
        bool clean = true;
        if (st >= masked_from) {
          if constexpr (M == kWords) {
            const int sh = (st & 1) * 16;
            mw[0] = (m_next.x >> sh) & 0xffffu;
            mw[1] = (m_next.y >> sh) & 0xffffu;
            mw[2] = (m_next.z >> sh) & 0xffffu;
            mw[3] = (m_next.w >> sh) & 0xffffu;
          } else {
#pragma unroll
            for (int jb = 0; jb < 4; ++jb)
              mw[jb] = __ballot_sync(0xffffffffu, ((m_next.x >> (8 * jb)) & 0xffu) != 0u);
          }
          clean = (mw[0] | mw[1] | mw[2] | mw[3]) == 0u;
        }
        if (st + 1 >= masked_from && st + 1 < hi) fetch_mask(st + 1);

        ok = mbar_wait(bar(FULL + s), ring, abort_flag) && mbar_wait(bar(S_FULL + r), turn, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        float x[64];
        tmem_ld32(tS, reinterpret_cast<uint32_t*>(x));
        tmem_ld32(tS + 32, reinterpret_cast<uint32_t*>(x) + 32);
        tmem_wait_ld();

        const uint8_t* brow = gbase + bias_off(s) + t * 128;
#pragma unroll
        for (int gq = 0; gq < 8; ++gq) {
          const uint4 u = *reinterpret_cast<const uint4*>(brow + ((gq ^ (t & 7)) << 4));
          float b0, b1;
          unpack2<T>(u.x, b0, b1);
          ffma2(x[gq * 8 + 0], x[gq * 8 + 1], x[gq * 8 + 0], x[gq * 8 + 1], scale, scale, b0, b1);
          unpack2<T>(u.y, b0, b1);
          ffma2(x[gq * 8 + 2], x[gq * 8 + 3], x[gq * 8 + 2], x[gq * 8 + 3], scale, scale, b0, b1);
          unpack2<T>(u.z, b0, b1);
          ffma2(x[gq * 8 + 4], x[gq * 8 + 5], x[gq * 8 + 4], x[gq * 8 + 5], scale, scale, b0, b1);
          unpack2<T>(u.w, b0, b1);
          ffma2(x[gq * 8 + 6], x[gq * 8 + 7], x[gq * 8 + 6], x[gq * 8 + 7], scale, scale, b0, b1);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(EMPTY + s));  // bias tile consumed by this warp

        if constexpr (M == kAlone)
          if (row_full)
#pragma unroll
            for (int c = 0; c < 64; ++c) x[c] = 0.f;
        if (!clean) {
#pragma unroll
          for (int c = 0; c < 64; ++c)
            if ((mw[c & 3] >> (c >> 2)) & 1u) x[c] = -INFINITY;
        }
        // four independent chains for the row maximum and the row sum
        float mx[4] = {x[0], x[1], x[2], x[3]};
#pragma unroll
        for (int c = 4; c < 60; c += 8) {  // 3-input max: two scores per instruction
          mx[0] = fmax3(mx[0], x[c + 0], x[c + 1]);
          mx[1] = fmax3(mx[1], x[c + 2], x[c + 3]);
          mx[2] = fmax3(mx[2], x[c + 4], x[c + 5]);
          mx[3] = fmax3(mx[3], x[c + 6], x[c + 7]);
        }
        mx[0] = fmax3(mx[0], x[60], x[61]);
        mx[1] = fmax3(mx[1], x[62], x[63]);
        const float mt = fmaxf(fmax3(mx[0], mx[1], mx[2]), mx[3]);
        // running maximum (see lazy_tau)
        const float m_new = (mt > m_run + lazy_tau<D>()) ? mt : m_run;
        const float neg = -m_new * kLog2e;
        // (difference first: exactly 1 when the maximum stays, also at the initial value,
        // where a fused m_run * log2e + neg would leave the rounding residue of 1e30 * log2e
        // in the exponent and turn a key step with no open key into inf * 0)
        const float alpha = ex2((m_run - m_new) * kLog2e);
        m_run = m_new;

        // (this S being complete, so is the O += P V before it)
        if (st > lo && __any_sync(0xffffffffu, alpha != 1.f)) {
          constexpr int kCols = D == 32 ? 32 : 16;   // (d = 64: registers)
#pragma unroll
          for (int c = 0; c < D; c += kCols) {
            uint32_t acc[kCols];
            tmem_ld_cols<kCols>(tO + c, acc);
            tmem_wait_ld();
            float* f = reinterpret_cast<float*>(acc);
#pragma unroll
            for (int e = 0; e < kCols; e += 2) fmul2(f[e], f[e + 1], f[e], f[e + 1], alpha, alpha);
            tmem_st_cols<kCols>(tO + c, acc);
          }
        }
        // exp and P store in chunks of 32 keys, so a packed chunk leaves the
        // registers as soon as it is made; four independent partial sums.
        float sm[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int ch = 0; ch < 2; ++ch) {
          uint32_t pk[16];
#pragma unroll
          for (int e = 0; e < 32; e += 4) {
            const int c = ch * 32 + e;
            float a0, a1, a2, a3;
            ffma2(a0, a1, x[c + 0], x[c + 1], log2e, log2e, neg, neg);
            ffma2(a2, a3, x[c + 2], x[c + 3], log2e, log2e, neg, neg);
            const float p0 = ex2(a0), p1 = ex2(a1), p2 = ex2(a2), p3 = ex2(a3);
            fadd2(sm[0], sm[1], sm[0], sm[1], p0, p1);
            fadd2(sm[2], sm[3], sm[2], sm[3], p2, p3);
            pk[(e >> 1) + 0] = pack2<T>(p0, p1);
            pk[(e >> 1) + 1] = pack2<T>(p2, p3);
          }
          tmem_st16(tP + ch * 16, pk);
        }
        l_run = fmaf(l_run, alpha, (sm[0] + sm[1]) + (sm[2] + sm[3]));
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(P_READY + r));
        turn ^= 1u;
        if (++s == NS) {
          s = 0;
          ring ^= 1u;
        }
      }
      if (!ok) break;

      if (M != kAlone) pass_steps(to - hi);
      if (!ok) break;

      // epilogue of the item: O / l and lse
      next_item(it + 1);   // (its record and, below, O arrive in each other's shadow)
      if (!ok) break;
      const bool do_store = im.i0 + r < dm.n_rows && !(row_full && M != kAlone);
      ok = __all_sync(0xffffffffu, mbar_wait(bar(O_DONE + r), it & 1, abort_flag));
      if (!ok) break;
      tc_fence_after();
      const int j = im.j0 + t;
      T* dst = reinterpret_cast<T*>(o.p) + b * o.sb + h * o.sh + (int64_t)i * o.si + (int64_t)j * o.sj;
      uint32_t acc[D];
      tmem_ld_cols<D>(tO, acc);
      tmem_wait_ld();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(O_FREE + r));  // the next item's first PV may overwrite O
      if (do_store && j < n) {
        const float inv = 1.f / l_run;
#pragma unroll
        for (int e = 0; e < D; e += 8) {
          uint4 u;
          u.x = pack2<T>(__uint_as_float(acc[e + 0]) * inv, __uint_as_float(acc[e + 1]) * inv);
          u.y = pack2<T>(__uint_as_float(acc[e + 2]) * inv, __uint_as_float(acc[e + 3]) * inv);
          u.z = pack2<T>(__uint_as_float(acc[e + 4]) * inv, __uint_as_float(acc[e + 5]) * inv);
          u.w = pack2<T>(__uint_as_float(acc[e + 6]) * inv, __uint_as_float(acc[e + 7]) * inv);
          *reinterpret_cast<uint4*>(dst + e) = u;
        }
        lse[(((int64_t)b * dm.heads + h) * dm.n_rows + i) * n + j] =
            row_full ? dm.sentinel : fmaf(lg2(l_run), kLn2, m_run);
      }
    }
  }
  }

  // ---------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    // A wait gave up: let copies and MMAs in flight land before TMEM and shared
    // memory are released, then report through the status word.
    const long long t0 = clock64();
    while (clock64() - t0 < 4000000LL) {
    }
    if (tid == 0) set_status(status, kStatusTimeoutFwd);
    __syncthreads();
  }
  if (warp == kTmaWarp + 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

template <typename T, int D>
cudaError_t launch(const FwdArgs& a, cudaStream_t stream) {
  using Cfg = FwdCfg<D>;
  const Dims& dm = a.dm;
  const bool bf16 = std::is_same<T, __nv_bfloat16>::value;
  const uint64_t eb = 2;
  CUtensorMap mq, mk, mv, mbias;
  const uint64_t dims5[5] = {(uint64_t)D, (uint64_t)dm.n, (uint64_t)dm.n_rows, (uint64_t)dm.heads,
                             (uint64_t)dm.batch};
  const uint32_t box_q[5] = {(uint32_t)D, kBJ, 1, 1, 1}, box_kv[5] = {(uint32_t)D, kBK, 1, 1, 1};
  const CUtensorMapSwizzle swz = (CUtensorMapSwizzle)RowSwizzle<D>::kTma;
  auto map5 = [&](CUtensorMap* m, const View5& v, const uint32_t* box5) {
    const uint64_t st[4] = {(uint64_t)v.sj * eb, (uint64_t)v.si * eb, (uint64_t)v.sh * eb,
                            (uint64_t)v.sb * eb};
    return make_tensor_map(m, bf16, 5, v.p, dims5, st, box5, swz);
  };
  if (!map5(&mq, a.q, box_q) || !map5(&mk, a.k, box_kv) || !map5(&mv, a.v, box_kv))
    return cudaErrorInvalidValue;
  {
    // the bias itself when its rows are 16-byte pitched, else the padded copy
    const uint64_t n = dm.n, np = dm.n_pad;
    const uint64_t dims4[4] = {n, n, (uint64_t)dm.heads, (uint64_t)dm.batch};
    const uint64_t st_user[3] = {(uint64_t)a.bias.sj * eb, (uint64_t)a.bias.sh * eb, (uint64_t)a.bias.sb * eb};
    const uint64_t st_pad[3] = {np * eb, n * np * eb, n * np * dm.heads * eb};
    const uint32_t box4[4] = {64, 128, 1, 1};
    if (!make_tensor_map(&mbias, bf16, 4, a.bias_pad ? a.bias_pad : (void*)a.bias.p, dims4,
                         a.bias_pad ? st_pad : st_user, box4, CU_TENSOR_MAP_SWIZZLE_128B))
      return cudaErrorInvalidValue;
  }
  constexpr auto kern_w = tc_fwd_kernel<T, D, kWords>;
  constexpr auto kern_b = tc_fwd_kernel<T, D, kBytes>;
  constexpr auto kern_a = tc_fwd_kernel<T, D, kAlone>;
  const auto kern = a.maskbits ? kern_w : a.rowrange ? kern_b : kern_a;
  cudaError_t e = a.maskbits   ? opt_in_smem<kern_w, true>(Cfg::kSmemBytes)
                  : a.rowrange ? opt_in_smem<kern_b, true>(Cfg::kSmemBytes)
                               : opt_in_smem<kern_a, true>(Cfg::kSmemBytes);
  if (e != cudaSuccess) return e;
  ItemGrid items;
  items.njt = (dm.n + kBJ - 1) / kBJ;
  items.nrg = (dm.n_rows + kR - 1) / kR;
  const int sms = sm_count(), groups = items.njt * items.nrg * dm.batch * dm.heads;
  const int rest = groups % sms;
  items.full = 2 * rest <= sms ? groups - rest : groups;
  items.total = items.full + 2 * (groups - items.full);
  const int grid = items.total < sms ? items.total : sms;
  return launch_early(kern, grid, Cfg::kThreads, Cfg::kSmemBytes, stream, mq, mk, mv, mbias, a.o, a.lse, a.mask,
                      a.maskbits, a.mask_words, a.rowrange, dm, items, a.status);
}

}  // namespace

namespace tc {

EncodeTiledFn get_encode_tiled() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}

static bool encode(CUtensorMap* map, CUtensorMapDataType dt, uint64_t elem_bytes, int rank,
                   void* base, const uint64_t* dims, const uint64_t* strides_bytes,
                   const uint32_t* box, CUtensorMapSwizzle swz) {
  EncodeTiledFn enc = get_encode_tiled();
  if (!enc) return false;
  cuuint64_t gdim[5], gstr[4];
  cuuint32_t bx[5], es[5];
  for (int i = 0; i < rank; ++i) {
    gdim[i] = dims[i];
    bx[i] = box[i];
    es[i] = 1;
  }
  for (int i = 0; i + 1 < rank; ++i) {
    uint64_t s = strides_bytes[i];
    // extent-1 dimensions may come with arbitrary strides: give them the dense pitch
    // (rounded up to the 16 bytes a stride must be a multiple of; it is never stepped)
    if (dims[i + 1] == 1)
      s = (i == 0) ? ((dims[0] * elem_bytes + 15) & ~(uint64_t)15) : gstr[i - 1] * dims[i];
    if (s == 0 || (s & 15)) return false;
    gstr[i] = s;
  }
  const CUresult r = enc(map, dt, (cuuint32_t)rank, base, gdim, gstr, bx, es,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, swz, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

bool make_tensor_map(CUtensorMap* map, bool bf16, int rank, void* base, const uint64_t* dims,
                     const uint64_t* strides_bytes, const uint32_t* box, CUtensorMapSwizzle swz) {
  return encode(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2,
                rank, base, dims, strides_bytes, box, swz);
}

bool make_tensor_map_f32(CUtensorMap* map, int rank, void* base, const uint64_t* dims,
                         const uint64_t* strides_bytes, const uint32_t* box) {
  return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, rank, base, dims, strides_bytes, box,
                CU_TENSOR_MAP_SWIZZLE_NONE);
}

}  // namespace tc

bool tc_forward_supported(const Dims& dm, int dtype, const FwdArgs* a) {
  if (dtype != TRIFAST_BF16 && dtype != TRIFAST_F16) return false;
  if (dm.d != 16 && dm.d != 32 && dm.d != 64) return false;
  if (dm.n < kMinTensorCoreN) return false;
  if (a) {
    if (((uintptr_t)a->o.p) & 15 || (a->o.sj * 2) % 16) return false;
    const bool have_ws = a->bias_pad && a->maskbits && a->rowfull;
    if (!have_ws) {
      // without the prepared copies the bias goes through TMA as it is (16-byte row
      // pitch) and the key mask is read four bytes at a time
      if (dm.n % 8 != 0 || !bias_fits_tma(a->bias, dm)) return false;
      if (((uintptr_t)a->mask.p) & 3 || a->mask.sb % 4 || a->mask.si % 4) return false;
    }
  }
  return tc::get_encode_tiled() != nullptr;
}

cudaError_t tc_forward(const FwdArgs& a, cudaStream_t s) {
  const bool bf16 = a.dtype == TRIFAST_BF16;
  switch (a.dm.d) {
    case 16: return bf16 ? launch<__nv_bfloat16, 16>(a, s) : launch<__half, 16>(a, s);
    case 32: return bf16 ? launch<__nv_bfloat16, 32>(a, s) : launch<__half, 32>(a, s);
    default: return bf16 ? launch<__nv_bfloat16, 64>(a, s) : launch<__half, 64>(a, s);
  }
}

}  // namespace trifast
