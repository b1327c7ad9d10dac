// dq, and dk / dv, of triangle attention at head dim 128 on the tensor cores (bf16 / fp16).
//
// dK + dV (256 TMEM columns) beside S^T, dP^T, P^T and dS^T leave no room for dQ of even one
// 128-query tile, so the two directions are two launches of one kernel.  Both walk a resident
// pair of 128-row tiles over a streamed pair of 64-row tiles of the same pair row:
//     dq   : resident Q, dO (128 queries),  streamed K, V;    lanes = queries
//            S = Q K^T, dP = dO V^T,  dS = P (dP - delta),    dQ += dS K
//     dk/dv: resident K, V (128 keys),      streamed Q, dO;   lanes = keys
//            S^T = K Q^T, dP^T = V dO^T,                      dV += P^T dO,  dK += dS^T Q
// with P = exp2(S c + bias log2e - lse log2e).
//
// Precision: P and dS enter the products as the sum of two 16-bit operands each, the rounded value
// and the remainder (split2), so every accumulating product runs twice.  dq, dk and dv then
// carry the rounding of the result and no more: against float64 at n = 512, dq 1.707e-3 (bf16) and
// 2.133e-4 (fp16) in the 2-norm, the digits that fp32 products on the CUDA cores give; with P
// and dS rounded to one operand 2.391e-3 and 2.988e-4.  fp16 has a range to keep to as well: P is
// held times 2^15, dS times a power of two per pair row that the prepare step takes from the
// largest |dO| and |v| (ds_up), both undone on the accumulators.
//
// A row of 128 elements is two 128-byte swizzle spans: every tile is two [rows x 64] halves (two
// TMA boxes); K-major operands take their K slices from one half or the other, MN-major ones
// get the halves as their two N atoms.
//
// The bias tile is the one operand that is not transposed with the rest: lanes = keys read
// it down its columns, 2 bytes per lane and query from unswizzled 256-byte rows (a warp reads
// 64 consecutive bytes), which spares the transposed copy of the bias that the kernels for
// smaller head dims keep in the workspace.
//
// Warps 0-7: elementwise (warps w and w + 4 share the lanes and take 32 of a step's 64
// columns each); 8 TMA; 9 S / dP MMAs and the TMEM allocation; 10 accumulating MMAs; 11
// completes the warpgroup whose registers are handed over.  Work items are persistent over
// the SMs, and three stages are kept in flight: a stage is held for two steps plus its load
// latency, so two stages would stall on it.  A step of dq and one of dk/dv cost about 6900 cycles
// together, of which the MMAs hold the tensor pipe for about 2500: the hops between the warps
// bound it, as in the kernels for smaller head dims.  Measured at n = 512, h = 4: dq and dk/dv
// together 1.42 ms in bf16 and 1.50 ms in fp16 (1.56 and 1.75 before an elected lane issued the
// MMAs, and then 1.32 and 1.39 with P and dS in one 16-bit operand each), where the CUDA-core
// kernels took 85.6 ms (db, one row as two stages of half the head dim in tc_bwd_db.cu: 379 us
// against 22.3 ms).
//
// Stands in for `_bwd_q` and `_bwd_kv` of the reference (src/trifast/triton.py:268-383,
// :137-263).  Masked keys weigh exactly zero; rows whose keys are all masked use P = 1/n
// (the PyTorch semantics, src/trifast/equiv.py:42-69).

#include <math.h>

#include <type_traits>

#include "kernels.h"
#include "tc_common.cuh"

namespace trifast {
namespace {
using namespace tc;

constexpr int kD = 128, kStep = 64, kStages = 3;
constexpr float kLog2e = 1.4426950408889634f;
// Register hand-over (setmaxnreg): 384 threads launch with 168 registers each; what the math
// warpgroups gain must not exceed what the issue warpgroup releases.
constexpr int kRegsIssue = 56, kRegsMath = 224;
static_assert(256 * kRegsMath + 128 * kRegsIssue <= 384 * 168, "setmaxnreg pool");

constexpr int kResHalf = 128 * 128, kResBytes = 2 * kResHalf;       // resident tile: 128 rows
constexpr int kStrHalf = kStep * 128, kStrBytes = 2 * kStrHalf;     // streamed tile: 64 rows
constexpr int kBiasBytes = 128 * kStep * 2;
constexpr int kStageBytes = 2 * kStrBytes + kBiasBytes;             // 48 KiB
constexpr int kVecBytes = kStep * 4;                                // -lse log2e or delta of 64 queries
constexpr int kHeader = 3072;                                       // barriers, flags, vectors
constexpr int kVecOff = 1024;                                       // [stage][2][64] floats
constexpr int kSmemBytes = 1024 + kHeader + 2 * kResBytes + kStages * kStageBytes;
static_assert(kVecOff + kStages * 2 * kVecBytes <= kHeader && kSmemBytes <= 232448, "shared memory");

struct Grid {
  int tiles;   // 128-row resident tiles per pair row
  int steps;   // 64-row streamed tiles per pair row
  int total;   // work items
};

template <typename T, bool kKv>
__global__ void __launch_bounds__(384, 1)
tc_bwd_d128_kernel(const __grid_constant__ CUtensorMap map_a1, const __grid_constant__ CUtensorMap map_a2,
                   const __grid_constant__ CUtensorMap map_b1, const __grid_constant__ CUtensorMap map_b2,
                   const __grid_constant__ CUtensorMap map_bias,
                   const __grid_constant__ CUtensorMap map_nlse,
                   const __grid_constant__ CUtensorMap map_delta, View5 out1, View5 out2,
                   const float* __restrict__ neg_lse2, const float* __restrict__ delta,
                   const float* __restrict__ ds_up, const uint8_t* __restrict__ rowfull, const uint32_t* __restrict__ maskbits_lin,
                   int mask_words, const uint32_t* __restrict__ rowrange, Dims dm, Grid grid,
                   unsigned int* status) {
  // TMEM columns: SB buffers of S, dP (64 each), then dS (and P) as 16-bit pairs, the rounded
  // values and the remainders (32 columns each), then the accumulators
  constexpr int SB = kKv ? 1 : 2;
  constexpr int kDsCol = SB * 128, kPCol = kDsCol + 64;
  constexpr int kAcc1 = kKv ? kPCol + 64 : kDsCol + 64;   // dQ, or dK
  constexpr int kAcc2 = kAcc1 + kD;                       // dV
  // fp16: P times 2^15 and dS times ds_up, so that neither leaves the type's normal range
  constexpr bool kUp = std::is_same<T, __half>::value;
  constexpr float kUpLog2 = kUp ? 15.f : 0.f, kUpP = kUp ? 32768.f : 1.f;
  static_assert((kKv ? kAcc2 : kAcc1) + kD <= 512, "TMEM columns");
  constexpr int A_FULL = 0, A_EMPTY = 1, FULL = 2, EMPTY = FULL + kStages, S_FULL = EMPTY + kStages,
                S_FREE = S_FULL + 2, P_READY = S_FREE + 2, ACC_DONE = P_READY + 2,
                ACC_FREE = ACC_DONE + 2, NBARS = ACC_FREE + 1;
  static_assert(NBARS * 8 <= 256, "barrier area");

  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* gbase = smem_raw + (base - raw);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gbase + 256);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gbase + 260);

  const int n = dm.n;
  auto bar = [&](int i) -> uint32_t { return base + 8u * i; };
  const uint32_t a1_tile = base + kHeader, a2_tile = a1_tile + kResBytes;
  auto stage_off = [&](int s) -> uint32_t { return kHeader + 2 * kResBytes + s * kStageBytes; };
  auto b1_tile = [&](int s) -> uint32_t { return base + stage_off(s); };
  auto b2_tile = [&](int s) -> uint32_t { return base + stage_off(s) + kStrBytes; };
  auto bias_off = [&](int s) -> uint32_t { return stage_off(s) + 2 * kStrBytes; };
  auto vec_off = [&](int s) -> uint32_t { return kVecOff + s * 2 * kVecBytes; };
  struct Item {
    int tile, i, h, b;
  };
  // tile fastest, then row, then (b, h): the CTAs running together share streamed tiles and
  // bias in L2
  auto decode = [&](int w) -> Item {
    Item it;
    it.tile = w % grid.tiles;
    const int rest = w / grid.tiles;
    it.i = rest % dm.n_rows;
    const int bh = rest / dm.n_rows;
    it.h = bh % dm.heads;
    it.b = bh / dm.heads;
    return it;
  };
  // Steps [lo, hi) an item walks, as lo | hi << 16.  dq: the key tiles of the row that hold
  // an open key; dk/dv: every query, or nothing when the item's key tile holds no open key.
  auto item_steps = [&](int w) -> uint32_t {
    if (w >= grid.total) return 0u;
    const Item it = decode(w);
    const uint32_t v = uniform(__ldg(rowrange + it.b * dm.n_rows + it.i));
    const int lo = v & 0xffffu, hi = v >> 16;
    if (kKv) return (it.tile >= lo && it.tile < hi) ? (uint32_t)grid.steps << 16 : 0u;
    return (uint32_t)(2 * lo) | (uint32_t)min(2 * hi, grid.steps) << 16;
  };

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&map_a1);
    tma_prefetch_desc(&map_a2);
    tma_prefetch_desc(&map_b1);
    tma_prefetch_desc(&map_b2);
    tma_prefetch_desc(&map_bias);
    if (kKv) {
      tma_prefetch_desc(&map_nlse);
      tma_prefetch_desc(&map_delta);
    }
  }
  after_previous();

  if (*reinterpret_cast<volatile unsigned int*>(status) != 0u) return;

  const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;
  if (tid == 0) {
    mbar_init(bar(A_FULL), 1);
    mbar_init(bar(A_EMPTY), 1);
    for (int s = 0; s < kStages; ++s) {
      mbar_init(bar(FULL + s), 1);
      mbar_init(bar(EMPTY + s), 9);   // the accumulating commit + the 8 elementwise warps
    }
    for (int u = 0; u < 2; ++u) {
      mbar_init(bar(S_FULL + u), 1);
      mbar_init(bar(S_FREE + u), 8);
      mbar_init(bar(P_READY + u), 8);
      mbar_init(bar(ACC_DONE + u), 1);
    }
    mbar_init(bar(ACC_FREE), 8);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 9) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = uniform(*tmem_slot);

  if (warp >= 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsIssue));
    if (warp == 8) {
      // ------------------------------------------------------------ TMA producer
      {
        int g = 0, it = 0;   // running step and (walked) item counters: barrier phases
        bool ok = true;
        uint32_t next = item_steps(blockIdx.x);
        for (int w = blockIdx.x; w < grid.total && ok; w += gridDim.x) {
          const int lo = next & 0xffffu, hi = next >> 16;
          next = item_steps(w + gridDim.x);
          if (lo >= hi) continue;
          const Item im = decode(w);
          if (it > 0) ok = __all_sync(0xffffffffu, mbar_wait(bar(A_EMPTY), (it - 1) & 1, abort_flag));
          if (!ok) break;
          ++it;
          if (elect_one()) {
            mbar_arrive_expect_tx(bar(A_FULL), 2 * kResBytes);
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
              tma_load_5d(a1_tile + hf * kResHalf, &map_a1, bar(A_FULL), hf * 64, im.tile * 128, im.i, im.h, im.b);
              tma_load_5d(a2_tile + hf * kResHalf, &map_a2, bar(A_FULL), hf * 64, im.tile * 128, im.i, im.h, im.b);
            }
          }
          __syncwarp();
          for (int st = lo; st < hi; ++st, ++g) {
            const int s = g % kStages;
            if (g >= kStages)
              ok = __all_sync(0xffffffffu, mbar_wait(bar(EMPTY + s), (g / kStages - 1) & 1, abort_flag));
            if (!ok) break;
            const uint32_t full = bar(FULL + s);
            if (elect_one()) {
              mbar_arrive_expect_tx(full, kStageBytes + (kKv ? 2 * kVecBytes : 0));
#pragma unroll
              for (int hf = 0; hf < 2; ++hf) {
                tma_load_5d(b1_tile(s) + hf * kStrHalf, &map_b1, full, hf * 64, st * kStep, im.i, im.h, im.b);
                tma_load_5d(b2_tile(s) + hf * kStrHalf, &map_b2, full, hf * 64, st * kStep, im.i, im.h, im.b);
              }
              // (keys innermost in both cases)
              tma_load_4d(base + bias_off(s), &map_bias, full, kKv ? im.tile * 128 : st * kStep,
                          kKv ? st * kStep : im.tile * 128, im.h, im.b);
              if (kKv) {
                tma_load_4d(base + vec_off(s), &map_nlse, full, st * kStep, im.i, im.h, im.b);
                tma_load_4d(base + vec_off(s) + kVecBytes, &map_delta, full, st * kStep, im.i, im.h, im.b);
              }
            }
            __syncwarp();
          }
        }
      }
    } else if (warp == 9) {
      // ------------------------------------------------------------ S / dP issuer
      constexpr bool kBf16 = std::is_same<T, __nv_bfloat16>::value;
      constexpr uint32_t idesc = make_idesc(128, kStep, kBf16, false, false);
      int g = 0, it = 0;
      bool ok = true;
      uint32_t next = item_steps(blockIdx.x);
      for (int w = blockIdx.x; w < grid.total && ok; w += gridDim.x) {
        const int lo = next & 0xffffu, hi = next >> 16;
        next = item_steps(w + gridDim.x);
        if (lo >= hi) continue;
        for (int st = lo; st < hi; ++st, ++g) {
          const int s = g % kStages, gp = g - SB;   // the buffer was last read at step g - SB
          ok = (st > lo || mbar_wait(bar(A_FULL), it & 1, abort_flag)) &&
               mbar_wait(bar(FULL + s), (g / kStages) & 1, abort_flag) &&
               (gp < 0 || mbar_wait(bar(S_FREE + (gp & 1)), (gp >> 1) & 1, abort_flag));
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tc_fence_after();
          const uint32_t t_s = tmem_base + (g % SB) * 128;
          const uint64_t d1 = make_smem_desc(a1_tile, 16, 1024, kSwizzle128);
          const uint64_t d2 = make_smem_desc(a2_tile, 16, 1024, kSwizzle128);
          const uint64_t e1 = make_smem_desc(b1_tile(s), 16, 1024, kSwizzle128);
          const uint64_t e2 = make_smem_desc(b2_tile(s), 16, 1024, kSwizzle128);
          if (elect_one()) {
            // K slice kk: 32 bytes further along the row, the upper four in the second half
#pragma unroll
            for (int kk = 0; kk < kD / 16; ++kk)
              umma_ss(t_s, d1 + ((kk >> 2) * (kResHalf >> 4) + (kk & 3) * 2),
                      e1 + ((kk >> 2) * (kStrHalf >> 4) + (kk & 3) * 2), idesc, kk > 0);
#pragma unroll
            for (int kk = 0; kk < kD / 16; ++kk)
              umma_ss(t_s + 64, d2 + ((kk >> 2) * (kResHalf >> 4) + (kk & 3) * 2),
                      e2 + ((kk >> 2) * (kStrHalf >> 4) + (kk & 3) * 2), idesc, kk > 0);
            umma_commit(bar(S_FULL + (g & 1)));
            if (st == hi - 1) umma_commit(bar(A_EMPTY));   // last read of the resident tiles
          }
          __syncwarp();
        }
        ++it;
      }
    } else if (warp == 10) {
      // ------------------------------------------------------------ accumulating issuer
      constexpr bool kBf16 = std::is_same<T, __nv_bfloat16>::value;
      constexpr uint32_t idesc = make_idesc(128, kD, kBf16, false, true);
      int g = 0, it = 0;
      bool ok = true;
      uint32_t next = item_steps(blockIdx.x);
      for (int w = blockIdx.x; w < grid.total && ok; w += gridDim.x) {
        const int lo = next & 0xffffu, hi = next >> 16;
        next = item_steps(w + gridDim.x);
        if (lo >= hi) continue;
        for (int st = lo; st < hi; ++st, ++g) {
          const int s = g % kStages;
          // an item's first MMAs overwrite the accumulators: the previous item's epilogue must
          // have read them
          ok = mbar_wait(bar(P_READY + (g & 1)), (g >> 1) & 1, abort_flag) &&
               (st > lo || it == 0 || mbar_wait(bar(ACC_FREE), (it - 1) & 1, abort_flag));
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tc_fence_after();
          // 16 rows of a streamed tile are 2 KiB; its two halves are the two N atoms
          const uint64_t e1 = make_smem_desc(b1_tile(s), kStrHalf, 1024, kSwizzle128);
          const uint64_t e2 = make_smem_desc(b2_tile(s), kStrHalf, 1024, kSwizzle128);
          if (elect_one()) {
            if (kKv) {
#pragma unroll
              for (int ks = 0; ks < kStep / 16; ++ks)
#pragma unroll
                for (int lo_part = 0; lo_part < 2; ++lo_part)
                  umma_ts(tmem_base + kAcc2, tmem_base + kPCol + lo_part * 32 + ks * 8, e2 + ks * 128, idesc,
                          st > lo || ks > 0 || lo_part > 0);
            }
#pragma unroll
            for (int ks = 0; ks < kStep / 16; ++ks)
#pragma unroll
              for (int lo_part = 0; lo_part < 2; ++lo_part)
                umma_ts(tmem_base + kAcc1, tmem_base + kDsCol + lo_part * 32 + ks * 8, e1 + ks * 128, idesc,
                        st > lo || ks > 0 || lo_part > 0);
            umma_commit(bar(ACC_DONE + (g & 1)));
            umma_commit(bar(EMPTY + s));
          }
          __syncwarp();
        }
        ++it;
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsMath));
    // -------------------------------------------------------------- elementwise warps
    // Thread = one query (dq) or one key (dk/dv), columns [32 half, 32 half + 32) of a step.
    const int half = warp >> 2, wq = warp & 3, t = tid & 127;
    const uint32_t lane_base = (uint32_t)(wq * 32) << 16;
    const uint32_t tS0 = tmem_base + lane_base + half * 32;
    const uint32_t tDS = tmem_base + lane_base + kDsCol + half * 16;
    const uint32_t tP = tmem_base + lane_base + kPCol + half * 16;
    const float c1 = dm.scale * kLog2e;
    const float p_full = kUpP / (float)n;

    int g = 0;
    bool ok = true;
    uint32_t next = item_steps(blockIdx.x);
    for (int w = blockIdx.x; w < grid.total && ok; w += gridDim.x) {
      const int lo = next & 0xffffu, hi = next >> 16;
      next = item_steps(w + gridDim.x);
      const Item im = decode(w);
      const int i = im.i, b = im.b, h = im.h;
      const int row = im.tile * 128 + t;   // this thread's query or key
      auto out_row = [&](const View5& o) -> T* {
        return reinterpret_cast<T*>(o.p) + b * o.sb + h * o.sh + (int64_t)i * o.si + (int64_t)row * o.sj;
      };
      if (lo >= hi) {   // (dk/dv only) no open key in this tile: zero
        if (row < n) {
          T* dst = out_row(half ? out2 : out1);
#pragma unroll
          for (int e = 0; e < kD; e += 8) *reinterpret_cast<uint4*>(dst + e) = make_uint4(0u, 0u, 0u, 0u);
        }
        continue;
      }
      const bool row_full = rowfull[b * dm.n_rows + i] != 0;
      // key mask in key order (bit set = dropped or beyond n; on a fully masked row only beyond n)
      const uint32_t* mrow = maskbits_lin + ((int64_t)b * dm.n_rows + i) * mask_words;
      // dS is P (dP - delta) times `up`, of which P already carries kUpP
      const float up = kUp ? __ldg(ds_up + ((int64_t)b * dm.heads + h) * dm.n_rows + i) : 1.f;
      const float up_dp = up / kUpP;
      float nl_row = 0.f, ndl_row = 0.f;
      uint32_t mw_next = 0u;
      bool dropped = false;
      if (kKv) {
        dropped = ((__ldg(mrow + im.tile * 4 + wq) >> lane) & 1u) != 0u;
      } else {
        const int64_t at = (((int64_t)b * dm.heads + h) * dm.n_rows + i) * dm.n_pad + min(row, n - 1);
        nl_row = __ldg(neg_lse2 + at) + kUpLog2;
        ndl_row = -__ldg(delta + at) * up_dp;
        mw_next = __ldg(mrow + lo * 2 + half);
      }
      auto steps = [&](auto full_tag) {
        constexpr bool kRowFull = decltype(full_tag)::value;
        for (int st = lo; st < hi; ++st, ++g) {
          const int s = g % kStages;
          const uint32_t mw = mw_next;   // dq: this warp's 32 keys, fetched one step ahead
          if (!kKv && st + 1 < hi) mw_next = __ldg(mrow + (st + 1) * 2 + half);
          ok = __all_sync(0xffffffffu,
                          mbar_wait(bar(S_FULL + (g & 1)), (g >> 1) & 1, abort_flag) &&
                              mbar_wait(bar(FULL + s), (g / kStages) & 1, abort_flag));
          if (!ok) break;
          tc_fence_after();
          float x[32], gd[32];
          const uint32_t tS = tS0 + (g % SB) * 128;
          tmem_ld32(tS, reinterpret_cast<uint32_t*>(x));
          tmem_ld32(tS + 64, reinterpret_cast<uint32_t*>(gd));
          tmem_wait_ld();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(S_FREE + (g & 1)));

          uint32_t pp[16], pp_lo[16], pd[16], pd_lo[16];
          const uint8_t* bias_s = gbase + bias_off(s);
          const float4* nl4 = reinterpret_cast<const float4*>(gbase + vec_off(s)) + half * 8;
          const float4* dl4 = nl4 + kVecBytes / 16;
#pragma unroll
          for (int q8 = 0; q8 < 4; ++q8) {
            float bv[8], nl[8], dl[8];   // (dl: delta, or -delta up_dp where the query is this thread's)
            if (kKv) {
              const float4 da = dl4[q8 * 2], db = dl4[q8 * 2 + 1];
              dl[0] = da.x; dl[1] = da.y; dl[2] = da.z; dl[3] = da.w;
              dl[4] = db.x; dl[5] = db.y; dl[6] = db.z; dl[7] = db.w;
              if (!kRowFull) {
                const float4 la = nl4[q8 * 2], lb = nl4[q8 * 2 + 1];
                nl[0] = la.x; nl[1] = la.y; nl[2] = la.z; nl[3] = la.w;
                nl[4] = lb.x; nl[5] = lb.y; nl[6] = lb.z; nl[7] = lb.w;
#pragma unroll
                for (int e = 0; e < 8; ++e)
                  bv[e] = to_f32<T>(*reinterpret_cast<const T*>(bias_s + (half * 32 + q8 * 8 + e) * 256 + t * 2));
              }
            } else {
#pragma unroll
              for (int e = 0; e < 8; ++e) {
                nl[e] = nl_row;
                dl[e] = ndl_row;
              }
              if (!kRowFull) {
                const uint4 u = *reinterpret_cast<const uint4*>(bias_s + t * 128 + (((half * 4 + q8) ^ (t & 7)) << 4));
                unpack2<T>(u.x, bv[0], bv[1]);
                unpack2<T>(u.y, bv[2], bv[3]);
                unpack2<T>(u.z, bv[4], bv[5]);
                unpack2<T>(u.w, bv[6], bv[7]);
              }
            }
#pragma unroll
            for (int e = 0; e < 8; e += 2) {   // packed fp32 pairs: two scores per instruction
              const int col = q8 * 8 + e;
              float p0 = p_full, p1 = p_full;
              if (!kRowFull) {
                float t0, t1, a0, a1;
                if (kKv && kUp) fadd2(nl[e], nl[e + 1], nl[e], nl[e + 1], kUpLog2, kUpLog2);
                ffma2(t0, t1, bv[e], bv[e + 1], kLog2e, kLog2e, nl[e], nl[e + 1]);
                ffma2(a0, a1, x[col], x[col + 1], c1, c1, t0, t1);
                p0 = ex2(a0);
                p1 = ex2(a1);
              }
              if (kKv) {
                p0 = dropped ? 0.f : p0;
                p1 = dropped ? 0.f : p1;
              } else {
                p0 = ((mw >> col) & 1u) ? 0.f : p0;
                p1 = ((mw >> (col + 1)) & 1u) ? 0.f : p1;
              }
              float s0, s1, d0, d1;   // (dP - delta) up_dp
              if (kKv && !kUp) {
                ffma2(s0, s1, dl[e], dl[e + 1], -1.f, -1.f, gd[col], gd[col + 1]);
              } else {
                if (kKv) fmul2(dl[e], dl[e + 1], dl[e], dl[e + 1], -up_dp, -up_dp);
                ffma2(s0, s1, gd[col], gd[col + 1], up_dp, up_dp, dl[e], dl[e + 1]);
              }
              fmul2(d0, d1, p0, p1, s0, s1);
              if (kKv) split2<T>(p0, p1, pp[col >> 1], pp_lo[col >> 1]);
              split2<T>(d0, d1, pd[col >> 1], pd_lo[col >> 1]);
            }
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(EMPTY + s));   // bias and vectors consumed by this warp

          if (g >= 1) {   // the previous step's accumulating MMAs still read P, dS
            ok = __all_sync(0xffffffffu, mbar_wait(bar(ACC_DONE + ((g - 1) & 1)),
                                                        ((g - 1) >> 1) & 1, abort_flag));
            if (!ok) break;
          }
          if (kKv) {
            tmem_st16(tP, pp);
            tmem_st16(tP + 32, pp_lo);
          }
          tmem_st16(tDS, pd);
          tmem_st16(tDS + 32, pd_lo);
          tmem_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(P_READY + (g & 1)));
        }
      };
      if (row_full) steps(std::true_type{}); else steps(std::false_type{});
      if (!ok) break;

      // epilogue: dk/dv: half 0 takes dK, half 1 dV; dq: 64 columns each
      ok = __all_sync(0xffffffffu, mbar_wait(bar(ACC_DONE + ((g - 1) & 1)), ((g - 1) >> 1) & 1,
                                                  abort_flag));
      if (!ok) break;
      tc_fence_after();
      constexpr int kCols = kKv ? kD : kD / 2;
      const uint32_t tAcc = tmem_base + lane_base + (kKv && half ? kAcc2 : kAcc1) + (kKv ? 0 : half * kCols);
      const float sc = (kKv && half) ? 1.f / kUpP : dm.scale / up;
      // a dropped key gets exactly zero, also where a query's dO, lse or delta is not finite
      const bool zero = kKv && dropped;
      uint32_t acc[kCols];
      tmem_ld_cols<kCols>(tAcc, acc);
      tmem_wait_ld();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(ACC_FREE));
      if (row < n) {
        T* dst = out_row(kKv && half ? out2 : out1) + (kKv ? 0 : half * kCols);
#pragma unroll
        for (int e = 0; e < kCols; e += 8) {
          uint4 u;
          u.x = pack2<T>(__uint_as_float(acc[e + 0]) * sc, __uint_as_float(acc[e + 1]) * sc);
          u.y = pack2<T>(__uint_as_float(acc[e + 2]) * sc, __uint_as_float(acc[e + 3]) * sc);
          u.z = pack2<T>(__uint_as_float(acc[e + 4]) * sc, __uint_as_float(acc[e + 5]) * sc);
          u.w = pack2<T>(__uint_as_float(acc[e + 6]) * sc, __uint_as_float(acc[e + 7]) * sc);
          if (zero) u = make_uint4(0u, 0u, 0u, 0u);
          *reinterpret_cast<uint4*>(dst + e) = u;
        }
      }
    }
  }

  // ---------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    // a wait gave up: let copies and MMAs in flight land before TMEM and shared memory go
    const long long t0 = clock64();
    while (clock64() - t0 < 4000000LL) {
    }
    if (tid == 0) set_status(status, kKv ? kStatusTimeoutBwdDkv : kStatusTimeoutBwdDq);
    __syncthreads();
  }
  if (warp == 9) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

template <typename T, bool kKv>
cudaError_t launch(const BwdArgs& a, cudaStream_t stream) {
  const Dims& dm = a.dm;
  const bool bf16 = std::is_same<T, __nv_bfloat16>::value;
  const uint64_t eb = 2, n = dm.n, np = dm.n_pad, rows = dm.n_rows, heads = dm.heads, batch = dm.batch;
  const uint64_t dims5[5] = {(uint64_t)kD, n, rows, heads, batch};
  auto map5 = [&](CUtensorMap* m, const View5& v, uint32_t box_rows) {
    const uint32_t box[5] = {64, box_rows, 1, 1, 1};
    const uint64_t st[4] = {(uint64_t)v.sj * eb, (uint64_t)v.si * eb, (uint64_t)v.sh * eb, (uint64_t)v.sb * eb};
    return make_tensor_map(m, bf16, 5, v.p, dims5, st, box, CU_TENSOR_MAP_SWIZZLE_128B);
  };
  CUtensorMap a1, a2, b1, b2, mb, mnl, mdl;
  if (!map5(&a1, kKv ? a.k : a.q, 128) || !map5(&a2, kKv ? a.v : a.d_o, 128) ||
      !map5(&b1, kKv ? a.q : a.k, kStep) || !map5(&b2, kKv ? a.d_o : a.v, kStep))
    return cudaErrorInvalidValue;
  {   // the bias itself when its rows are 16-byte pitched, else the padded copy
    const uint64_t dims4[4] = {n, n, heads, batch};
    const uint64_t st_user[3] = {(uint64_t)a.bias.sj * eb, (uint64_t)a.bias.sh * eb, (uint64_t)a.bias.sb * eb};
    const uint64_t st_pad[3] = {np * eb, n * np * eb, n * np * heads * eb};
    const uint32_t box_kv[4] = {128, kStep, 1, 1}, box_q[4] = {kStep, 128, 1, 1};
    if (!make_tensor_map(&mb, bf16, 4, a.bias_pad ? a.bias_pad : (void*)a.bias.p, dims4,
                         a.bias_pad ? st_pad : st_user, kKv ? box_kv : box_q,
                         kKv ? CU_TENSOR_MAP_SWIZZLE_NONE : CU_TENSOR_MAP_SWIZZLE_128B))
      return cudaErrorInvalidValue;
  }
  {   // -lse log2e and delta: (b, h, rows, n_pad) fp32, made by the prepare step
    const uint64_t dims4[4] = {n, rows, heads, batch};
    const uint64_t st[3] = {np * 4, np * rows * 4, np * rows * heads * 4};
    const uint32_t box4[4] = {kStep, 1, 1, 1};
    if (!make_tensor_map_f32(&mnl, 4, a.neg_lse2, dims4, st, box4) ||
        !make_tensor_map_f32(&mdl, 4, a.delta, dims4, st, box4))
      return cudaErrorInvalidValue;
  }
  constexpr auto kern = tc_bwd_d128_kernel<T, kKv>;
  cudaError_t e = opt_in_smem<kern>(kSmemBytes);
  if (e != cudaSuccess) return e;
  Grid grid;
  grid.tiles = (dm.n + 127) / 128;
  grid.steps = (dm.n + kStep - 1) / kStep;
  grid.total = grid.tiles * dm.n_rows * dm.heads * dm.batch;
  const int sms = sm_count() - a.reserve_sms > 0 ? sm_count() - a.reserve_sms : 1;
  return launch_early(
      kern, grid.total < sms ? grid.total : sms, 384, kSmemBytes, stream,
      a1, a2, b1, b2, mb, mnl, mdl, kKv ? a.dk : a.dq, kKv ? a.dv : a.dq, a.neg_lse2, a.delta, a.ds_up,
      a.rowfull, a.maskbits_lin, a.mask_words, a.rowrange, dm, grid, a.status);
}

}  // namespace

bool tc_bwd_d128_supported(const BwdArgs& a) {
  if (a.dtype != TRIFAST_BF16 && a.dtype != TRIFAST_F16) return false;
  if (a.dm.d != kD || a.dm.n < kMinTensorCoreN) return false;
  if (!a.neg_lse2 || !a.maskbits_lin || !a.rowrange) return false;
  // without the padded copy the bias goes through TMA as it is
  if (!a.bias_pad && (a.dm.n % 8 != 0 || !bias_fits_tma(a.bias, a.dm))) return false;
  return get_encode_tiled() != nullptr;
}

cudaError_t tc_bwd_d128_dq(const BwdArgs& a, cudaStream_t s) {
  return a.dtype == TRIFAST_BF16 ? launch<__nv_bfloat16, false>(a, s) : launch<__half, false>(a, s);
}
cudaError_t tc_bwd_d128_dkv(const BwdArgs& a, cudaStream_t s) {
  return a.dtype == TRIFAST_BF16 ? launch<__nv_bfloat16, true>(a, s) : launch<__half, true>(a, s);
}

}  // namespace trifast
