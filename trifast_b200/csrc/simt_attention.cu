// CUDA-core triangle attention: fp32 arithmetic throughout, every dtype, every n (ragged
// included), d in {16, 32, 64, 128}.  Serves the fp32 contract and the shapes the tcgen05
// kernels do not take.
//
// One scheme for the three row kernels.  A CTA of 128 threads owns one pair row's tile of
// RESIDENT rows (queries in the forward and dq, keys in dk/dv) and walks the row's other side
// in tiles of STREAMED rows (32 or 64), both staged in shared memory as fp32.  A thread owns R
// resident rows and every eighth streamed row: it evaluates their scores, keeps the weights in
// registers and adds to its own accumulators, R rows of DL = 16 (d = 128: 32) elements; G = d / DL
// neighbouring lanes share the elements of a row and sum their partial products by shuffles.
// The eight streams of a resident row are only merged once, at the end: no weight goes
// through shared memory and no barrier separates the two products.
//
// What bounds it: shared-memory reads (ncu, n = 256: their pipe 60 % busy, the FMA pipe 45 %) and
// with 8 to 12 warps per SM, all that the accumulators leave room for, their latency.  Both
// operands of a packed FMA (fma.rn.f32x2, two head dims) come from 16-byte reads as they are.
// Row pitches of d + 4 G floats keep the eight rows (or the G parts of fewer rows) of a
// quarter-warp on different banks.  Tried and slower: the queries in registers (fewer reads,
// one CTA per SM less: 369 -> 430 us), 8 x 4 scores per thread in db (443 -> 567 us), three
// CTAs per SM by spilling (dk/dv 718 -> 805 us).  Measured at n = 256, h = 4, d = 32, fp32:
// forward 369 us, dq 597, dk/dv 718, db 443, where one thread per row with every operand from
// shared memory took 704, 717, 1100 and 764.
//
// db: a CTA owns a (j, k) tile of one (b, h) and a block of pair rows and sums dS in
// registers; fixed order, no atomics.
//
// Semantics follow the reference's PyTorch path (src/trifast/equiv.py:42-69): masked keys
// weigh exactly 0; a row whose keys are all masked gets uniform weights 1/n in the forward
// and in the backward.

#include <math.h>

#include <type_traits>

#include "kernels.h"

namespace trifast {
namespace {

constexpr float kMaxInit = -1e30f;  // finite start of the running max: exp(-inf - m) stays 0, never NaN
// The forward's running reference of a row moves only when a score exceeds it by more than
// this: weights then reach e^8 instead of 1, which fp32 holds at the same relative precision,
// and the accumulators are rescaled for the first keys of a row only.
constexpr float kLazyTau = 8.f;
constexpr int kThreads = 128, kStreams = 8;

__device__ __forceinline__ float2 ffma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n\t.reg .b64 ra, rb, rc, rd;\n\t"
      "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tmov.b64 rc, {%6, %7};\n\t"
      "fma.rn.f32x2 rd, ra, rb, rc;\n\t"
      "mov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 lo2(const float4& v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(const float4& v) { return make_float2(v.z, v.w); }

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
// 16 or 4 bytes global -> shared, or zeros when !valid
template <int kBytes>
__device__ __forceinline__ void cp_async(uint32_t dst, const void* src, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(kBytes),
               "r"(valid ? kBytes : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Four consecutive elements as fp32 (T* 16-byte rows: the address is a multiple of 4 elements).
template <typename T> __device__ __forceinline__ float4 load4(const T* p);
template <> __device__ __forceinline__ float4 load4<float>(const float* p) {
  return *reinterpret_cast<const float4*>(p);
}
template <typename T> __device__ __forceinline__ float4 load4(const T* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  const T* e = reinterpret_cast<const T*>(&u);
  return make_float4(to_f32<T>(e[0]), to_f32<T>(e[1]), to_f32<T>(e[2]), to_f32<T>(e[3]));
}
template <typename T> __device__ __forceinline__ void store4(T* p, float4 v);
template <> __device__ __forceinline__ void store4<float>(float* p, float4 v) {
  *reinterpret_cast<float4*>(p) = v;
}
template <typename T> __device__ __forceinline__ void store4(T* p, float4 v) {
  const T e[4] = {from_f32<T>(v.x), from_f32<T>(v.y), from_f32<T>(v.z), from_f32<T>(v.w)};
  *reinterpret_cast<uint2*>(p) = *reinterpret_cast<const uint2*>(e);
}

// ROWS rows of D elements starting at `src` (row stride `stride`), rows from `valid` on as
// zeros, into shared memory with pitch P: asynchronously when T is fp32, else converted.
template <typename T, int D, int P, int ROWS, int NT>
__device__ __forceinline__ void stage_rows(float* dst, const T* src, int64_t stride, int valid) {
  static_assert(ROWS * D / 4 % NT == 0 || ROWS * D / 4 < NT, "whole passes");
#pragma unroll 1   // (unrolled, every copy's addresses stay live through the caller's loop)
  for (int it = 0; it < (ROWS * D / 4 + NT - 1) / NT; ++it) {
    const int idx = it * NT + threadIdx.x, r = idx / (D / 4), c = idx % (D / 4) * 4;
    if (ROWS * D / 4 < NT && r >= ROWS) break;
    const bool ok = r < valid;
    const T* p = src + (ok ? r : 0) * stride + c;
    if constexpr (std::is_same<T, float>::value) {
      cp_async<16>(smem_addr(dst + r * P + c), p, ok);
    } else {
      *reinterpret_cast<float4*>(dst + r * P + c) = ok ? load4<T>(p) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
}

// ROWS x COLS values of a matrix (a bias tile), zeros outside valid_r x valid_c.  `wide`: its
// columns are contiguous and its rows allow 16-byte accesses.
template <typename T, int P, int ROWS, int COLS, int NT>
__device__ __forceinline__ void stage_matrix(float* dst, const T* src, int64_t stride, int64_t stride_c,
                                             int valid_r, int valid_c, bool wide) {
  if constexpr (std::is_same<T, float>::value) {
    if (wide) {
#pragma unroll 1
      for (int idx = threadIdx.x; idx < ROWS * COLS / 4; idx += NT) {
        const int r = idx / (COLS / 4), c = idx % (COLS / 4) * 4;
        const bool ok = r < valid_r && c < valid_c;   // valid_c is a multiple of 4 with wide rows
        cp_async<16>(smem_addr(dst + r * P + c), src + (ok ? r * stride + c : 0), ok);
      }
      return;
    }
  }
#pragma unroll 1
  for (int idx = threadIdx.x; idx < ROWS * COLS; idx += NT) {
    const int r = idx / COLS, c = idx % COLS;
    const bool ok = r < valid_r && c < valid_c;
    if constexpr (std::is_same<T, float>::value)
      cp_async<4>(smem_addr(dst + r * P + c), src + (ok ? r * stride + c * stride_c : 0), ok);
    else
      dst[r * P + c] = ok ? to_f32<T>(src[r * stride + c * stride_c]) : 0.f;
  }
}

template <int D, int R>
struct Cfg {
  static constexpr int DL = D < 128 ? 16 : 32;           // elements of a row per lane
  static constexpr int G = D / DL;                       // lanes that share a row
  static_assert(G * kStreams <= 32, "a row's lanes are in one warp");
  static constexpr int Q = DL / 4;                       // 16-byte chunks per lane: p, p + G, ...
  static constexpr int P = D + 4 * G;                    // row pitch (floats)
  static constexpr int TY = kThreads / (kStreams * G);   // groups of lanes: group y owns rows y, y + TY, ...
  static constexpr int BR = TY * R;                      // resident rows of a CTA
  static constexpr int TS = D <= 32 ? 64 : 32;           // streamed rows of a tile
  static constexpr int C = 4;                            // streamed rows of a thread at a time
};

// Shared-memory reads stay behind this point: the unrolled products below would otherwise be
// scheduled with all their reads first, hundreds of registers' worth.
__device__ __forceinline__ void hold_loads() { asm volatile("" ::: "memory"); }

// Sum over the G lanes that share a row.
template <int G> __device__ __forceinline__ float sum_parts(float x) {
#pragma unroll
  for (int o = 1; o < G; o <<= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// s[r][c] = resident row r . streamed row c, over this lane's chunks, then summed over parts
template <int D, int R, int C>
__device__ __forceinline__ void dots(const float* res, const float* str, float (&s)[R][C]) {
  using F = Cfg<D, R>;
  float2 acc[R][C];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int c = 0; c < C; ++c) acc[r][c] = make_float2(0.f, 0.f);
#pragma unroll
  for (int q = 0; q < F::Q; ++q) {
    if (q % 2 == 0) hold_loads();
    float4 a[R];
#pragma unroll
    for (int r = 0; r < R; ++r)
      a[r] = *reinterpret_cast<const float4*>(res + r * F::TY * F::P + q * F::G * 4);
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const float4 b = *reinterpret_cast<const float4*>(str + c * kStreams * F::P + q * F::G * 4);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        acc[r][c] = ffma2(lo2(a[r]), lo2(b), acc[r][c]);
        acc[r][c] = ffma2(hi2(a[r]), hi2(b), acc[r][c]);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int c = 0; c < C; ++c) s[r][c] = sum_parts<F::G>(acc[r][c].x + acc[r][c].y);
}

// acc[r] += sum_c w[r][c] * streamed row c, this lane's chunks
template <int D, int R, int C>
__device__ __forceinline__ void accumulate(const float (&w)[R][C], const float* str,
                                           float2 (&acc)[R][Cfg<D, R>::Q * 2]) {
  using F = Cfg<D, R>;
#pragma unroll
  for (int c = 0; c < C; ++c) {
    hold_loads();
#pragma unroll
    for (int q = 0; q < F::Q; ++q) {
      const float4 b = *reinterpret_cast<const float4*>(str + c * kStreams * F::P + q * F::G * 4);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float2 ww = make_float2(w[r][c], w[r][c]);
        acc[r][2 * q] = ffma2(ww, lo2(b), acc[r][2 * q]);
        acc[r][2 * q + 1] = ffma2(ww, hi2(b), acc[r][2 * q + 1]);
      }
    }
  }
}

// Sum over the eight streams (lanes G, 2G, 4G apart).
template <int G> __device__ __forceinline__ float sum_streams(float x) {
#pragma unroll
  for (int o = G; o < kStreams * G; o <<= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// Merges the eight streams of one resident row (every lane ends with the sum) and stores it,
// scaled: stream x writes chunks x, x + 8, ...
template <typename T, int D, int R>
__device__ __forceinline__ void store_row(float2 (&acc)[Cfg<D, R>::Q * 2], float scale, T* dst, int stream,
                                          int part, bool valid) {
  using F = Cfg<D, R>;
#pragma unroll
  for (int q = 0; q < F::Q; ++q) {
    const float4 v = make_float4(sum_streams<F::G>(acc[2 * q].x) * scale, sum_streams<F::G>(acc[2 * q].y) * scale,
                                 sum_streams<F::G>(acc[2 * q + 1].x) * scale,
                                 sum_streams<F::G>(acc[2 * q + 1].y) * scale);
    if (valid && stream == q % kStreams) store4<T>(dst + (q * F::G + part) * 4, v);
  }
}

template <typename T, int D, int R>
__device__ __forceinline__ void zero_row(T* dst, int stream, int part) {
  using F = Cfg<D, R>;
#pragma unroll
  for (int q = 0; q < F::Q; ++q)
    if (stream == q % kStreams) store4<T>(dst + (q * F::G + part) * 4, make_float4(0.f, 0.f, 0.f, 0.f));
}

// Where a thread stands: lane part p of its rows, stream x, group y.
template <int D, int R> struct Place {
  int p, x, y;
  __device__ __forceinline__ Place()
      : p(threadIdx.x % Cfg<D, R>::G), x(threadIdx.x / Cfg<D, R>::G % kStreams),
        y(threadIdx.x / (Cfg<D, R>::G * kStreams)) {}
};

template <typename T>
__device__ __forceinline__ T* row_ptr(const View5& t, int b, int h, int i, int j) {
  return reinterpret_cast<T*>(t.p) + b * t.sb + h * t.sh + (int64_t)i * t.si + (int64_t)j * t.sj;
}
template <typename T>
__device__ __forceinline__ const T* bias_ptr(const View4& t, int b, int h, int j) {
  return reinterpret_cast<const T*>(t.p) + b * t.sb + h * t.sh + (int64_t)j * t.sj;
}
template <typename T>
__device__ __forceinline__ bool wide_bias(const View4& t, int n) {
  return std::is_same<T, float>::value && t.sk == 1 && n % 4 == 0 && t.sj % 4 == 0 && t.sh % 4 == 0 && t.sb % 4 == 0 &&
         (reinterpret_cast<uintptr_t>(t.p) & 15) == 0;
}

// The tiles of the streamed side: fp32 inputs are copied asynchronously, one tile ahead into
// the other of two buffers; 16-bit inputs are converted on the way, into one buffer.
template <typename T, typename Stage, typename Work>
__device__ __forceinline__ void stream_tiles(int tiles, Stage stage, Work work) {
  if constexpr (std::is_same<T, float>::value) {
    stage(0, 0);
    cp_async_commit();
    for (int t = 0; t < tiles; ++t) {
      if (t + 1 < tiles) {
        stage(t + 1, (t + 1) & 1);
        cp_async_commit();
        cp_async_wait<1>();
      } else {
        cp_async_wait<0>();
      }
      __syncthreads();
      work(t, t & 1);
      __syncthreads();
    }
  } else {
    for (int t = 0; t < tiles; ++t) {
      stage(t, 0);
      __syncthreads();
      work(t, 0);
      __syncthreads();
    }
  }
}
template <typename T> constexpr int buffers() { return std::is_same<T, float>::value ? 2 : 1; }

// ------------------------------------------------------------------ forward
template <int D, int R> struct FwdSmem {
  using F = Cfg<D, R>;
  static constexpr int kBiasP = F::TS + 8;               // groups of a warp on different banks
  static constexpr int kRes = F::BR * F::P, kStr = F::TS * F::P, kBias = F::BR * kBiasP;
  static constexpr int kBuf = 2 * kStr + kBias + F::TS;  // K, V, bias, key flags
  template <typename T> static constexpr int bytes() { return (kRes + buffers<T>() * kBuf) * 4; }
};

template <typename T, int D, int R>
__global__ void __launch_bounds__(kThreads) simt_fwd_kernel(View5 q, View5 k, View5 v, View4 bias,
                                                            MaskView mask, View5 o, float* lse, Dims dm) {
  using F = Cfg<D, R>;
  using S = FwdSmem<D, R>;
  extern __shared__ __align__(16) float sm[];
  after_previous();
  const int n = dm.n, i = blockIdx.y, b = blockIdx.z / dm.heads, h = blockIdx.z % dm.heads;
  const int j0 = blockIdx.x * F::BR;
  const Place<D, R> at;
  const uint8_t* mrow = mask.p + b * mask.sb + (int64_t)i * mask.si;
  int open = 0;
  for (int c = threadIdx.x; c < n; c += kThreads) open |= mrow[c * mask.sk] == 0;
  const bool row_full = !__syncthreads_or(open);
  const bool wide = wide_bias<T>(bias, n);

  stage_rows<T, D, F::P, F::BR, kThreads>(sm, row_ptr<const T>(q, b, h, i, j0), q.sj, n - j0);
  const float* res = sm + at.y * F::P + at.p * 4;

  float2 acc[R][F::Q * 2];
  float m[R], l[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    m[r] = kMaxInit;
    l[r] = 0.f;
#pragma unroll
    for (int e = 0; e < F::Q * 2; ++e) acc[r][e] = make_float2(0.f, 0.f);
  }

  auto buf = [&](int u) { return sm + S::kRes + u * S::kBuf; };
  auto stage = [&](int t, int u) {
    const int k0 = t * F::TS, valid = n - k0;
    float* d = buf(u);
    stage_rows<T, D, F::P, F::TS, kThreads>(d, row_ptr<const T>(k, b, h, i, k0), k.sj, valid);
    stage_rows<T, D, F::P, F::TS, kThreads>(d + S::kStr, row_ptr<const T>(v, b, h, i, k0), v.sj, valid);
    stage_matrix<T, S::kBiasP, F::BR, F::TS, kThreads>(d + 2 * S::kStr, bias_ptr<T>(bias, b, h, j0) + k0 * bias.sk,
                                                       bias.sj, bias.sk, n - j0, valid, wide);
    if (threadIdx.x < F::TS) {
      const int c = threadIdx.x;
      d[2 * S::kStr + S::kBias + c] = (c < valid && (row_full || mrow[(k0 + c) * mask.sk] == 0)) ? 1.f : 0.f;
    }
  };
  auto work = [&](int, int u) {
    const float* d = buf(u);
    const float* bs = d + 2 * S::kStr + at.y * S::kBiasP + at.x;
    const float* keep = d + 2 * S::kStr + S::kBias + at.x;
#pragma unroll 1
    for (int c0 = 0; c0 < F::TS / kStreams; c0 += F::C) {
      const float* ks = d + (at.x + c0 * kStreams) * F::P + at.p * 4;
      float w[R][F::C];
      dots<D, R, F::C>(res, ks, w);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        float mt = -INFINITY;
#pragma unroll
        for (int c = 0; c < F::C; ++c) {
          const float bv = bs[r * F::TY * S::kBiasP + (c0 + c) * kStreams];
          float x = row_full ? 0.f : fmaf(w[r][c], dm.scale, bv);
          x = keep[(c0 + c) * kStreams] != 0.f ? x : -INFINITY;
          w[r][c] = x;
          mt = fmaxf(mt, x);
        }
        if (mt > m[r] + kLazyTau) {
          const float alpha = expf(m[r] - mt);
          m[r] = mt;
          l[r] *= alpha;
#pragma unroll
          for (int e = 0; e < F::Q * 2; ++e) {
            acc[r][e].x *= alpha;
            acc[r][e].y *= alpha;
          }
        }
#pragma unroll
        for (int c = 0; c < F::C; ++c) {
          w[r][c] = expf(w[r][c] - m[r]);
          l[r] += w[r][c];
        }
      }
      accumulate<D, R, F::C>(w, ks + S::kStr, acc);
    }
  };
  stream_tiles<T>((n + F::TS - 1) / F::TS, stage, work);

#pragma unroll
  for (int r = 0; r < R; ++r) {
    // the eight streams' references, sums and accumulators become one
    float mm = m[r];
#pragma unroll
    for (int s = F::G; s < kStreams * F::G; s <<= 1) mm = fmaxf(mm, __shfl_xor_sync(0xffffffffu, mm, s));
    const float f = expf(m[r] - mm);
    const float ll = sum_streams<F::G>(l[r] * f);
#pragma unroll
    for (int e = 0; e < F::Q * 2; ++e) {
      acc[r][e].x *= f;
      acc[r][e].y *= f;
    }
    const int j = j0 + at.y + r * F::TY;
    store_row<T, D, R>(acc[r], 1.f / ll, row_ptr<T>(o, b, h, i, min(j, n - 1)), at.x, at.p, j < n);
    if (j < n && at.x == 0 && at.p == 0)
      lse[(((int64_t)b * dm.heads + h) * dm.n_rows + i) * n + j] = row_full ? dm.sentinel : mm + logf(ll);
  }
}

// ------------------------------------------------------------------ dq, and dk / dv
// Resident A1, A2 and streamed B1, B2: (Q, dO; K, V) for dq, (K, V; Q, dO) for dk/dv.
template <int D, int R, bool kKv> struct BwdSmem {
  using F = Cfg<D, R>;
  // the bias tile keeps its orientation, queries x keys
  static constexpr int kBiasP = kKv ? F::BR + 4 : F::TS + 8;
  static constexpr int kRes = F::BR * F::P, kStr = F::TS * F::P, kBias = (kKv ? F::TS : F::BR) * kBiasP;
  static constexpr int kBuf = 2 * kStr + kBias + 2 * F::TS;  // B1, B2, bias, lse, delta
  template <typename T> static constexpr int bytes() { return (2 * kRes + buffers<T>() * kBuf) * 4; }
};

template <typename T, int D, int R, bool kKv>
__global__ void __launch_bounds__(kThreads) simt_bwd_kernel(View5 a1, View5 a2, View5 b1, View5 b2, View4 bias,
                                                            View5 out1, View5 out2, const float* lse,
                                                            const float* delta, const uint8_t* rowfull,
                                                            const uint32_t* maskbits_lin, int mask_words,
                                                            Dims dm) {
  using F = Cfg<D, R>;
  using S = BwdSmem<D, R, kKv>;
  extern __shared__ __align__(16) float sm[];
  after_previous();
  const int n = dm.n, i = blockIdx.y, b = blockIdx.z / dm.heads, h = blockIdx.z % dm.heads;
  const int r0 = blockIdx.x * F::BR;
  const Place<D, R> at;
  const bool row_full = rowfull[b * dm.n_rows + i] != 0, wide = wide_bias<T>(bias, n);
  const float uniform = 1.f / (float)n;
  // bit set = key dropped or beyond n (on a fully masked row only beyond n)
  const uint32_t* mwords = maskbits_lin + ((int64_t)b * dm.n_rows + i) * mask_words;
  const int64_t row = ((int64_t)b * dm.heads + h) * dm.n_rows + i;
  const float* lse_row = lse + row * n;
  const float* delta_row = delta + row * dm.n_pad;

  stage_rows<T, D, F::P, F::BR, kThreads>(sm, row_ptr<const T>(a1, b, h, i, r0), a1.sj, n - r0);
  stage_rows<T, D, F::P, F::BR, kThreads>(sm + S::kRes, row_ptr<const T>(a2, b, h, i, r0), a2.sj, n - r0);
  const float* res = sm + at.y * F::P + at.p * 4;

  float2 acc1[R][F::Q * 2], acc2[R][kKv ? F::Q * 2 : 1];
  float lr[R], dr[R];      // dq: lse and delta of this thread's queries
  bool dropped[R];         // dk/dv: this thread's keys
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int a = r0 + at.y + r * F::TY, ac = min(a, n - 1);
    lr[r] = kKv ? 0.f : lse_row[ac];
    dr[r] = kKv ? 0.f : delta_row[ac];
    dropped[r] = kKv && (a >= n || ((mwords[ac >> 5] >> (ac & 31)) & 1u));
#pragma unroll
    for (int e = 0; e < F::Q * 2; ++e) {
      acc1[r][e] = make_float2(0.f, 0.f);
      if (kKv) acc2[r][e] = make_float2(0.f, 0.f);
    }
  }

  auto buf = [&](int u) { return sm + 2 * S::kRes + u * S::kBuf; };
  auto stage = [&](int t, int u) {
    const int s0 = t * F::TS, valid = n - s0;
    float* d = buf(u);
    stage_rows<T, D, F::P, F::TS, kThreads>(d, row_ptr<const T>(b1, b, h, i, s0), b1.sj, valid);
    stage_rows<T, D, F::P, F::TS, kThreads>(d + S::kStr, row_ptr<const T>(b2, b, h, i, s0), b2.sj, valid);
    if constexpr (kKv)
      stage_matrix<T, S::kBiasP, F::TS, F::BR, kThreads>(d + 2 * S::kStr, bias_ptr<T>(bias, b, h, s0) + r0 * bias.sk,
                                                         bias.sj, bias.sk, valid, n - r0, wide);
    else
      stage_matrix<T, S::kBiasP, F::BR, F::TS, kThreads>(d + 2 * S::kStr, bias_ptr<T>(bias, b, h, r0) + s0 * bias.sk,
                                                         bias.sj, bias.sk, n - r0, valid, wide);
    if (kKv && threadIdx.x < F::TS) {
      const int c = threadIdx.x, cc = min(s0 + c, n - 1);
      d[2 * S::kStr + S::kBias + c] = lse_row[cc];
      d[2 * S::kStr + S::kBias + F::TS + c] = delta_row[cc];
    }
  };
  auto work = [&](int t, int u) {
    const float* d = buf(u);
    const float* bs = d + 2 * S::kStr + (kKv ? at.x * S::kBiasP + at.y : at.y * S::kBiasP + at.x);
    const float* vec = d + 2 * S::kStr + S::kBias + at.x;
#pragma unroll 1
    for (int c0 = 0; c0 < F::TS / kStreams; c0 += F::C) {
      const float* str = d + (at.x + c0 * kStreams) * F::P + at.p * 4;
      float w[R][F::C], g[R][F::C];
      dots<D, R, F::C>(res, str, w);
      dots<D, R, F::C>(res + S::kRes, str + S::kStr, g);
#pragma unroll
      for (int c = 0; c < F::C; ++c) {
        const int key = t * F::TS + (c0 + c) * kStreams + at.x;   // the streamed row
        const bool out = kKv ? key >= n : ((mwords[key >> 5] >> (key & 31)) & 1u) != 0u;
        const float lc = kKv ? vec[(c0 + c) * kStreams] : 0.f;
        const float dc = kKv ? vec[F::TS + (c0 + c) * kStreams] : 0.f;
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const float bv = kKv ? bs[(c0 + c) * kStreams * S::kBiasP + r * F::TY]
                               : bs[r * F::TY * S::kBiasP + (c0 + c) * kStreams];
          float p = row_full ? uniform : expf(fmaf(w[r][c], dm.scale, bv) - (kKv ? lc : lr[r]));
          p = (out || dropped[r]) ? 0.f : p;
          w[r][c] = p;
          g[r][c] = p * (g[r][c] - (kKv ? dc : dr[r]));
        }
      }
      accumulate<D, R, F::C>(g, str, acc1);
      if constexpr (kKv) accumulate<D, R, F::C>(w, str + S::kStr, acc2);
    }
  };
  stream_tiles<T>((n + F::TS - 1) / F::TS, stage, work);

#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int a = r0 + at.y + r * F::TY, ac = min(a, n - 1);
    store_row<T, D, R>(acc1[r], dm.scale, row_ptr<T>(out1, b, h, i, ac), at.x, at.p, a < n);
    if constexpr (kKv) {
      store_row<T, D, R>(acc2[r], 1.f, row_ptr<T>(out2, b, h, i, ac), at.x, at.p, a < n);
      // a dropped key gets exactly zero, also where a query's dO, lse or delta is not finite: the
      // lanes that stored its row overwrite it (a select on the way costs the other rows 1 %)
      if (dropped[r] && a < n) {
        zero_row<T, D, R>(row_ptr<T>(out1, b, h, i, a), at.x, at.p);
        zero_row<T, D, R>(row_ptr<T>(out2, b, h, i, a), at.x, at.p);
      }
    }
  }
}

// ------------------------------------------------------------------ db
// Thread (y, x) of TY x TX owns queries y + TY a and keys x + TX c, EA x EC of them.  A warp is 4
// groups y by 8 keys x, which keeps its 16-byte reads on different banks.  The head dim is
// walked in chunks of DC.
template <typename T, int D, int EA, int EC, int TILE_> struct DbSmem {
  static constexpr int DC = D < 32 ? D : 32, P = DC + 4, TILE = TILE_;
  static constexpr int TY = TILE / EA, TX = TILE / EC, NT = TY * TX;
  static constexpr int kBuf = 4 * TILE * P + 2 * TILE;   // Q, dO, K, V, lse, delta
  static constexpr int kBytes = buffers<T>() * kBuf * 4;
};

template <typename T, int D, int EA, int EC, int TILE>
__global__ void __launch_bounds__(TILE / EA * (TILE / EC), 2) simt_db_kernel(View5 q, View5 k, View5 v, View4 bias, View5 d_o,
                                                      const float* lse, const float* delta,
                                                      const uint8_t* rowfull, const uint32_t* maskbits_lin,
                                                      int mask_words, float* out, int splits, Dims dm) {
  using S = DbSmem<T, D, EA, EC, TILE>;
  constexpr int NC = D / S::DC;
  extern __shared__ __align__(16) float sm[];
  after_previous();
  const int n = dm.n, tiles_k = (n + S::TILE - 1) / S::TILE;
  const int j0 = blockIdx.x / tiles_k * S::TILE, k0 = blockIdx.x % tiles_k * S::TILE;
  const int split = blockIdx.y, bh = blockIdx.z, b = bh / dm.heads, h = bh % dm.heads;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int y = warp / (S::TX / 8) * 4 + (lane >> 3), x = warp % (S::TX / 8) * 8 + (lane & 7);
  const float uniform = 1.f / (float)n;
  // rows of a split: a contiguous block, the same partition for every tile
  const int per = (dm.n_rows + splits - 1) / splits;
  const int i0 = split * per, rows = max(0, min(dm.n_rows, i0 + per) - i0);

  float bv[EA][EC], acc[EA][EC];
#pragma unroll
  for (int a = 0; a < EA; ++a)
#pragma unroll
    for (int c = 0; c < EC; ++c) {
      const int j = j0 + y + S::TY * a, key = k0 + x + S::TX * c;
      bv[a][c] = (j < n && key < n) ? to_f32<T>(bias_ptr<T>(bias, b, h, j)[key * bias.sk]) : 0.f;
      acc[a][c] = 0.f;
    }
  auto buf = [&](int u) { return sm + u * S::kBuf; };
  auto stage = [&](int t, int u) {   // step t: row t / NC, chunk t % NC
    const int i = i0 + t / NC, c0 = t % NC * S::DC;
    float* d = buf(u);
    constexpr int kT = S::TILE * S::P;
    stage_rows<T, S::DC, S::P, S::TILE, S::NT>(d, row_ptr<const T>(q, b, h, i, j0) + c0, q.sj, n - j0);
    stage_rows<T, S::DC, S::P, S::TILE, S::NT>(d + kT, row_ptr<const T>(d_o, b, h, i, j0) + c0, d_o.sj, n - j0);
    stage_rows<T, S::DC, S::P, S::TILE, S::NT>(d + 2 * kT, row_ptr<const T>(k, b, h, i, k0) + c0, k.sj, n - k0);
    stage_rows<T, S::DC, S::P, S::TILE, S::NT>(d + 3 * kT, row_ptr<const T>(v, b, h, i, k0) + c0, v.sj, n - k0);
    if (threadIdx.x < S::TILE) {
      const int64_t row = ((int64_t)b * dm.heads + h) * dm.n_rows + i;
      const int j = min(j0 + (int)threadIdx.x, n - 1);
      d[4 * kT + threadIdx.x] = lse[row * n + j];
      d[4 * kT + S::TILE + threadIdx.x] = delta[row * dm.n_pad + j];
    }
  };
  float2 s2[EA][EC], g2[EA][EC];
  auto work = [&](int t, int u) {
    constexpr int kT = S::TILE * S::P;
    const float* d = buf(u);
    if (t % NC == 0) {
#pragma unroll
      for (int a = 0; a < EA; ++a)
#pragma unroll
        for (int c = 0; c < EC; ++c) s2[a][c] = g2[a][c] = make_float2(0.f, 0.f);
    }
    auto mul = [&](const float* rows_, const float* cols, float2 (&sum)[EA][EC]) {
#pragma unroll
      for (int e = 0; e < S::DC; e += 4) {
        hold_loads();
        float4 l4[EA];
#pragma unroll
        for (int a = 0; a < EA; ++a) l4[a] = *reinterpret_cast<const float4*>(rows_ + (y + S::TY * a) * S::P + e);
#pragma unroll
        for (int c = 0; c < EC; ++c) {
          const float4 r4 = *reinterpret_cast<const float4*>(cols + (x + S::TX * c) * S::P + e);
#pragma unroll
          for (int a = 0; a < EA; ++a) {
            sum[a][c] = ffma2(lo2(l4[a]), lo2(r4), sum[a][c]);
            sum[a][c] = ffma2(hi2(l4[a]), hi2(r4), sum[a][c]);
          }
        }
      }
    };
    mul(d, d + 2 * kT, s2);
    mul(d + kT, d + 3 * kT, g2);
    if (t % NC != NC - 1) return;
    const int i = i0 + t / NC;
    const bool row_full = rowfull[b * dm.n_rows + i] != 0;
    const uint32_t* mwords = maskbits_lin + ((int64_t)b * dm.n_rows + i) * mask_words;
#pragma unroll
    for (int c = 0; c < EC; ++c) {
      const int key = k0 + x + S::TX * c;
      const bool dropped = (__ldg(mwords + (key >> 5)) >> (key & 31)) & 1u;
#pragma unroll
      for (int a = 0; a < EA; ++a) {
        const float ls = d[4 * kT + y + S::TY * a], dl = d[4 * kT + S::TILE + y + S::TY * a];
        float p = row_full ? uniform : expf(fmaf(s2[a][c].x + s2[a][c].y, dm.scale, bv[a][c]) - ls);
        p = dropped ? 0.f : p;
        acc[a][c] = fmaf(p, (g2[a][c].x + g2[a][c].y) - dl, acc[a][c]);
      }
    }
  };
  if (rows > 0) stream_tiles<T>(rows * NC, stage, work);
  float* dst = out + ((int64_t)split * dm.batch * dm.heads + bh) * n * n;
#pragma unroll
  for (int a = 0; a < EA; ++a)
#pragma unroll
    for (int c = 0; c < EC; ++c) {
      const int j = j0 + y + S::TY * a, key = k0 + x + S::TX * c;
      if (j < n && key < n) dst[(int64_t)j * n + key] = acc[a][c];
    }
}

// ------------------------------------------------------------------ dispatch on (dtype, d)
template <typename F>
cudaError_t dispatch(int dtype, int d, F&& f) {
  auto on_d = [&](auto* tp) -> cudaError_t {
    switch (d) {
      case 16: return f(tp, std::integral_constant<int, 16>{});
      case 32: return f(tp, std::integral_constant<int, 32>{});
      case 64: return f(tp, std::integral_constant<int, 64>{});
      case 128: return f(tp, std::integral_constant<int, 128>{});
      default: return cudaErrorInvalidValue;
    }
  };
  switch (dtype) {
    case TRIFAST_F32: return on_d((float*)nullptr);
    case TRIFAST_BF16: return on_d((__nv_bfloat16*)nullptr);
    case TRIFAST_F16: return on_d((__half*)nullptr);
    default: return cudaErrorInvalidValue;
  }
}

template <typename T, int D, int R>
cudaError_t launch_fwd(const FwdArgs& a, cudaStream_t s) {
  const Dims& dm = a.dm;
  constexpr int kBytes = FwdSmem<D, R>::template bytes<T>();
  constexpr auto kern = simt_fwd_kernel<T, D, R>;
  if (cudaError_t e = opt_in_smem<kern>(kBytes)) return e;
  const dim3 grid((dm.n + Cfg<D, R>::BR - 1) / Cfg<D, R>::BR, dm.n_rows, dm.batch * dm.heads);
  return launch_early(kern, grid, kThreads, kBytes, s, a.q, a.k, a.v, a.bias, a.mask, a.o, a.lse, dm);
}

template <typename T, int D, int R, bool kKv>
cudaError_t launch_bwd(const BwdArgs& a, cudaStream_t s) {
  const Dims& dm = a.dm;
  constexpr int kBytes = BwdSmem<D, R, kKv>::template bytes<T>();
  constexpr auto kern = simt_bwd_kernel<T, D, R, kKv>;
  if (cudaError_t e = opt_in_smem<kern>(kBytes)) return e;
  const dim3 grid((dm.n + Cfg<D, R>::BR - 1) / Cfg<D, R>::BR, dm.n_rows, dm.batch * dm.heads);
  return launch_early(kern, grid, kThreads, kBytes, s, kKv ? a.k : a.q, kKv ? a.v : a.d_o, kKv ? a.q : a.k,
                      kKv ? a.d_o : a.v, a.bias, kKv ? a.dk : a.dq, kKv ? a.dv : a.dq, a.lse, a.delta, a.rowfull,
                      a.maskbits_lin, a.mask_words, dm);
}

template <typename T, int D, int EA, int EC, int TILE>
cudaError_t launch_db(const BwdArgs& a, cudaStream_t s) {
  using S = DbSmem<T, D, EA, EC, TILE>;
  const Dims& dm = a.dm;
  constexpr auto kern = simt_db_kernel<T, D, EA, EC, TILE>;
  if (cudaError_t e = opt_in_smem<kern>(S::kBytes)) return e;
  const int t = (dm.n + S::TILE - 1) / S::TILE;
  return launch_early(kern, dim3(t * t, a.splits, dm.batch * dm.heads), S::NT, S::kBytes, s, a.q, a.k, a.v, a.bias,
                      a.d_o, a.lse, a.delta, a.rowfull, a.maskbits_lin, a.mask_words,
                      a.splits > 1 ? a.db_partials : a.db_f32, a.splits, dm);
}

}  // namespace

// Rows of 64 resident queries need n > 32 to be half full (d <= 32; wider heads have smaller
// tiles already).
cudaError_t simt_forward(const FwdArgs& a, cudaStream_t s) {
  return dispatch(a.dtype, a.dm.d, [&](auto* tp, auto dc) {
    using T = std::remove_pointer_t<decltype(tp)>;
    constexpr int D = decltype(dc)::value;
    if constexpr (D <= 32)
      if (a.dm.n <= 32) return launch_fwd<T, D, 2>(a, s);
    return launch_fwd<T, D, 4>(a, s);
  });
}

cudaError_t simt_bwd_dq(const BwdArgs& a, cudaStream_t s) {
  return dispatch(a.dtype, a.dm.d, [&](auto* tp, auto dc) {
    using T = std::remove_pointer_t<decltype(tp)>;
    constexpr int D = decltype(dc)::value;
    if constexpr (D <= 32)
      if (a.dm.n <= 32) return launch_bwd<T, D, 2, false>(a, s);
    return launch_bwd<T, D, D < 128 ? 4 : 2, false>(a, s);
  });
}

cudaError_t simt_bwd_dkv(const BwdArgs& a, cudaStream_t s) {
  return dispatch(a.dtype, a.dm.d, [&](auto* tp, auto dc) {
    using T = std::remove_pointer_t<decltype(tp)>;
    constexpr int D = decltype(dc)::value;
    return launch_bwd<T, D, D < 128 ? 4 : 2, true>(a, s);
  });
}

// 64 x 64 tiles where they are at least half full.
cudaError_t simt_bwd_db(const BwdArgs& a, cudaStream_t s) {
  return dispatch(a.dtype, a.dm.d, [&](auto* tp, auto dc) {
    using T = std::remove_pointer_t<decltype(tp)>;
    constexpr int D = decltype(dc)::value;
    return a.dm.n <= 32 ? launch_db<T, D, 2, 2, 32>(a, s) : launch_db<T, D, 4, 4, 64>(a, s);
  });
}

}  // namespace trifast
