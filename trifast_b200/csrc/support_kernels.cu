// Small kernels around the attention kernels of both families: one prepare kernel per call
// (row flags, packed key masks, live key-tile ranges, bias copies, delta) and the sum of db's
// row splits with its cast.
//
// On small problems every launch counts (about 3 us of host time and 2 us of device time each):
// the parts of the prepare step are independent of one another, so they are block ranges of
// one launch, and the sum over row splits writes the gradient in its own type.

#include <math.h>

#include <type_traits>

#include "kernels.h"

namespace trifast {
namespace {

constexpr int kPrepThreads = 256;
constexpr float kLog2e = 1.4426950408889634f;

struct Prep {
  MaskView mask;
  View4 bias;
  uint8_t* rowfull;
  uint32_t *maskbits, *maskbits_lin, *rowrange;
  int mask_words;
  uint16_t *bias_t, *bias_pad;
  Dims dm;
  unsigned int* status;
  View5 v;
  float* ds_up;
  // forward at head dims up to 64: rows without an open key are finished here (o: the mean of
  // all values, lse: the sentinel) and their range of key tiles is empty
  View5 o;
  float* lse;
  int dtype;
  int fill_blocks;   // blocks per row, which share its heads
  // block ranges, in this order: one row of the mask each (or fill_blocks of them); 64 x 64 bias
  // tiles; one (b, h, i) of ds_up each; the rest delta
  int mask_blocks, bias_tiles, bias_blocks, scale_blocks;
};

// (volatile: the loads of a thread go out together, in this order)
__device__ __forceinline__ uint4 load_once(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}

// ---------------------------------------------------------------------------
// Output of a pair row (b, i) without an open key, `heads` heads from h0 on: the mean of its n values for
// every query, which the tensor-core kernel would spend a walk over all keys on.  A thread
// owns 16 bytes of a head's row and every so-manieth key, so that all heads' loads are in flight
// together (head after head the block took 25 us at n = 512, h = 4, so 11).  Sums in fp32.
// ---------------------------------------------------------------------------
__device__ void fill_masked_row(const Prep& a, int b, int i, int h0, int heads) {
  __shared__ float sums[8][kPrepThreads];
  const int n = a.dm.n, parts = a.dm.d / 8, columns = parts * heads;
  int wide = 1;   // columns of a pass, a power of two
  while (wide < columns && wide < kPrepThreads / 2) wide *= 2;
  const int rows = kPrepThreads / wide, first = threadIdx.x / wide;
  const bool bf16 = a.dtype == TRIFAST_BF16;
  for (int c0 = 0; c0 < columns; c0 += wide) {
    const int column = c0 + threadIdx.x % wide, h = h0 + column / parts, part = column % parts;
    const bool mine = column < columns;
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (mine) {
      const uint16_t* v = (const uint16_t*)a.v.p + b * a.v.sb + h * a.v.sh + (int64_t)i * a.v.si + part * 8;
      constexpr int U = 8;   // loads in flight
      for (int k0 = first; k0 < n; k0 += U * rows) {
        uint4 u[U];
#pragma unroll
        for (int c = 0; c < U; ++c) u[c] = load_once(v + (int64_t)min(k0 + c * rows, n - 1) * a.v.sj);
#pragma unroll
        for (int c = 0; c < U; ++c) {
          const uint32_t w[4] = {u[c].x, u[c].y, u[c].z, u[c].w};
          const bool in = k0 + c * rows < n;
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const uint16_t x = in ? (uint16_t)(w[e >> 1] >> (16 * (e & 1))) : (uint16_t)0;
            acc[e] += bf16 ? __uint_as_float((uint32_t)x << 16) : __half2float(__ushort_as_half(x));
          }
        }
      }
    }
    __syncthreads();   // (the previous pass's sums have been read)
#pragma unroll
    for (int e = 0; e < 8; ++e) sums[e][threadIdx.x] = acc[e];
    for (int half = kPrepThreads / 2; half >= wide; half >>= 1) {
      __syncthreads();
      if (threadIdx.x < half)
#pragma unroll
        for (int e = 0; e < 8; ++e) sums[e][threadIdx.x] += sums[e][threadIdx.x + half];
    }
    __syncthreads();
    if (!mine) continue;
    const float inv = 1.f / (float)n;
    const int at = threadIdx.x % wide;
    uint32_t w[4];
#pragma unroll
    for (int e = 0; e < 8; e += 2) {
      const float lo = sums[e][at] * inv, hi = sums[e + 1][at] * inv;
      w[e >> 1] = bf16 ? (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(lo)) |
                             (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(hi)) << 16
                       : (uint32_t)__half_as_ushort(__float2half_rn(lo)) |
                             (uint32_t)__half_as_ushort(__float2half_rn(hi)) << 16;
    }
    uint16_t* o = (uint16_t*)a.o.p + b * a.o.sb + h * a.o.sh + (int64_t)i * a.o.si + part * 8;
    for (int j = first; j < n; j += rows)
      *reinterpret_cast<uint4*>(o + (int64_t)j * a.o.sj) = make_uint4(w[0], w[1], w[2], w[3]);
  }
  for (int h = h0; h < h0 + heads; ++h) {
    float* lse = a.lse + (((int64_t)b * a.dm.heads + h) * a.dm.n_rows + i) * n;
    for (int j = threadIdx.x; j < n; j += kPrepThreads) lse[j] = a.dm.sentinel;
  }
}

// ---------------------------------------------------------------------------
// One pair row of the mask: rowfull = 1 when every key is masked, the packed key masks, the
// range of 128-key tiles that hold an open key.
// ---------------------------------------------------------------------------
// kFill: the forward's, which also finishes rows without an open key.  The backward's kernel is spared
// the registers and shared memory of that, 64 and 16.7 KB instead of 47 and 8.5 (d = 32); its time was the
// same with them (n = 1024, h = 4: 116 us).
template <bool kFill>
__device__ void prepare_mask_row(const Prep& a, int block) {
  const int n = a.dm.n, n_rows = a.dm.n_rows;
  const int bi = kFill ? block / a.fill_blocks : block, share = kFill ? block % a.fill_blocks : 0;
  const int b = bi / n_rows, i = bi % n_rows;
  const uint8_t* row = a.mask.p + b * a.mask.sb + (int64_t)i * a.mask.si;
  const int64_t sk = a.mask.sk;
  __shared__ int first_open, last_open, dropped_any;
  if (threadIdx.x == 0) {
    first_open = n;
    last_open = -1;
    dropped_any = 0;
  }
  __syncthreads();
  int lo = n, hi = -1;
  bool dropped = false;
  for (int k = threadIdx.x; k < n; k += kPrepThreads) {
    if (row[k * sk] == 0) {
      lo = min(lo, k);
      hi = max(hi, k);
    } else {
      dropped = true;
    }
  }
  if (dropped) dropped_any = 1;
  if (hi >= 0) {
    atomicMin(&first_open, lo);
    atomicMax(&last_open, hi);
  }
  __syncthreads();
  const int open = last_open >= 0;
  if (threadIdx.x == 0 && share == 0) {
    if (a.rowfull) a.rowfull[bi] = open ? 0 : 1;
    // 128-key tiles [first, last + 1) that hold an open key: the tensor-core kernels walk
    // only those.  A fully masked row weighs all n keys: every tile, or none where it is
    // finished here; there, the top bit says that no key is dropped.
    if (a.rowrange) {
      const uint32_t t0 = open ? (uint32_t)(first_open >> 7) : a.lse ? 0xffffu : 0u;
      const uint32_t t1 = open ? (uint32_t)(last_open >> 7) + 1u : a.lse ? 0u : (uint32_t)((n + 127) >> 7);
      a.rowrange[bi] = t0 | (t1 << 16) | (a.lse && !dropped_any ? 0x80000000u : 0u);
    }
  }
  if constexpr (kFill)
    if (!open && a.lse) {
      const int h0 = share * a.dm.heads / a.fill_blocks;
      fill_masked_row(a, b, i, h0, (share + 1) * a.dm.heads / a.fill_blocks - h0);
    }
  if (!a.maskbits || share > 0) return;
  // Packed key mask (bit set = key dropped or beyond n).  A fully masked row keeps
  // all n keys with uniform weight, so only the keys beyond n stay set.  Layout per
  // 128-key chunk c: word c*4 + jb holds, at bit l, key c*128 + 4*l + jb (the order
  // in which a warp reading four mask bytes per lane produces the words).
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int w = warp; w < a.mask_words; w += kPrepThreads / 32) {
    const int k = (w >> 2) * 128 + 4 * lane + (w & 3);
    const int dropped = (k < n) ? (open ? (row[k * sk] != 0) : 0) : 1;
    const unsigned bits = __ballot_sync(0xffffffffu, dropped);
    if (lane == 0) a.maskbits[(int64_t)bi * a.mask_words + w] = bits;
  }
  // The same bits in key order (word w, bit l: key 32 * w + l), when asked for.
  if (a.maskbits_lin) {
    for (int w = warp; w < a.mask_words; w += kPrepThreads / 32) {
      const int k = w * 32 + lane;
      const int dropped = (k < n) ? (open ? (row[k * sk] != 0) : 0) : 1;
      const unsigned bits = __ballot_sync(0xffffffffu, dropped);
      if (lane == 0) a.maskbits_lin[(int64_t)bi * a.mask_words + w] = bits;
    }
  }
}

// ---------------------------------------------------------------------------
// 64 x 64 tile of the bias (2-byte elements) into the copies asked for, both with row pitch
// n_pad (a multiple of 16 bytes, as TMA needs): bias_t[b, h, k, j] with keys on the rows, and
// bias_pad[b, h, j, k] where the bias itself cannot be described to TMA.  Elements of the pad
// columns are zero in bias_pad.
// ---------------------------------------------------------------------------
__device__ void prepare_bias_tile(const Prep& a, int w) {
  __shared__ uint16_t tile[64][66];
  const int n = a.dm.n, n_pad = a.dm.n_pad;
  const int k0 = w % a.bias_tiles * 64, j0 = w / a.bias_tiles % a.bias_tiles * 64;
  const int bh = w / (a.bias_tiles * a.bias_tiles), b = bh / a.dm.heads, h = bh % a.dm.heads;
  const View4& bias = a.bias;
  const uint16_t* src = (const uint16_t*)bias.p + b * bias.sb + h * bias.sh;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
  const bool pairs_in = bias.sk == 1 && (bias.sj % 2 == 0) && (bias.sh % 2 == 0) && (bias.sb % 2 == 0) &&
                        ((reinterpret_cast<uintptr_t>(bias.p) & 3) == 0);
#pragma unroll
  for (int it = 0; it < 8; ++it) {
    const int r = ty + 8 * it, j = j0 + r, k = k0 + 2 * tx;
    uint16_t e0 = 0, e1 = 0;
    if (j < n) {
      const uint16_t* p = src + (int64_t)j * bias.sj + (int64_t)k * bias.sk;
      if (pairs_in && k + 1 < n) {
        const uint32_t u = *reinterpret_cast<const uint32_t*>(p);
        e0 = (uint16_t)(u & 0xffffu);
        e1 = (uint16_t)(u >> 16);
      } else {
        if (k < n) e0 = p[0];
        if (k + 1 < n) e1 = p[bias.sk];
      }
    }
    if (a.bias_pad && j < n && k < n_pad)   // n_pad is even: a pair never straddles it
      *reinterpret_cast<uint32_t*>(a.bias_pad + ((int64_t)bh * n + j) * n_pad + k) =
          (uint32_t)e0 | ((uint32_t)e1 << 16);
    tile[r][2 * tx] = e0;
    tile[r][2 * tx + 1] = e1;
  }
  if (!a.bias_t) return;
  __syncthreads();
  uint16_t* dst = a.bias_t + (int64_t)bh * n * n_pad;
#pragma unroll
  for (int it = 0; it < 8; ++it) {  // output row k0 + r holds queries j0 .. j0 + 63
    const int r = ty + 8 * it, k = k0 + r, j = j0 + 2 * tx;
    if (k < n && j < n_pad) {
      const uint32_t u = (uint32_t)tile[2 * tx][r] | ((uint32_t)tile[2 * tx + 1][r] << 16);
      *reinterpret_cast<uint32_t*>(dst + (int64_t)k * n_pad + j) = u;
    }
  }
}

// ---------------------------------------------------------------------------
// delta[b, h, i, j] = sum_d o * dO (fp32; never rounded to the input dtype) and
// neg_lse2 = -lse * log2(e), row pitch n_pad.
// ---------------------------------------------------------------------------
// A group of G threads owns a (b, h, i, j) row of D elements, 16 bytes per thread and step, so
// that a warp reads whole 128-byte lines of o and dO; U rows per thread keep several loads in
// flight (one row at a time read 3.5 TB/s of the 6.5 a copy reaches).
template <typename T, int D> struct DeltaCfg {
  static constexpr int kVec = 16 / sizeof(T);   // elements per 16-byte load
  static constexpr int G = (D / kVec) < 4 ? (D / kVec) : 4;
  static constexpr int kSteps = D / (kVec * G);
  static constexpr int U = kSteps == 1 ? 4 : kSteps == 2 ? 2 : 1;
  static constexpr int kRows = kPrepThreads / G * U;   // rows of a block
};

template <typename T, int D>
__device__ void prepare_delta(const View5& o, const View5& d_o, const float* lse, float* delta,
                              float* neg_lse2, const Dims& dm, unsigned block) {
  using C = DeltaCfg<T, D>;
  const unsigned n = dm.n, n_rows = dm.n_rows, heads = dm.heads;
  const unsigned total = (unsigned)dm.batch * heads * n_rows * n;   // < 2^31: 16 bytes each fit memory
  const int part = threadIdx.x % C::G;
  uint4 uo[C::U][C::kSteps], ud[C::U][C::kSteps];
  unsigned idx[C::U], row[C::U];
#pragma unroll
  for (int u = 0; u < C::U; ++u) {
    idx[u] = block * C::kRows + u * (kPrepThreads / C::G) + threadIdx.x / C::G;
    const unsigned at = min(idx[u], total - 1);
    row[u] = at / n;
    const unsigned j = at - row[u] * n, i = row[u] % n_rows, bh = row[u] / n_rows;
    const unsigned h = bh % heads, b = bh / heads;
    const T* po = (const T*)o.p + b * o.sb + h * o.sh + (int64_t)i * o.si + (int64_t)j * o.sj;
    const T* pd = (const T*)d_o.p + b * d_o.sb + h * d_o.sh + (int64_t)i * d_o.si + (int64_t)j * d_o.sj;
#pragma unroll
    for (int st = 0; st < C::kSteps; ++st) {
      const int off = (st * C::G + part) * C::kVec;
      uo[u][st] = load_once(po + off);
      ud[u][st] = load_once(pd + off);
    }
  }
#pragma unroll
  for (int u = 0; u < C::U; ++u) {
    float acc = 0.f;
#pragma unroll
    for (int st = 0; st < C::kSteps; ++st) {
      const T* eo = reinterpret_cast<const T*>(&uo[u][st]);
      const T* ed = reinterpret_cast<const T*>(&ud[u][st]);
#pragma unroll
      for (int c = 0; c < C::kVec; ++c) acc = fmaf(to_f32<T>(eo[c]), to_f32<T>(ed[c]), acc);
    }
#pragma unroll
    for (int m = C::G / 2; m > 0; m >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, m);
    if (idx[u] < total && part == 0) {
      const int64_t out = (int64_t)row[u] * dm.n_pad + (idx[u] - row[u] * n);
      delta[out] = acc;
      neg_lse2[out] = -lse[idx[u]] * kLog2e;
    }
  }
}

// ---------------------------------------------------------------------------
// ds_up[b, h, i] (fp16, D = 128): the power of two that scales the pair row's dS to at most
// 2^15.  dS = P (dP - delta) with P <= 1 and |dP|, |delta| <= D max|dO| max|v|, the largest finite
// values of the row, v over its open keys.  Without it a gradient of 1e-5 leaves dS among fp16's
// subnormals and one of 1e4 beyond its range.  Bound by memory: dO and v once more (120 us at
// n = 512, h = 4).
// ---------------------------------------------------------------------------
template <int D>
__device__ void prepare_row_scale(const Prep& a, const View5& d_o, int w) {
  constexpr int kParts = D / 8, kRows = kPrepThreads / kParts;   // 16-byte parts of a row, rows at a time
  const int n = a.dm.n, i = w % a.dm.n_rows, bh = w / a.dm.n_rows, b = bh / a.dm.heads, h = bh % a.dm.heads;
  const uint8_t* mrow = a.mask.p + b * a.mask.sb + (int64_t)i * a.mask.si;
  int open = 0;
  for (int k = threadIdx.x; k < n; k += kPrepThreads) open |= mrow[k * a.mask.sk] == 0;
  const bool row_full = !__syncthreads_or(open);
  const int part = threadIdx.x % kParts * 8;
  const __half* po = (const __half*)d_o.p + b * d_o.sb + h * d_o.sh + (int64_t)i * d_o.si + part;
  const __half* pv = (const __half*)a.v.p + b * a.v.sb + h * a.v.sh + (int64_t)i * a.v.si + part;
  // magnitudes as 16-bit integers, in order; 0x7c00 and above are not finite
  uint32_t most_o = 0u, most_v = 0u;
  auto most = [](uint32_t m, uint32_t u) {
    u &= 0x7fff7fffu;
    return __vmaxu2(m, u & __vcmpltu2(u, 0x7c007c00u));
  };
#pragma unroll 4
  for (int r = threadIdx.x / kParts; r < n; r += kRows) {
    const uint4 g = __ldg(reinterpret_cast<const uint4*>(po + (int64_t)r * d_o.sj));
    most_o = most(most(most(most(most_o, g.x), g.y), g.z), g.w);
    if (row_full || mrow[r * a.mask.sk] == 0) {
      const uint4 u = __ldg(reinterpret_cast<const uint4*>(pv + (int64_t)r * a.v.sj));
      most_v = most(most(most(most(most_v, u.x), u.y), u.z), u.w);
    }
  }
  __shared__ uint32_t shared_most[2];
  if (threadIdx.x < 2) shared_most[threadIdx.x] = 0u;
  __syncthreads();
  const uint32_t mo = __reduce_max_sync(0xffffffffu, max(most_o & 0xffffu, most_o >> 16));
  const uint32_t mv = __reduce_max_sync(0xffffffffu, max(most_v & 0xffffu, most_v >> 16));
  if ((threadIdx.x & 31) == 0) {
    atomicMax(&shared_most[0], mo);
    atomicMax(&shared_most[1], mv);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const float fo = __half2float(__ushort_as_half((unsigned short)shared_most[0]));
    const float fv = __half2float(__ushort_as_half((unsigned short)shared_most[1]));
    // |x| < 2^(ilogb(x) + 1); 2 D = 2^8
    static_assert(D == 128, "exponent of 2 D");
    a.ds_up[w] = fo > 0.f && fv > 0.f ? ldexpf(1.f, 15 - 8 - (ilogbf(fo) + 1) - (ilogbf(fv) + 1)) : 1.f;
  }
}

__global__ void __launch_bounds__(kPrepThreads) fwd_prepare_kernel(Prep a) {
  after_previous();
  int w = blockIdx.x;
  if (w == 0 && threadIdx.x == 0) repeat_status(a.status);
  if (w < a.mask_blocks) return prepare_mask_row<true>(a, w);
  prepare_bias_tile(a, w - a.mask_blocks);
}

template <typename T, int D>
__global__ void __launch_bounds__(kPrepThreads) bwd_prepare_kernel(Prep a, View5 o, View5 d_o, const float* lse,
                                                                   float* delta, float* neg_lse2) {
  after_previous();
  int w = blockIdx.x;
  if (w == 0 && threadIdx.x == 0) repeat_status(a.status);
  if (w < a.mask_blocks) return prepare_mask_row<false>(a, w);
  w -= a.mask_blocks;
  if (w < a.bias_blocks) return prepare_bias_tile(a, w);
  w -= a.bias_blocks;
  if constexpr (std::is_same<T, __half>::value && D == 128) {
    if (w < a.scale_blocks) return prepare_row_scale<D>(a, d_o, w);
  }
  prepare_delta<T, D>(o, d_o, lse, delta, neg_lse2, a.dm, w - a.scale_blocks);
}

// ---------------------------------------------------------------------------
// db: the row-split partials summed in split order (fixed order => deterministic), written as
// fp32 or in the gradient's type.  kWide: four keys of one row per thread (n % 4 == 0, rows
// aligned to four elements).
// ---------------------------------------------------------------------------
template <typename T, bool kWide>
__global__ void db_finish_kernel(const float* partials, int splits, View4 db, int heads, int n, int64_t count) {
  after_previous();
  constexpr int V = kWide ? 4 : 1;
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx * V >= count) return;
  float acc[V];
  for (int s = 0; s < splits; ++s) {
    if constexpr (kWide) {
      const float4 v = __ldg(reinterpret_cast<const float4*>(partials + s * count) + idx);
      const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int c = 0; c < V; ++c) acc[c] = s ? acc[c] + e[c] : e[c];
    } else {
      const float e = __ldg(partials + s * count + idx);
      acc[0] = s ? acc[0] + e : e;
    }
  }
  const int per_row = n / V, key = (int)(idx % per_row) * V;
  int64_t r = idx / per_row;
  const int j = (int)(r % n);
  r /= n;
  const int h = (int)(r % heads), b = (int)(r / heads);
  T* dst = (T*)db.p + b * db.sb + h * db.sh + (int64_t)j * db.sj + key;
  if constexpr (!kWide) {
    dst[0] = from_f32<T>(acc[0]);
  } else if constexpr (sizeof(T) == 4) {
    *reinterpret_cast<float4*>(dst) = make_float4(acc[0], acc[1], acc[2], acc[3]);
  } else {
    const T o4[4] = {from_f32<T>(acc[0]), from_f32<T>(acc[1]), from_f32<T>(acc[2]), from_f32<T>(acc[3])};
    *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(o4);
  }
}

template <typename T>
cudaError_t launch_finish(const float* partials, int splits, View4 db, int batch, int heads, int n, cudaStream_t s) {
  const int64_t count = (int64_t)batch * heads * n * n;
  const int64_t row_bytes = 4 * sizeof(T);
  const bool wide = n % 4 == 0 && db.sj % 4 == 0 && db.sh % 4 == 0 && db.sb % 4 == 0 &&
                    reinterpret_cast<uintptr_t>(db.p) % row_bytes == 0 &&
                    (reinterpret_cast<uintptr_t>(partials) & 15) == 0;
  const int64_t threads = wide ? count / 4 : count;
  const unsigned blocks = (unsigned)((threads + 255) / 256);
  if (wide)
    return launch_early(db_finish_kernel<T, true>, blocks, 256, 0, s, partials, splits, db, heads, n, count);
  return launch_early(db_finish_kernel<T, false>, blocks, 256, 0, s, partials, splits, db, heads, n, count);
}

Prep make_prep(const MaskView& mask, const View4& bias, const Dims& dm) {
  Prep p{};
  p.mask = mask;
  p.bias = bias;
  p.dm = dm;
  p.mask_blocks = dm.batch * dm.n_rows;
  p.fill_blocks = 1;
  p.bias_tiles = (dm.n + 63) / 64;
  return p;
}

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

}  // namespace

cudaError_t bwd_prepare(const BwdArgs& a, cudaStream_t s) {
  const Dims& dm = a.dm;
  Prep p = make_prep(a.mask, a.bias, dm);
  p.rowfull = a.rowfull;
  p.maskbits = a.maskbits;
  p.maskbits_lin = a.maskbits_lin;
  p.mask_words = a.mask_words;
  p.rowrange = a.rowrange;
  p.bias_t = (uint16_t*)a.bias_t;
  p.bias_pad = (uint16_t*)a.bias_pad;
  p.status = a.status;
  p.bias_blocks = a.bias_t || a.bias_pad ? p.bias_tiles * p.bias_tiles * dm.batch * dm.heads : 0;
  p.v = a.v;
  p.ds_up = a.ds_up;
  p.scale_blocks = a.ds_up ? dm.batch * dm.heads * dm.n_rows : 0;
  return dispatch(a.dtype, dm.d, [&](auto* tp, auto dc) {
    using T = std::remove_pointer_t<decltype(tp)>;
    constexpr int D = decltype(dc)::value;
    constexpr int kRows = DeltaCfg<T, D>::kRows;
    const int64_t rows = (int64_t)dm.batch * dm.heads * dm.n_rows * dm.n;
    const unsigned blocks =
        (unsigned)(p.mask_blocks + p.bias_blocks + p.scale_blocks + (rows + kRows - 1) / kRows);
    return launch_early(bwd_prepare_kernel<T, D>, blocks, kPrepThreads, 0, s, p, a.o, a.d_o, a.lse, a.delta, a.neg_lse2);
  });
}

cudaError_t fwd_prepare(const FwdArgs& a, cudaStream_t s) {
  // the live key-tile range of every row always; the packed masks, row flags and the padded
  // bias copy only where the workspace holds them
  Prep p = make_prep(a.mask, a.bias, a.dm);
  p.rowfull = a.rowfull;
  p.maskbits = a.maskbits;
  p.mask_words = a.mask_words;
  p.rowrange = a.rowrange;
  p.bias_pad = (uint16_t*)a.bias_pad;
  p.status = a.status;
  p.bias_blocks = a.bias_pad ? p.bias_tiles * p.bias_tiles * a.dm.batch * a.dm.heads : 0;
  if (a.dm.d <= 64) {
    p.v = a.v;
    p.o = a.o;
    p.lse = a.lse;
    p.dtype = a.dtype;
    // A row's heads are shared by as many blocks as one round holds (four blocks an SM): beside few
    // rows the kernel lasts as long as its slowest one.  The forward with one row of eight without an
    // open key, one block a row and so: n = 1024, h = 8, d = 64 82 -> 46 us, n = 2048 230 -> 145 us,
    // n = 4096, h = 4, d = 32 271 -> 232 us.
    const int most = 4 * sm_count() / p.mask_blocks;
    p.fill_blocks = most < 1 ? 1 : most < a.dm.heads ? most : a.dm.heads;
    p.mask_blocks *= p.fill_blocks;
  }
  return launch_early(fwd_prepare_kernel, p.mask_blocks + p.bias_blocks, kPrepThreads, 0, s, p);
}

cudaError_t db_reduce_splits(const BwdArgs& a, cudaStream_t s) {
  if (a.splits <= 1) return cudaSuccess;
  const int64_t n = a.dm.n;
  const View4 out{(char*)a.db_f32, n * n * a.dm.heads, n * n, n, 1};
  return launch_finish<float>(a.db_partials, a.splits, out, a.dm.batch, a.dm.heads, a.dm.n, s);
}

cudaError_t db_cast(const float* partials, int splits, View4 db, int dtype, int batch, int heads, int n,
                    cudaStream_t s) {
  switch (dtype) {
    case TRIFAST_F32: return launch_finish<float>(partials, splits, db, batch, heads, n, s);
    case TRIFAST_BF16: return launch_finish<__nv_bfloat16>(partials, splits, db, batch, heads, n, s);
    case TRIFAST_F16: return launch_finish<__half>(partials, splits, db, batch, heads, n, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace trifast
