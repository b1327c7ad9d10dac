// Small kernels around the attention kernels of both families: row flags and packed key
// masks, delta, bias copies, the sum of db's row splits and its cast.

#include <math.h>

#include <type_traits>

#include "kernels.h"

namespace trifast {
namespace {

constexpr float kMinusInf = -INFINITY;
constexpr float kMaxInit = -1e30f;  // finite start of the running max: exp(-inf - m) stays 0, never NaN

template <typename T>
__device__ __forceinline__ const T* row5(const View5& t, int b, int h, int i, int j) {
  return (const T*)t.p + b * t.sb + h * t.sh + (int64_t)i * t.si + (int64_t)j * t.sj;
}
template <typename T>
__device__ __forceinline__ T* row5w(const View5& t, int b, int h, int i, int j) {
  return (T*)t.p + b * t.sb + h * t.sh + (int64_t)i * t.si + (int64_t)j * t.sj;
}
template <typename T>
__device__ __forceinline__ const T* row4(const View4& t, int b, int h, int j) {
  return (const T*)t.p + b * t.sb + h * t.sh + (int64_t)j * t.sj;
}

// ---------------------------------------------------------------------------
// rowfull[b, i] = 1 when every key of pair row i is masked.
// ---------------------------------------------------------------------------
__global__ void rowfull_kernel(MaskView mask, int n, int n_rows, uint8_t* rowfull,
                               uint32_t* maskbits, uint32_t* maskbits_lin, int mask_words,
                               uint32_t* rowrange, unsigned int* status) {
  const int bi = blockIdx.x;
  if (bi == 0 && threadIdx.x == 0) repeat_status(status);
  const int b = bi / n_rows, i = bi % n_rows;
  const uint8_t* row = mask.p + b * mask.sb + (int64_t)i * mask.si;
  __shared__ int first_open, last_open;
  if (threadIdx.x == 0) {
    first_open = n;
    last_open = -1;
  }
  __syncthreads();
  int lo = n, hi = -1;
  for (int k = threadIdx.x; k < n; k += blockDim.x) {
    if (row[k] == 0) {
      lo = min(lo, k);
      hi = max(hi, k);
    }
  }
  if (hi >= 0) {
    atomicMin(&first_open, lo);
    atomicMax(&last_open, hi);
  }
  __syncthreads();
  const int open = last_open >= 0;
  if (threadIdx.x == 0) {
    if (rowfull) rowfull[bi] = open ? 0 : 1;
    // 128-key tiles [first, last + 1) that hold an open key: the tensor-core kernels walk
    // only those.  A fully masked row weighs all n keys: every tile.
    if (rowrange) {
      const uint32_t t0 = open ? (uint32_t)(first_open >> 7) : 0u;
      const uint32_t t1 = open ? (uint32_t)(last_open >> 7) + 1u : (uint32_t)((n + 127) >> 7);
      rowrange[bi] = t0 | (t1 << 16);
    }
  }
  if (!maskbits) return;
  // Packed key mask (bit set = key dropped or beyond n).  A fully masked row keeps
  // all n keys with uniform weight, so only the keys beyond n stay set.  Layout per
  // 128-key chunk c: word c*4 + jb holds, at bit l, key c*128 + 4*l + jb (the order
  // in which a warp reading four mask bytes per lane produces the words).
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int c = warp; c < mask_words / 4; c += blockDim.x >> 5) {
#pragma unroll
    for (int jb = 0; jb < 4; ++jb) {
      const int k = c * 128 + 4 * lane + jb;
      const int dropped = (k < n) ? (open ? (row[k] != 0) : 0) : 1;
      const unsigned bits = __ballot_sync(0xffffffffu, dropped);
      if (lane == 0) maskbits[(int64_t)bi * mask_words + c * 4 + jb] = bits;
    }
  }
  // The same bits in key order (word w, bit l: key 32 * w + l), when asked for.
  if (maskbits_lin) {
    for (int w = warp; w < mask_words; w += blockDim.x >> 5) {
      const int k = w * 32 + lane;
      const int dropped = (k < n) ? (open ? (row[k] != 0) : 0) : 1;
      const unsigned bits = __ballot_sync(0xffffffffu, dropped);
      if (lane == 0) maskbits_lin[(int64_t)bi * mask_words + w] = bits;
    }
  }
}

// bias_pad[b, h, j, 0..n_pad) = bias[b, h, j, 0..n) (pad = 0): a copy whose row pitch
// is a multiple of 16 bytes, as TMA needs, for n % 8 != 0.
__global__ void bias_pad_kernel(View4 bias, uint16_t* out, int heads, int n, int n_pad) {
  const int bh = blockIdx.z, b = bh / heads, h = bh % heads;
  const int j = blockIdx.y;
  const uint16_t* src = (const uint16_t*)bias.p + b * bias.sb + h * bias.sh + (int64_t)j * bias.sj;
  uint16_t* dst = out + ((int64_t)bh * n + j) * n_pad;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n_pad; k += gridDim.x * blockDim.x)
    dst[k] = (k < n) ? src[k] : (uint16_t)0;
}

// ---------------------------------------------------------------------------
// delta[b, h, i, j] = sum_d o * dO   (fp32; never rounded to the input dtype)
// ---------------------------------------------------------------------------
template <typename T, int D>
__global__ void delta_kernel(View5 o, View5 d_o, const float* lse, float* delta, float* neg_lse2,
                             Dims dm) {
  // A group of G threads owns one (b, h, i, j) row of D elements, 16 bytes per thread
  // and step, so that a warp reads whole 128-byte lines of o and dO.
  constexpr int kVec = 16 / sizeof(T);   // elements per 16-byte load
  constexpr int G = (D / kVec) < 4 ? (D / kVec) : 4;
  constexpr int kSteps = D / (kVec * G);
  const int64_t total = (int64_t)dm.batch * dm.heads * dm.n_rows * dm.n;
  const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t idx = gid / G;
  const int part = (int)(gid % G);
  const bool valid = idx < total;
  float acc = 0.f;
  if (valid) {
    const int j = idx % dm.n;
    int64_t r = idx / dm.n;
    const int i = r % dm.n_rows;
    r /= dm.n_rows;
    const int h = r % dm.heads, b = r / dm.heads;
    const T* po = row5<T>(o, b, h, i, j);
    const T* pd = row5<T>(d_o, b, h, i, j);
#pragma unroll
    for (int st = 0; st < kSteps; ++st) {
      const int off = (st * G + part) * kVec;
      const uint4 uo = *reinterpret_cast<const uint4*>(po + off);
      const uint4 ud = *reinterpret_cast<const uint4*>(pd + off);
      const T* eo = reinterpret_cast<const T*>(&uo);
      const T* ed = reinterpret_cast<const T*>(&ud);
#pragma unroll
      for (int c = 0; c < kVec; ++c) acc = fmaf(to_f32<T>(eo[c]), to_f32<T>(ed[c]), acc);
    }
  }
#pragma unroll
  for (int m = G / 2; m > 0; m >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, m);
  if (valid && part == 0) {
    const int64_t out = (idx / dm.n) * dm.n_pad + idx % dm.n;  // row pitch n_pad
    delta[out] = acc;
    neg_lse2[out] = -lse[idx] * 1.4426950408889634f;
  }
}

// bias_t[b, h, k, j] = bias[b, h, j, k] (row pitch n_pad) for 2-byte elements (the dk/dv kernel reads
// the bias with keys on the rows).  64 x 64 tiles; 4-byte accesses on both sides when the rows allow it.
__global__ void __launch_bounds__(256)
bias_transpose_kernel(View4 bias, uint16_t* out, int heads, int n, int n_pad) {
  __shared__ uint16_t tile[64][66];
  const int bh = blockIdx.z, b = bh / heads, h = bh % heads;
  const uint16_t* src = (const uint16_t*)bias.p + b * bias.sb + h * bias.sh;
  uint16_t* dst = out + (int64_t)bh * n * n_pad;
  const int j0 = blockIdx.y * 64, k0 = blockIdx.x * 64;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
  const bool pairs_in = (bias.sj % 2 == 0) && (bias.sh % 2 == 0) && (bias.sb % 2 == 0) &&
                        ((reinterpret_cast<uintptr_t>(bias.p) & 3) == 0);
  for (int r = ty; r < 64; r += 8) {
    const int j = j0 + r, k = k0 + 2 * tx;
    if (j < n) {
      if (pairs_in && k + 1 < n) {
        const uint32_t u = *reinterpret_cast<const uint32_t*>(src + (int64_t)j * bias.sj + k);
        tile[r][2 * tx] = (uint16_t)(u & 0xffffu);
        tile[r][2 * tx + 1] = (uint16_t)(u >> 16);
      } else {
        if (k < n) tile[r][2 * tx] = src[(int64_t)j * bias.sj + k];
        if (k + 1 < n) tile[r][2 * tx + 1] = src[(int64_t)j * bias.sj + k + 1];
      }
    }
  }
  __syncthreads();
  for (int r = ty; r < 64; r += 8) {  // output row k0 + r holds queries j0 .. j0 + 63
    const int k = k0 + r, j = j0 + 2 * tx;
    if (k < n) {
      if (j + 1 < n) {  // n_pad is even and dst 4-byte aligned: a pair never straddles
        const uint32_t u = (uint32_t)tile[2 * tx][r] | ((uint32_t)tile[2 * tx + 1][r] << 16);
        *reinterpret_cast<uint32_t*>(dst + (int64_t)k * n_pad + j) = u;
      } else if (j < n) {
        dst[(int64_t)k * n_pad + j] = tile[2 * tx][r];
      }
    }
  }
}

// Sum the row-split partials in split order (fixed order => deterministic).
__global__ void db_reduce_kernel(const float* partials, float* out, int splits, int64_t count) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= count) return;
  float acc = partials[idx];
  for (int s = 1; s < splits; ++s) acc += partials[(int64_t)s * count + idx];
  out[idx] = acc;
}

// four elements per thread (count % 4 == 0)
__global__ void db_reduce4_kernel(const float4* partials, float4* out, int splits, int64_t count4) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= count4) return;
  float4 acc = __ldg(partials + idx);
  for (int s = 1; s < splits; ++s) {  // fixed split order: deterministic
    const float4 v = __ldg(partials + (int64_t)s * count4 + idx);
    acc.x += v.x;
    acc.y += v.y;
    acc.z += v.z;
    acc.w += v.w;
  }
  out[idx] = acc;
}

// four keys of one row per thread (n % 4 == 0, destination rows 8-byte aligned; T is 16 bits)
template <typename T>
__global__ void db_cast4_kernel(const float4* src, View4 db, int heads, int n, int64_t count4) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= count4) return;
  const int n4 = n >> 2;
  const int key = (int)(idx % n4) * 4;
  int64_t r = idx / n4;
  const int j = (int)(r % n);
  r /= n;
  const int h = (int)(r % heads), b = (int)(r / heads);
  const float4 v = __ldg(src + idx);
  T* dst = (T*)db.p + b * db.sb + h * db.sh + (int64_t)j * db.sj + key;
  const T o4[4] = {from_f32<T>(v.x), from_f32<T>(v.y), from_f32<T>(v.z), from_f32<T>(v.w)};
  *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(o4);
}

template <typename T>
__global__ void db_cast_kernel(const float* src, View4 db, int heads, int n, int64_t count) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= count) return;
  const int key = idx % n;
  int64_t r = idx / n;
  const int j = r % n;
  r /= n;
  const int h = r % heads, b = r / heads;
  T* dst = (T*)db.p + b * db.sb + h * db.sh + (int64_t)j * db.sj;
  dst[key] = from_f32<T>(src[idx]);
}

// ---------------------------------------------------------------------------
// dispatch on (dtype, d)
// ---------------------------------------------------------------------------
template <typename F>
cudaError_t dispatch(int dtype, int d, F&& f) {
#define TRIFAST_D_CASES(T)                                 \
  switch (d) {                                             \
    case 16: f((T*)nullptr, std::integral_constant<int, 16>{}); break;   \
    case 32: f((T*)nullptr, std::integral_constant<int, 32>{}); break;   \
    case 64: f((T*)nullptr, std::integral_constant<int, 64>{}); break;   \
    case 128: f((T*)nullptr, std::integral_constant<int, 128>{}); break; \
    default: return cudaErrorInvalidValue;                 \
  }
  switch (dtype) {
    case TRIFAST_F32: TRIFAST_D_CASES(float) break;
    case TRIFAST_BF16: TRIFAST_D_CASES(__nv_bfloat16) break;
    case TRIFAST_F16: TRIFAST_D_CASES(__half) break;
    default: return cudaErrorInvalidValue;
  }
#undef TRIFAST_D_CASES
  return cudaGetLastError();
}

}  // namespace

cudaError_t bwd_prepare(const BwdArgs& a, cudaStream_t s) {
  const Dims& dm = a.dm;
  rowfull_kernel<<<dm.batch * dm.n_rows, 128, 0, s>>>(a.mask, dm.n, dm.n_rows, a.rowfull, a.maskbits,
                                                      a.maskbits_lin, a.mask_words, a.rowrange, a.status);
  if (a.bias_t) {
    dim3 grid((dm.n + 63) / 64, (dm.n + 63) / 64, dm.batch * dm.heads);
    bias_transpose_kernel<<<grid, 256, 0, s>>>(a.bias, (uint16_t*)a.bias_t, dm.heads, dm.n,
                                                       dm.n_pad);
  }
  if (a.bias_pad) {
    dim3 grid(1, dm.n, dm.batch * dm.heads);
    bias_pad_kernel<<<grid, 256, 0, s>>>(a.bias, (uint16_t*)a.bias_pad, dm.heads, dm.n, dm.n_pad);
  }
  return dispatch(a.dtype, dm.d, [&](auto* tp, auto dc) {
    using T = std::remove_pointer_t<decltype(tp)>;
    constexpr int D = decltype(dc)::value;
    constexpr int kVec = 16 / sizeof(T);
    constexpr int G = (D / kVec) < 4 ? (D / kVec) : 4;
    const int64_t threads = (int64_t)dm.batch * dm.heads * dm.n_rows * dm.n * G;
    delta_kernel<T, D><<<(unsigned)((threads + 255) / 256), 256, 0, s>>>(a.o, a.d_o, a.lse, a.delta,
                                                                       a.neg_lse2, dm);
  });
}

cudaError_t fwd_prepare(const FwdArgs& a, cudaStream_t s) {
  const Dims& dm = a.dm;
  // the live key-tile range of every row always; the packed masks, row flags and the padded
  // bias copy only where the workspace holds them (n % 8 != 0)
  rowfull_kernel<<<dm.batch * dm.n_rows, 128, 0, s>>>(a.mask, dm.n, dm.n_rows, a.rowfull, a.maskbits,
                                                      nullptr, a.mask_words, a.rowrange, a.status);
  if (a.bias_pad) {
    dim3 grid(1, dm.n, dm.batch * dm.heads);
    bias_pad_kernel<<<grid, 256, 0, s>>>(a.bias, (uint16_t*)a.bias_pad, dm.heads, dm.n, dm.n_pad);
  }
  return cudaGetLastError();
}

cudaError_t db_reduce_splits(const BwdArgs& a, cudaStream_t s) {
  if (a.splits <= 1) return cudaSuccess;
  const int64_t count = (int64_t)a.dm.batch * a.dm.heads * a.dm.n * a.dm.n;
  if (count % 4 == 0) {  // the partials and db_f32 sit on 256-byte boundaries of the workspace
    const int64_t c4 = count / 4;
    db_reduce4_kernel<<<(unsigned)((c4 + 255) / 256), 256, 0, s>>>(
        reinterpret_cast<const float4*>(a.db_partials), reinterpret_cast<float4*>(a.db_f32), a.splits,
        c4);
    return cudaGetLastError();
  }
  db_reduce_kernel<<<(unsigned)((count + 255) / 256), 256, 0, s>>>(a.db_partials, a.db_f32,
                                                                 a.splits, count);
  return cudaGetLastError();
}

cudaError_t db_cast(const float* db_f32, View4 db, int dtype, int batch, int heads, int n,
                    cudaStream_t s) {
  const int64_t count = (int64_t)batch * heads * n * n;
  const bool wide = dtype != TRIFAST_F32 && n % 4 == 0 && db.sj % 4 == 0 && db.sh % 4 == 0 &&
                    db.sb % 4 == 0 && (reinterpret_cast<uintptr_t>(db.p) & 7) == 0 &&
                    (reinterpret_cast<uintptr_t>(db_f32) & 15) == 0;
  if (wide) {
    const int64_t c4 = count / 4;
    const unsigned blocks4 = (unsigned)((c4 + 255) / 256);
    const float4* src = reinterpret_cast<const float4*>(db_f32);
    if (dtype == TRIFAST_BF16)
      db_cast4_kernel<__nv_bfloat16><<<blocks4, 256, 0, s>>>(src, db, heads, n, c4);
    else
      db_cast4_kernel<__half><<<blocks4, 256, 0, s>>>(src, db, heads, n, c4);
    return cudaGetLastError();
  }
  const unsigned blocks = (unsigned)((count + 255) / 256);
  switch (dtype) {
    case TRIFAST_F32: db_cast_kernel<float><<<blocks, 256, 0, s>>>(db_f32, db, heads, n, count); break;
    case TRIFAST_BF16: db_cast_kernel<__nv_bfloat16><<<blocks, 256, 0, s>>>(db_f32, db, heads, n, count); break;
    case TRIFAST_F16: db_cast_kernel<__half><<<blocks, 256, 0, s>>>(db_f32, db, heads, n, count); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

}  // namespace trifast
