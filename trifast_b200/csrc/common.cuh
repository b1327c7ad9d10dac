// Shared device/host helpers of the triangle-attention kernels.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include "../../include/trifast_b200.h"

namespace trifast {

// Smallest n the tensor-core kernels take: one 128 x 128 tile at least a quarter full.
constexpr int kMinTensorCoreN = 64;


// (b, h, i, j, d) view with element strides; d contiguous.
struct View5 {
  char* p;
  int64_t sb, sh, si, sj;
};
// (b, h, j, k) view with element strides; sk is 1 except for a caller's bias under
// TRIFAST_FLAG_STRIDED.
struct View4 {
  char* p;
  int64_t sb, sh, sj, sk;
};
// (b, i, k) byte mask; sk as above.
struct MaskView {
  const uint8_t* p;
  int64_t sb, si, sk;
};

struct Dims {
  int batch, heads, n, n_rows, d;
  int n_pad;       // n rounded up to 8: row pitch (elements) of workspace vectors and bias copies
  float scale;     // d^-0.5
  float sentinel;  // finfo(dtype).min as float: stored as lse of fully masked rows
};

inline View5 make_view(const trifast_t5* t) {
  return View5{(char*)t->data, t->stride[0], t->stride[1], t->stride[2], t->stride[3]};
}
inline View4 make_view(const trifast_t4* t) {
  return View4{(char*)t->data, t->stride[0], t->stride[1], t->stride[2], 1};
}
inline MaskView make_view(const trifast_mask* t) {
  return MaskView{t->data, t->stride[0], t->stride[1], 1};
}

// The bias and mask of a call: with TRIFAST_FLAG_STRIDED the descriptors are the longer
// structs, whose innermost dimension has a stride of its own.
inline View4 bias_view(const trifast_t4* t, int flags) {
  View4 v = make_view(t);
  if (flags & TRIFAST_FLAG_STRIDED) v.sk = reinterpret_cast<const trifast_t4_strided*>(t)->stride[3];
  return v;
}
inline MaskView mask_view(const trifast_mask* t, int flags) {
  MaskView v = make_view(t);
  if (flags & TRIFAST_FLAG_STRIDED) v.sk = reinterpret_cast<const trifast_mask_strided*>(t)->stride[2];
  return v;
}

template <typename T> __device__ __forceinline__ float to_f32(T x);
template <> __device__ __forceinline__ float to_f32<float>(float x) { return x; }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 x) {
  return __bfloat162float(x);
}
template <> __device__ __forceinline__ float to_f32<__half>(__half x) { return __half2float(x); }

template <typename T> __device__ __forceinline__ T from_f32(float x);
template <> __device__ __forceinline__ float from_f32<float>(float x) { return x; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float x) {
  return __float2bfloat16_rn(x);
}
template <> __device__ __forceinline__ __half from_f32<__half>(float x) {
  return __float2half_rn(x);
}

// Kernels whose bounded waits give up OR a non-zero code into a device status
// word (they never trap); its address is handed to them as a kernel argument.  Next to the
// word lies the address of a pinned host word, or null: whoever sets the status also writes
// it there (and the prepare kernels repeat it while it stays set), so that a binding learns
// of the time-out from host memory, without a copy enqueued behind each call.
struct DeviceStatus {
  unsigned int bits;
  unsigned int unused;
  unsigned int* host;
};
enum DeviceStatusBits : unsigned int {
  kStatusTimeoutFwd = 1u,
  kStatusTimeoutBwdDb = 2u,
  kStatusTimeoutBwdDq = 4u,
  kStatusTimeoutBwdDkv = 8u,
  kStatusTimeoutBwdFused = 16u,
  kStatusTimeoutProbe = 32u,
  kStatusTimeoutPushReduce = 64u,
};

// (out of line, so that the cold path leaves the code of the kernels' loops alone)
static __device__ __noinline__ void mirror_status(unsigned int* status, unsigned int bits) {
  unsigned int* host = reinterpret_cast<DeviceStatus*>(status)->host;
  if (host) {
    *reinterpret_cast<volatile unsigned int*>(host) = bits;
    __threadfence_system();
  }
}
// For the prepare kernels, which run first in a call.
__device__ __forceinline__ void repeat_status(unsigned int* status) {
  const unsigned int bits = *reinterpret_cast<volatile unsigned int*>(status);
  if (bits != 0u) mirror_status(status, bits);
}
__device__ __forceinline__ void set_status(unsigned int* status, unsigned int bits) {
  mirror_status(status, atomicOr(status, bits) | bits);
}

// Kernels of a call are launched with programmatic serialization (launch_early): the launch itself
// and the placing of the blocks need not wait until the kernel before has been flushed out; the
// blocks wait here for that, first of all and before any early return, so that a kernel that is
// complete implies that all before it are.  No kernel lets the next one start before its own
// blocks have ended (griddepcontrol.launch_dependents at their start was slower for all but the
// smallest calls: n = 384 445 us a step, n = 733 717 us a forward).
__device__ __forceinline__ void after_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Launches a kernel that calls after_previous().  Against plain launches, h = 4, d = 32, calls back to
// back: forward and backward (six kernels) at n = 256 154.8 -> 143.8 us, n = 384 428 -> 415, n = 512 (15 %
// padding) 823 -> 813; forward alone at n = 733 703 -> 699 us.
template <typename... P, typename... A>
cudaError_t launch_early(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t s, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// SMs of the current device.
int sm_count();

// Opts a kernel in to `bytes` of dynamic shared memory: one runtime call per kernel, device
// and growth of the size, not one per launch.
// kFirst: the kernel's tiles count on the dynamic shared memory lying first, on the SM's 1024-byte
// boundary (the atoms of the swizzles); with static shared memory before it the kernel is refused.
template <auto Kernel, bool kFirst = false>
cudaError_t opt_in_smem(int bytes) {
  static std::atomic<int> have[64];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (have[dev].load(std::memory_order_acquire) >= bytes) return cudaSuccess;
  e = cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) return e;
  if (kFirst) {
    cudaFuncAttributes at;
    if ((e = cudaFuncGetAttributes(&at, Kernel)) != cudaSuccess) return e;
    if (at.sharedSizeBytes != 0) return cudaErrorInvalidValue;
  }
  int seen = have[dev].load(std::memory_order_relaxed);
  while (seen < bytes && !have[dev].compare_exchange_weak(seen, bytes, std::memory_order_release)) {
  }
  return cudaSuccess;
}

}  // namespace trifast
