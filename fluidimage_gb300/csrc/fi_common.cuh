// Shared helpers of the fluidimage_gb300 CUDA library.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>

#include "../../include/fluidimage_gb300.h"

namespace fi {

// Last error message of the calling host thread (returned by fi_last_error()).
void set_error(const char* fmt, ...);

// Counts kernel launches made by the library (fi_launch_count()).
void add_launches(int k);

// Checks a CUDA call inside an entry point; returns FI_ERR_CUDA on failure.
#define FI_CUDA_TRY(call)                                                     \
  do {                                                                        \
    cudaError_t fi_err_ = (call);                                             \
    if (fi_err_ != cudaSuccess) {                                             \
      ::fi::set_error("%s: %s (%s:%d)", #call, cudaGetErrorString(fi_err_),   \
                      __FILE__, __LINE__);                                    \
      return FI_ERR_CUDA;                                                     \
    }                                                                         \
  } while (0)

#define FI_REQUIRE(cond, ...)                                                 \
  do {                                                                        \
    if (!(cond)) {                                                            \
      ::fi::set_error(__VA_ARGS__);                                           \
      return FI_ERR_INVALID;                                                  \
    }                                                                         \
  } while (0)

// Raises a kernel's dynamic shared-memory limit to at least `bytes` on the current device,
// calling the runtime only when the limit has to grow there.  Without a call it is 48 KB
// less the kernel's own (static) shared memory, asked for once.  The attribute is per
// device, so the call site's record keeps the limit for each device (0: not asked yet),
// read and written under one mutex so that host threads launching concurrently never
// lower it.
inline std::mutex& smem_limit_mutex() {
  static std::mutex m;
  return m;
}
constexpr int FI_SMEM_DEVICES = 64;
struct SmemLimit {
  size_t bytes[FI_SMEM_DEVICES] = {};
};
template <typename Kernel>
inline cudaError_t raise_smem_limit(Kernel* kernel, size_t bytes, SmemLimit& rec) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lock(smem_limit_mutex());
  const bool cached = dev >= 0 && dev < FI_SMEM_DEVICES;
  size_t limit = cached ? rec.bytes[dev] : 0;
  if (limit == 0) {
    cudaFuncAttributes attr;
    e = cudaFuncGetAttributes(&attr, kernel);
    if (e != cudaSuccess) return e;
    limit = 48 * 1024 - attr.sharedSizeBytes;
  }
  if (bytes > limit) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return e;
    limit = bytes;
  }
  if (cached) rec.bytes[dev] = limit;
  return cudaSuccess;
}

// SMs of the device that was current at the first call.
inline int num_sms() {
  static const int sms = [] {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 152;
  }();
  return sms;
}

inline int check_launch(const char* what, int kernels = 1) {
  add_launches(kernels);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error("%s launch failed: %s", what, cudaGetErrorString(e));
    return FI_ERR_CUDA;
  }
  return FI_OK;
}

// Pixel loads for the three image element types.
__device__ __forceinline__ float load_px(const void* im, int dtype, int64_t idx) {
  switch (dtype) {
    case FI_U8: return (float)__ldg(reinterpret_cast<const uint8_t*>(im) + idx);
    case FI_U16: return (float)__ldg(reinterpret_cast<const uint16_t*>(im) + idx);
    default: return __ldg(reinterpret_cast<const float*>(im) + idx);
  }
}

__device__ __forceinline__ int load_px_int(const void* im, int dtype, int64_t idx) {
  return (dtype == FI_U8) ? (int)__ldg(reinterpret_cast<const uint8_t*>(im) + idx)
                          : (int)__ldg(reinterpret_cast<const uint16_t*>(im) + idx);
}

// Minimum of 16 bytes of pixels (u8: 16, u16: 8, f32: 4 values).
__device__ __forceinline__ float min16(uint4 v, int dtype) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
  if (dtype == FI_F32) {
    return fminf(fminf(__uint_as_float(w[0]), __uint_as_float(w[1])),
                 fminf(__uint_as_float(w[2]), __uint_as_float(w[3])));
  }
  uint32_t m = 0xffffffffu;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (dtype == FI_U16) {
      m = min(m, min(w[k] & 0xffffu, w[k] >> 16));
    } else {
      m = min(m, min(min(w[k] & 0xffu, (w[k] >> 8) & 0xffu),
                     min((w[k] >> 16) & 0xffu, w[k] >> 24)));
    }
  }
  return (float)m;  // exact: below 2^16
}

// The minima (m0, m1) of two images of `count` pixels over thread `tid` of `stride`:
// 16-byte loads, four of each image in flight, when both images are 16-byte aligned.
__device__ __forceinline__ void min_of_pair(const void* im0, const void* im1, int dtype,
                                            int64_t count, int64_t tid, int64_t stride,
                                            float& m0, float& m1) {
  const int esize = (dtype == FI_U8) ? 1 : (dtype == FI_U16 ? 2 : 4);
  int64_t vec = 0;  // pixels read by 16-byte loads
  if ((((uintptr_t)im0 | (uintptr_t)im1) & 15) == 0) {
    const int per = 16 / esize;
    const int64_t nv = count / per;
    const uint4* a = reinterpret_cast<const uint4*>(im0);
    const uint4* b = reinterpret_cast<const uint4*>(im1);
    int64_t i = tid;
    for (; i + 3 * stride < nv; i += 4 * stride) {
      uint4 va[4], vb[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        va[k] = __ldg(a + i + k * stride);
        vb[k] = __ldg(b + i + k * stride);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        m0 = fminf(m0, min16(va[k], dtype));
        m1 = fminf(m1, min16(vb[k], dtype));
      }
    }
    for (; i < nv; i += stride) {
      m0 = fminf(m0, min16(__ldg(a + i), dtype));
      m1 = fminf(m1, min16(__ldg(b + i), dtype));
    }
    vec = nv * per;
  }
  for (int64_t i = vec + tid; i < count; i += stride) {
    m0 = fminf(m0, load_px(im0, dtype, i));
    m1 = fminf(m1, load_px(im1, dtype, i));
  }
}

// Order-preserving float <-> uint32 keys (for atomicMin over floats).
__device__ __forceinline__ uint32_t float_to_key(float f) {
  uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_to_float(uint32_t k) {
  uint32_t u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
  return __uint_as_float(u);
}

// Python/numpy floor division by 2 for int32.
__device__ __forceinline__ int floordiv2(int v) { return (v >= 0) ? (v / 2) : -((-v + 1) / 2); }

// Effective [s, e) of a numpy slice arr[start:stop] (step 1) on an axis of length L.
__host__ __device__ __forceinline__ void slice_bounds(int start, int stop, int L, int* s, int* e) {
  int a = start < 0 ? (start + L < 0 ? 0 : start + L) : (start > L ? L : start);
  int b = stop < 0 ? (stop + L < 0 ? 0 : stop + L) : (stop > L ? L : stop);
  *s = a;
  *e = b > a ? b : a;
}

}  // namespace fi
