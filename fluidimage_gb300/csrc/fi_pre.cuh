// Element access of the preprocessing kernels: the four image types, their
// order-preserving integer keys, scipy.ndimage's boundary extension, and
// img - weight * filtered in numpy's result type.
#pragma once

#include <cstdint>

#include "fi_common.cuh"

namespace fi {

__device__ __forceinline__ double load_d(const void* p, int dtype, int64_t i) {
  switch (dtype) {
    case FI_PRE_U8: return (double)static_cast<const uint8_t*>(p)[i];
    case FI_PRE_U16: return (double)static_cast<const uint16_t*>(p)[i];
    case FI_PRE_F32: return (double)static_cast<const float*>(p)[i];
    default: return static_cast<const double*>(p)[i];
  }
}

// Order-preserving unsigned key of an element (floats: the sign-magnitude order
// mapped to unsigned order).  NaN has no place in that order: callers reject
// images with NaN.
__device__ __forceinline__ uint64_t key_of(const void* p, int dtype, int64_t i) {
  switch (dtype) {
    case FI_PRE_U8: return static_cast<const uint8_t*>(p)[i];
    case FI_PRE_U16: return static_cast<const uint16_t*>(p)[i];
    case FI_PRE_F32: {
      const uint32_t u = __float_as_uint(static_cast<const float*>(p)[i]);
      return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
    }
    default: {
      const uint64_t u = (uint64_t)__double_as_longlong(static_cast<const double*>(p)[i]);
      return (u & 0x8000000000000000ull) ? ~u : (u | 0x8000000000000000ull);
    }
  }
}

__device__ __forceinline__ float key_float(uint32_t u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}
__device__ __forceinline__ double key_double(uint64_t u) {
  return __longlong_as_double(
      (long long)((u & 0x8000000000000000ull) ? (u & 0x7fffffffffffffffull) : ~u));
}

__device__ __forceinline__ void store_key(void* p, int dtype, int64_t i, uint64_t k) {
  switch (dtype) {
    case FI_PRE_U8: static_cast<uint8_t*>(p)[i] = (uint8_t)k; break;
    case FI_PRE_U16: static_cast<uint16_t*>(p)[i] = (uint16_t)k; break;
    case FI_PRE_F32: static_cast<float*>(p)[i] = key_float((uint32_t)k); break;
    default: static_cast<double*>(p)[i] = key_double(k);
  }
}

__device__ __forceinline__ int key_bits(int dtype) {
  return dtype == FI_PRE_U8 ? 8 : dtype == FI_PRE_U16 ? 16 : dtype == FI_PRE_F32 ? 32 : 64;
}

// scipy.ndimage boundary extension of index i on an axis of length n; -1 means
// "use cval" (mode 'constant').
__device__ __forceinline__ int64_t extend(int64_t i, int64_t n, int mode) {
  if (i >= 0 && i < n) return i;
  switch (mode) {
    case FI_MODE_NEAREST: return i < 0 ? 0 : n - 1;
    case FI_MODE_WRAP: {
      int64_t r = i % n;
      return r < 0 ? r + n : r;
    }
    case FI_MODE_CONSTANT: return -1;
    case FI_MODE_MIRROR: {
      if (n == 1) return 0;
      const int64_t p = 2 * n - 2;
      int64_t r = i % p;
      if (r < 0) r += p;
      return r < n ? r : p - r;
    }
    default: {  // reflect: d c b a | a b c d | d c b a
      const int64_t p = 2 * n;
      int64_t r = i % p;
      if (r < 0) r += p;
      return r < n ? r : p - 1 - r;
    }
  }
}

// v as a double on the integer pipe (the conversion runs on the narrow FP64 pipe)
__device__ __forceinline__ double int_to_double(int v) {
  if (v == 0) return 0.0;
  const unsigned a = v < 0 ? 0u - (unsigned)v : (unsigned)v;
  const int lz = __clz(a);
  const unsigned frac = (a << lz) << 1;  // the bits after the leading one
  const unsigned hi = ((unsigned)v & 0x80000000u) | ((unsigned)(1023 + 31 - lz) << 20) | (frac >> 12);
  return __hiloint2double((int)hi, (int)(frac << 20));
}

// img - weight * filtered in the numpy result type out_dtype: FI_PRE_F64 / FI_PRE_F32
// (float arithmetic; float32 for float32 images), or the image's integer type (an integer
// weight: wrapping integer arithmetic); clamp: negatives -> 0.
struct Subtract {
  int dtype, out_dtype, clamp;
  double weight;
  int iweight;    // the weight, when exact_int
  int exact_int;  // integer image, float64 result, whole weight up to 2^14: the exact
                  // difference fits 32 bits, so no FP64 instruction is needed

  static inline Subtract make(int dtype, double weight, int out_dtype, int clamp) {
    Subtract s;
    s.dtype = dtype;
    s.out_dtype = out_dtype;
    s.clamp = clamp;
    s.weight = weight;
    const bool whole = weight >= -16384.0 && weight <= 16384.0 && weight == (double)(int)weight;
    s.iweight = whole ? (int)weight : 0;
    s.exact_int = whole && out_dtype == FI_PRE_F64 && (dtype == FI_PRE_U8 || dtype == FI_PRE_U16);
    return s;
  }

  __device__ __forceinline__ double of_ints(int a, int b) const {
    const int v = a - iweight * b;
    return int_to_double(clamp && v < 0 ? 0 : v);
  }

  // element e from the keys (key_of) of the image's and the filtered value
  __device__ __forceinline__ void store_keys(void* out, int64_t e, uint64_t ka, uint64_t kb) const {
    if (exact_int) {
      static_cast<double*>(out)[e] = of_ints((int)ka, (int)kb);
    } else if (dtype == FI_PRE_F32) {
      const float a = key_float((uint32_t)ka), b = key_float((uint32_t)kb);
      if (out_dtype == FI_PRE_F32) {
        const float v = __fsub_rn(a, __fmul_rn((float)weight, b));
        static_cast<float*>(out)[e] = (clamp && v < 0.f) ? 0.f : v;
      } else {
        store(out, e, (double)a, (double)b);
      }
    } else if (dtype == FI_PRE_F64) {
      store(out, e, key_double(ka), key_double(kb));
    } else {
      store(out, e, int_to_double((int)ka), int_to_double((int)kb));
    }
  }

  // element e from the image's and the filtered value (each of the image's type, as a
  // double, exact)
  __device__ __forceinline__ void store(void* out, int64_t e, double a, double b) const {
    if (out_dtype == FI_PRE_F64) {
      // product rounded before the difference, like numpy (no FMA contraction)
      const double v = __dsub_rn(a, __dmul_rn(weight, b));
      static_cast<double*>(out)[e] = (clamp && v < 0.0) ? 0.0 : v;
    } else if (out_dtype == FI_PRE_F32) {
      const float v = __fsub_rn((float)a, __fmul_rn((float)weight, (float)b));
      static_cast<float*>(out)[e] = (clamp && v < 0.f) ? 0.f : v;
    } else {  // integer weight on an integer image: modular arithmetic of the dtype
      const int64_t w = (int64_t)weight;
      const int64_t v = (int64_t)a - w * (int64_t)b;
      if (out_dtype == FI_PRE_U8) static_cast<uint8_t*>(out)[e] = (uint8_t)v;
      else static_cast<uint16_t*>(out)[e] = (uint16_t)v;
    }
  }
};

// Whether the arrays of na bytes at a and nb bytes at b share any.
static inline bool overlap(const void* a, size_t na, const void* b, size_t nb) {
  return (uintptr_t)a < (uintptr_t)b + nb && (uintptr_t)b < (uintptr_t)a + na;
}

static inline size_t element_bytes(int dtype) {
  return dtype == FI_PRE_U8 ? 1 : dtype == FI_PRE_U16 ? 2 : dtype == FI_PRE_F32 ? 4 : 8;
}

static inline int grid_for(int64_t count) {
  const int64_t b = (count + 255) / 256;
  return (int)(b < 152 * 16 ? (b > 0 ? b : 1) : 152 * 16);
}

}  // namespace fi
