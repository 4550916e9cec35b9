// Activations as integers: one power-of-two scale and two signed base-256 digits per value, for the int8 tensor-core path.
//
// Over the 128 values of a scale group, x = 2^(m - 14) * (256 * hi + lo) with hi, lo in [-128, 127], where 2^m <= max |x| * (1 +
// 2^-7) < 2^(m+1).  A BF16 value of at least 1/128 of the group's largest magnitude is represented exactly; a smaller one is
// rounded to a multiple of 2^(m-14), an error of at most 2^-15 of that magnitude.  (The factor 1 + 2^-7 keeps the one
// BF16 mantissa whose upper digit would be 128 out of the top binade.)
#pragma once

#include <cuda_bf16.h>
#include <stdint.h>

namespace umaq {

constexpr int kDigitGroup = 128;           // values under one scale: the group of the packed weights' scales

#ifdef __CUDACC__

struct DigitScale {
  float to_int;      // value -> integer
  float to_value;    // integer -> value; NaN where the group holds an infinity or a NaN, which then reaches every sum over it
};
// `max_bits`: the largest magnitude of the group as the bits of a float.  Below 2^-112 the scale stays that of 2^-112 (steps of
// 2^-126): a smaller one would not be a normal float32.
__device__ __forceinline__ DigitScale digit_scale(uint32_t max_bits) {
  const uint32_t e = max(15u, __float_as_uint(__uint_as_float(max_bits) * 1.0078125f) >> 23);   // biased exponent of 2^m
  DigitScale s;
  s.to_int = __uint_as_float((268u - e) << 23);                                  // 2^(14 - m)
  s.to_value = __uint_as_float((e - 14u) << 23);
  if (max_bits >= 0x7f800000u) { s.to_int = 0.f; s.to_value = __uint_as_float(0x7fc00000u); }
  return s;
}
// The integer's upper digit, and the integer itself: its low byte is the lower digit (q - 256 * hi lies in [-128, 127])
__device__ __forceinline__ void to_digits(float value, float to_int, int& hi, int& lo) {
  const int q = __float2int_rn(value * to_int);      // NaN (infinity x 0) converts to 0
  hi = (q + 128) >> 8;
  lo = q;
}

#endif  // __CUDACC__

}  // namespace umaq
