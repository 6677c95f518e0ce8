// f32_round.cuh -- FP32 values of FP64 operands on the integer pipe.  A conversion to or
// from FP64 is an FP64 instruction (16 clocks of an SM for a warp), as is a difference.
#pragma once
#include "emu64.cuh"

namespace dem {

// |a - b| for finite a, b in FP32 without the FP64 pipe: the significands aligned to
// the larger exponent (bits of the smaller operand below the larger one's last are
// dropped: an error of at most 2^-52 of the larger operand) and subtracted as
// integers, the magnitude rounded to FP32 in two halves (relative 2^-22) and scaled
// by the power of two.  ok is cleared outside [2^-48, 2^112) (zeros aside); top
// becomes the largest biased exponent met.
__device__ __forceinline__ float diff_f32(double a, double b, bool& ok, uint32_t& top) {
  const uint64_t ua = emu_bits(a), ub = emu_bits(b);
  const uint32_t ea = (uint32_t)(ua >> 52) & 0x7ffu, eb = (uint32_t)(ub >> 52) & 0x7ffu;
  const uint32_t e = ea > eb ? ea : eb;
  const uint64_t frac = 0xfffffffffffffull;
  const uint32_t sa = e - ea, sb = e - eb;
  const int64_t ma = sa < 64u ? (int64_t)(((ua & frac) | (1ull << 52)) >> sa) : 0;
  const int64_t mb = sb < 64u ? (int64_t)(((ub & frac) | (1ull << 52)) >> sb) : 0;
  const int64_t d = ((int64_t)(ua ^ ub) < 0) ? ma + mb : ma - mb;
  const uint64_t m = (uint64_t)(d < 0 ? -d : d);
  ok = ok && e - (1075u - 100u) < 160u;
  top = top > e ? top : e;
  const float f = (float)(uint32_t)(m >> 32) * 4294967296.f + (float)(uint32_t)m;
  return f * __uint_as_float((e - 1075u + 127u) << 23);
}
// x > 0 cut to FP32 on the integer pipe (relative error below 2^-23, downwards)
__device__ __forceinline__ float trunc_f32(double x, bool& ok) {
  const uint64_t u = emu_bits(x);
  const uint32_t e = (uint32_t)(u >> 52);
  ok = ok && e - (1023u - 100u) < 200u;
  return __uint_as_float(((e - 1023u + 127u) << 23) | ((uint32_t)(u >> 29) & 0x7fffffu));
}

// Round to nearest even, (float)x, on the integer pipe (a conversion is an FP64
// instruction): the 29 low bits of the significand rounded off the packed exponent
// and significand.  Outside the normal FP32 range the conversion itself.
__device__ __forceinline__ float f32_rn(double x) {
  const uint64_t u = emu_bits(x);
  const uint32_t e = (uint32_t)(u >> 52) & 0x7ffu;
  if (e - (1023u - 126u) >= 253u) return (u << 1) == 0 ? __uint_as_float((uint32_t)(u >> 32)) : (float)x;
  const uint64_t m = u & 0x7fffffffffffffffull;
  const uint64_t r = (m + 0x0fffffffull + ((m >> 29) & 1ull)) >> 29;
  return __uint_as_float((uint32_t)(r - ((uint64_t)(1023 - 127) << 23)) | ((uint32_t)(u >> 32) & 0x80000000u));
}

}  // namespace dem
