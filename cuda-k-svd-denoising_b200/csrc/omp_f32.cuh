// The plain FP32 form on the tensor cores (kernels_omp_tc.cu, kernels_omp_tcb.cu):
// an FP16 correlation narrows the atoms down to those that could hold the
// largest FP32 one; what both kernels need for that.
#pragma once

#include "device_util.cuh"

namespace ksvd {

// Rounding of the FP32 sums (the scored one, the atom sums, the mean part) per
// feature, in units of |r| |d|.
constexpr float kF32Slack = 4.0f / 16777216.0f;

// Dictionaries of any scale: the 16-bit one is D / scale (a power of two, atoms of
// norm below 1); outside the range where that is exact enough, dmax is infinite
// and every atom is scored.  sq_bits: bits of the largest |d_a|^2.
struct F32Scale {
  float dmax, scale;
};

KSVD_DEV F32Scale f32_scale(unsigned sq_bits) {
  F32Scale t;
  t.dmax = sqrtf(__uint_as_float(sq_bits));
  t.scale = 1.0f;
  if (t.dmax > 1e-15f && t.dmax < 1e15f) {
    int e;
    frexpf(t.dmax, &e);
    t.scale = ldexpf(1.0f, e);
    t.dmax *= 1.0001f;
  } else {
    t.dmax = __int_as_float(0x7f800000);
  }
  return t;
}

// |c_fp32 - c_fp16| of a residual r for atoms of norm dmax at most: `err` (the
// 16-bit operands) of the part without the mean, `slack` (kF32Slack n) of the
// whole.  The norms are roots of FP32 sums of squares, which leave that range
// for values below 1e-19 or so (and for NaN): the bound is infinite then and
// every atom is scored.
KSVD_DEV float f32_bound(float dmax, float err, float centred, float slack, float norm) {
  return norm > 1e-15f ? dmax * (err * centred + slack * norm) : __int_as_float(0x7f800000);
}

}  // namespace ksvd
