// The stop test of the tensor-core OMP (|r| < 1e-3, cublas_matrix_omp.cu:218)
// at its threshold.  Their residual pass sums |r|^2 in an order of its own;
// where the order could decide, the norm is formed again in the order that
// the test is defined by.
#pragma once

#include "device_util.cuh"

namespace ksvd {

// Order of |r|^2: kStopQuarters, the 16-bit forms' (the 8-feature chunks of a
// padded row in four parts); kStopRanges, kernels_omp.cu's (eight ranges of
// features); above, kernels_omp_stream.cu's (chunks of that many features, each
// dealt to eight sums in turn).
constexpr int kStopQuarters = -1, kStopRanges = 0;

// The FP32 form stops where the FP32 kernel that it stands in for does.
inline int omp_stop_order(TcForm form, int n, int K, int L) {
  if (form != TcForm::kFp32) return kStopQuarters;
  if (omp_fp32_supported(n, K, L)) return kStopRanges;
  return omp_stream_supported(n, K, L) ? omp_stream_chunk(n, K, L) : kStopQuarters;
}

// The sums of |r|^2 differ by less than 5e-5 of it (n <= 512 terms, none
// negative, so at most n 2^-24 each).
KSVD_DEV bool stop_near(float norm2) { return fabsf(norm2 - 1.0e-6f) < 5.0e-11f; }

// |r|^2 of r = y - sum_s g_s d_s (s ascending), summed in `order`.  One thread;
// rare, so kept out of the kernels' registers.
static __device__ __noinline__ float stop_norm2(const float* y, const float* D, int n, const int* S, const float* g,
                                                int cnt, int order) {
  auto sum = [&](int k0, int k1, int step) {
    float t = 0.0f;
    for (int k = k0; k < k1; k += step) {
      float r = __ldg(y + k);
      for (int s = 0; s < cnt; ++s) r = fmaf(-g[s], __ldg(D + int64_t(S[s]) * n + k), r);
      t = fmaf(r, r, t);
    }
    return t;
  };
  float total = 0.0f;
  if (order == kStopQuarters) {
    const int nkc = 2 * ((n + 15) / 16);
    for (int q = 0; q < 4; ++q) total += sum(8 * ((nkc * q) / 4), min(n, 8 * ((nkc * (q + 1)) / 4)), 1);
  } else if (order == kStopRanges) {
    const int rows = (n + 7) / 8;
    for (int w = 0; w < 8; ++w) total += sum(w * rows, min(n, (w + 1) * rows), 1);
  } else {
    for (int w = 0; w < 8; ++w) {
      float part = 0.0f;
      for (int k0 = 0; k0 < n; k0 += order) part += sum(k0 + w, min(n, k0 + order), 8);
      total += part;
    }
  }
  return total;
}

}  // namespace ksvd
