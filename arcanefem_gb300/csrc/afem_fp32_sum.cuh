// FP32 sums that many values go through one lane of: compensated, and pairs
// where several partial sums meet.  A kernel that reads whole lines has a lane
// add 14 to 60 rows in turn where a thread per row had a shuffle tree; plain
// additions then carry 1.2 to 1.6 times the tree's rounding error (zero-mean
// sums of 129^2 to 513^2 rows), these 0.6 to 0.9 times.
#pragma once

#include <cmath>

#if defined(__CUDACC__)
#define AFEM_SUM_HD __host__ __device__ __forceinline__
#else
#define AFEM_SUM_HD inline
#endif

namespace afem {

// s + c is the sum; c collects what each addition to s rounds off (Knuth's
// two-sum, exact for any order of magnitudes).
struct Sum32 {
  float s = 0.f, c = 0.f;
  AFEM_SUM_HD void add(float x) {
    const float t = s + x, b = t - s;
    c += (s - (t - b)) + (x - b);
    s = t;
  }
  // a b with what its rounding takes off
  AFEM_SUM_HD void add_product(float a, float b) {
#if defined(__CUDA_ARCH__)
    const float y = __fmul_rn(a, b);   // not to be fused into the additions
#else
    const float y = a * b;
#endif
    add(y);
    c += fmaf(a, b, -y);
  }
  // of an infinite or NaN sum the compensation is NaN
  AFEM_SUM_HD float value() const { return c == c ? s + c : s; }
};

// v[0] + v[STRIDE] + ... (N terms, a power of two) in the order of a warp's shuffle tree
template <int N, int STRIDE = 1>
AFEM_SUM_HD float pair_sum(const float* v) {
  if constexpr (N == 1) return v[0];
  else return pair_sum<N / 2, 2 * STRIDE>(v) + pair_sum<N / 2, 2 * STRIDE>(v + STRIDE);
}

}  // namespace afem
