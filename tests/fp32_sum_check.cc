// Sums of afem_fp32_sum.cuh against sums in double, and against those of a
// thread per value and a tree over a warp's lanes in plain additions.  A block
// of 8 warps, each lane of a warp `chain` values in turn (Sum32) and the
// warps' sums in pairs; the tree takes the same values 32 at a time.
// Prints, for each chain: RMS error of the compensated sums, of the tree's;
// then 1 for each special value that comes out as plain additions give it.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <limits>
#include <random>
#include <vector>

#include "afem_fp32_sum.cuh"

using afem::Sum32;
using afem::pair_sum;

int main(int argc, char** argv) {
  const int trials = argc > 1 ? atoi(argv[1]) : 400;
  std::mt19937 rng(argc > 2 ? atoi(argv[2]) : 1);
  std::normal_distribution<float> normal;
  for (int chain : {1, 2, 14, 32, 64, 217}) {
    double mine = 0.0, tree = 0.0;
    for (int trial = 0; trial < trials; ++trial) {
      const int n = 8 * chain;
      std::vector<float> a(n), b(n);
      double want = 0.0;
      float warps[8];
      for (int i = 0; i < n; ++i) {
        a[i] = normal(rng);
        b[i] = normal(rng);
        want += (double)a[i] * b[i];
      }
      for (int w = 0; w < 8; ++w) {
        Sum32 s;
        for (int i = 0; i < chain; ++i) s.add_product(a[w * chain + i], b[w * chain + i]);
        warps[w] = s.value();
      }
      const double e = pair_sum<8>(warps) - want;
      std::vector<float> lane(a.size());
      for (int i = 0; i < n; ++i) lane[i] = a[i] * b[i];
      while (lane.size() > 1) {   // the shuffle tree of a thread per value
        const size_t half = (lane.size() + 1) / 2;
        for (size_t i = 0; i + half < lane.size(); ++i) lane[i] += lane[i + half];
        lane.resize(half);
      }
      const double t = lane[0] - want;
      mine += e * e;
      tree += t * t;
    }
    std::printf("%.9e %.9e\n", std::sqrt(mine / trials), std::sqrt(tree / trials));
  }
  const float inf = std::numeric_limits<float>::infinity(), nan = std::nanf("");
  auto sum = [](std::initializer_list<float> v) {
    Sum32 s;
    for (float x : v) s.add(x);
    return s.value();
  };
  Sum32 product;
  product.add_product(inf, 2.f);
  const float zeros[4] = {1e-45f, 0.f, -1e-45f, 0.f};
  std::printf("%d %d %d %d %d %d\n", sum({1.f, inf, 2.f}) == inf, sum({-inf, 1.f}) == -inf,
              (int)std::isnan(sum({inf, -inf, 1.f})), (int)std::isnan(sum({1.f, nan})), product.value() == inf,
              pair_sum<4>(zeros) == 0.f && sum({}) == 0.f);
  return 0;
}
