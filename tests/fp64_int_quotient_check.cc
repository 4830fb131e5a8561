// Quotients (i64fp::divisor / div, afem_fp64_int.cuh) against the host's IEEE
// division, bit for bit, over the exponents that quotient() of
// afem_krylov.cuh lets through: zero or within +-400 of one, the dividend's
// zeros of both signs among them; significands of few bits, of all ones and
// random ones, and dividends next to the divisor.  Also that
// i64fp::in_window<400> takes exactly those.
// Prints: mismatches of a / b, wrong range tests.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#include "afem_fp64_int.cuh"

using namespace afem::i64fp;

constexpr int kRange = 400;

static uint64_t bits(double x) { uint64_t u; std::memcpy(&u, &x, 8); return u; }
static double value(uint64_t u) { double x; std::memcpy(&x, &u, 8); return x; }
static bool taken(uint64_t u) { return in_window<kRange>((uint32_t)(u >> 32), (uint32_t)u); }

int main(int argc, char** argv) {
  const long count = argc > 1 ? atol(argv[1]) : 1000000;
  std::mt19937_64 rng(argc > 2 ? atol(argv[2]) : 1);
  auto draw = [&](bool zeros) -> uint64_t {
    const unsigned kind = rng() % 16;
    const uint64_t sign = rng() << 63;
    if (kind == 0 && zeros) return sign;
    uint64_t e = 1023 - kRange + rng() % (2 * kRange + 1);
    if (kind == 1) e = 1023 - kRange;
    if (kind == 2) e = 1023 + kRange;
    if (kind > 12) e = 1023 - 3 + rng() % 6;
    uint64_t m = rng() & kMant;
    if (kind % 4 == 1) m &= ~0ull << (rng() % 52);
    if (kind % 4 == 2) m |= ~(~0ull << (rng() % 52));
    return sign | e << 52 | (m & kMant);
  };
  long bad_div = 0, bad_range = 0;
  for (long i = 0; i < count; ++i) {
    const uint64_t a = draw(true), b = draw(false);
    const Divisor d = divisor(b);
    bad_div += div(operand(a), d) != bits(value(a) / value(b));
    const uint64_t near = (b & ~kMant) | ((b + rng() % 5 - 2) & kMant);
    bad_div += div(operand(near), d) != bits(value(near) / value(b));
    bad_range += !taken(a) || !taken(b);
  }
  for (uint64_t sign : {0ull, 1ull << 63}) {
    const uint64_t lo = (1023ull - kRange) << 52, hi = (1024ull + kRange) << 52;   // the first taken, the first past
    bad_range += !taken(sign) + !taken(sign | lo) + taken(sign | (lo - 1)) + !taken(sign | (hi - 1)) + taken(sign | hi);
    bad_range += taken(sign | 1) + taken(sign | bits(2e-308)) + taken(sign | bits(HUGE_VAL)) + taken(sign | bits(NAN));
  }
  std::printf("%ld %ld\n", bad_div, bad_range);
  return 0;
}
