// Products of unpacked operands (i64fp::operand / mul, afem_fp64_int.cuh)
// against the host's IEEE multiplication, bit for bit, for every operand the
// range test i64fp::in_window accepts: zeros of both signs, exponents over the
// whole window, significands of few bits (exact products and ties), of all
// ones and random ones, and products of a product with an operand.
// Quotients (i64fp::div) the same, over dividends that include the divisor's
// own significand and its neighbours, and by the constant divisor 6.
// Prints: mismatches of a * b, of (a * b) * c, of a / b, wrong range tests.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#include "afem_fp64_int.cuh"

using namespace afem::i64fp;

static uint64_t bits(double x) { uint64_t u; std::memcpy(&u, &x, 8); return u; }
static double value(uint64_t u) { double x; std::memcpy(&x, &u, 8); return x; }

int main(int argc, char** argv) {
  const long count = argc > 1 ? atol(argv[1]) : 1000000;
  std::mt19937_64 rng(argc > 2 ? atol(argv[2]) : 1);
  auto draw = [&]() -> uint64_t {
    const unsigned kind = rng() % 16;
    const uint64_t sign = rng() << 63;
    if (kind == 0) return sign;
    uint64_t e = 1023 - kWindow + rng() % (2 * kWindow + 1);
    if (kind < 8) e = 1023 - 12 + rng() % 24;
    if (kind == 1) e = 1023 - kWindow;
    if (kind == 2) e = 1023 + kWindow;
    uint64_t m = rng() & kMant;
    if (kind % 4 == 1) m &= ~0ull << (rng() % 52);
    if (kind % 4 == 2) m |= ~(~0ull << (rng() % 52));
    return sign | e << 52 | (m & kMant);
  };
  long bad2 = 0, bad3 = 0, bad_div = 0, bad_range = 0;
  const Divisor six = divisor(bits(6.0));
  for (long i = 0; i < count; ++i) {
    const uint64_t a = draw(), b = draw(), c = draw();
    const double ab = value(a) * value(b);
    const uint64_t r = mul(operand(a), operand(b));
    bad2 += r != bits(ab);
    bad3 += mul(operand(r), operand(c)) != bits(ab * value(c));
    if (b << 1) {
      const Divisor d = divisor(b);
      const uint64_t near = (a & ~kMant) | ((b + rng() % 5 - 2) & kMant);   // a significand next to the divisor's
      bad_div += div(operand(a), d) != bits(value(a) / value(b));
      if (near << 1 >> 53) bad_div += div(operand(near), d) != bits(value(near) / value(b));
    }
    bad_div += div(operand(a), six) != bits(value(a) / 6.0);
    bad_range += !in_window(a) || !in_window(b);
  }
  const double out[] = {value((1023ull - kWindow - 1) << 52), value((1023ull + kWindow + 1) << 52), 5e-324, 2e-308,
                        HUGE_VAL, NAN};
  for (double x : out) bad_range += in_window(bits(x)) || in_window(bits(-x));
  std::printf("%ld %ld %ld %ld\n", bad2, bad3, bad_div, bad_range);
  return 0;
}
