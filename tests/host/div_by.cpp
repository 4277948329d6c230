// div_by (athenak_b200/csrc/dustb_div.cuh) against the division: equal bits over its range.
// Usage: div_by COUNT SEED; prints the number of quotients compared, exits 1 at the first that
// differs.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "../../athenak_b200/csrc/dustb_div.cuh"

static uint64_t state;
static uint64_t next() {                          // SplitMix64
  uint64_t z = (state += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// a magnitude within 2^-hi .. 2^hi whose mantissa is random, or a few bits from a power of two on
// either side, or has a run of ones or zeros at its end
static double draw(int hi) {
  uint64_t m = next() & 0xFFFFFFFFFFFFFull;
  const uint64_t low = (1ull << (1 + next() % 51)) - 1;
  switch (next() % 6) {
    case 0: m = next() % 8; break;
    case 1: m = 0xFFFFFFFFFFFFFull - next() % 8; break;
    case 2: m |= low; break;
    case 3: m &= ~low; break;
    default: break;
  }
  const int e = (int)(next() % (2 * hi + 1)) - hi;
  const uint64_t b = ((uint64_t)(1023 + e) << 52) | m;
  double x;
  std::memcpy(&x, &b, 8);
  return x;
}

static bool same(double n, double d) {
  const double q = dustb::div_by(n, d, 1.0 / d), want = n / d;
  if (n == 0.0) return q == 0.0;
  if (std::memcmp(&q, &want, 8) == 0) return true;
  std::printf("%a / %a: %a, %a wanted\n", n, d, q, want);
  return false;
}

int main(int argc, char **argv) {
  const long long count = argc > 1 ? std::atoll(argv[1]) : 1000000;
  state = argc > 2 ? std::strtoull(argv[2], nullptr, 10) : 1;
  for (long long k = 0; k < count; ++k) {
    const int hi = (k & 1) ? 498 : 30;            // (2^498 = 8e149)
    const double d = draw(hi), n = draw(hi) * ((next() & 1) ? 1.0 : -1.0);
    if (!same(n, d)) return 1;
    // numerators about multiples of the divisor, whose quotients lie near the middle of two
    // doubles or on one
    const double m = d * (1.0 + (double)(next() % 1000) * 0x1p-52) * (double)(1 + next() % 4096);
    if (!same(m, d) || !same(std::nextafter(m, 0.0), d)) return 1;
  }
  if (!same(0.0, 0.01) || !same(-0.0, 0.01)) return 1;
  std::printf("%lld quotients\n", 3 * count + 2);
  return 0;
}
