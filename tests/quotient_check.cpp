// quotient_from against the division, on the host: random operands over many
// binades, denominators with fractions of nearly all ones, quotients next to
// a rounding boundary, and reciprocal approximations with errors up to 2^-19 of
// either sign.  Prints the number of mismatches.
#include "../solver_b200/csrc/quotient.cuh"

#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>

static double bits(uint64_t b) {
  double d;
  std::memcpy(&d, &b, 8);
  return d;
}
static uint64_t word(double d) {
  uint64_t b;
  std::memcpy(&b, &d, 8);
  return b;
}

int main() {
  std::mt19937_64 gen(20);
  auto real = [&](int lo, int hi, uint64_t fraction) {
    const uint64_t e = 1023 + lo + static_cast<int>(gen() % (hi - lo + 1));
    return bits(e << 52 | (fraction & 0xfffffffffffffull));
  };
  long long bad = 0, done = 0;
  for(int t = 0; t < 6000000; ++t) {
    uint64_t f = gen();
    switch(t % 6) {
      case 1: f = ~(1ull + gen() % 4); break;  // all ones but for the last bits
      case 2: f = ~(gen() % 64); break;
      case 3: f = gen() % 64; break;           // next to a power of two
      case 4: f = ~0ull << (gen() % 52); break;
    }
    double d = real(-46, 499, f);
    if(t & 1) d = -d;
    double n = real(-500, 959, gen());
    if(t % 4 == 1) {  // a quotient next to a midpoint of two doubles
      const double q = real(-100, 100, gen());
      n = std::fabs(std::fma(d, q, 0.5 * d * (std::nextafter(q, 2 * q) - q)));
      if(t % 8 == 1) n = std::nextafter(n, 0.0);
    } else if(t % 4 == 3) {
      n = real(-500, 900, t % 8 == 3 ? ~0ull : 0ull);
    }
    if(!ofb::quotient_in_range(static_cast<int>(word(n) >> 32), static_cast<int>(word(d) >> 32),
                               static_cast<int>(word(d))))
      continue;
    const double err = (t % 5 - 2) * 0.5 * 0x1p-19 * 0.999;
    const double r = (1.0 / d) * (1.0 + err);
    ++done;
    bad += ofb::quotient_from(n, d, r) != n / d;
  }
  std::printf("%lld of %lld\n", bad, done);
  return done > 2000000 && bad == 0 ? 0 : 1;
}
