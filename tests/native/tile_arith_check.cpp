// Host check of the integer forms that the tile walk's erosion adds to
// fs_bits.h: add_const_rn_bits (the uplift) against the FP64 addition, and
// quotient_tabled_bits against the IEEE division, on every result they accept:
// random operands, all exponent gaps, operands next to rounding ties and
// midpoints, carries, both ends of the binades, negative, huge, subnormal and
// non-finite operands. Also that they accept what they are for: every x at or
// above c's binade but 1 in 100, and all but 1 in 10^5 quotients of ordinary
// operands (a refused quotient costs a warp the FP64 division).
// Usage: tile_arith_check <cases> <seed>; exit 1 on the first mismatch.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#include "../../barnes2019-landscape_gb300/csrc/fs_bits.h"

static double dbl(uint64_t u) { double d; std::memcpy(&d, &u, 8); return d; }
static uint64_t bits(double d) { uint64_t u; std::memcpy(&u, &d, 8); return u; }

int main(int argc, char **argv) {
  const long n = argc > 1 ? std::atol(argv[1]) : 1000000;
  std::mt19937_64 g(argc > 2 ? std::strtoull(argv[2], nullptr, 10) : 1);
  const uint64_t kFrac = (1ull << 52) - 1;
  auto frac = [&]() -> uint64_t {
    switch (g() % 5) {
      case 0: return 0;
      case 1: return kFrac - (g() & 3);
      case 2: return g() & 7;
      case 3: return (g() & kFrac) & ~((1ull << (g() % 52)) - 1);
      default: return g() & kFrac;
    }
  };
  long want_add = 0, got_add = 0, want_q = 0, got_q = 0;
  for (long i = 0; i < n; i++) {
    // the uplift
    const uint64_t ec = i % 3 ? 1023 + g() % 12 : 1 + g() % 1900;
    const uint64_t c = ec << 52 | frac();
    uint64_t ex = ec + g() % 60;
    if (i % 7 == 0) ex = g() % 2048;
    if (ex > 2047) ex = 2047;
    uint64_t x = ex << 52 | frac();
    if (i % 4 == 1 && ex >= ec && ex - ec < 53 && ex < 2046) {  // next to a tie
      const uint64_t low = c & ((2ull << (ex - ec)) - 1);
      x = (x & ~0xFFull) | (low & 0xFF);
    }
    if (i % 11 == 0) x |= 1ull << 63;
    const uint64_t s = fs::add_const_rn_bits(x, c);
    {  // an ordinary elevation and uplift
      const uint64_t co = i & 1 ? bits(2.0) : 1020ull + g() % 10 << 52 | (g() & kFrac);
      const uint64_t o = ((co >> 52) + g() % 40) << 52 | (g() & kFrac);
      const uint64_t so = fs::add_const_rn_bits(o, co);
      ++want_add;
      got_add += so != 0;
      if (so && so != bits(dbl(o) + dbl(co))) {
        std::printf("MISMATCH add x=%a c=%a\n", dbl(o), dbl(co));
        return 1;
      }
    }
    if (s && s != bits(dbl(x) + dbl(c))) {
      std::printf("MISMATCH add x=%a c=%a\n", dbl(x), dbl(c));
      return 1;
    }
    // the quotient
    double D;
    switch (i % 5) {
      case 0: D = 1.0 + std::ldexp((double)(g() >> 11), -53 + (int)(g() % 80) - 40); break;
      case 1: D = dbl((uint64_t)(1023 + g() % 40) << 52 | frac()); break;
      case 2: D = 1.0 + std::ldexp((double)(g() >> 11), -60); break;
      case 3: D = dbl((uint64_t)(g() % 2048) << 52 | frac()); break;
      default: D = -dbl((uint64_t)(1023 + g() % 40) << 52 | frac()); break;
    }
    if (D == 0 || !std::isfinite(D)) continue;
    double num;
    const bool plain = i % 5 == 2;
    if (i & 1) {  // next to a midpoint
      const double m = dbl((uint64_t)(1023 + (int)(g() % 200) - 100) << 52 | frac());
      int e;
      std::frexp(m, &e);
      num = std::fma(D, m, D * std::ldexp(1.0, e - 54));
      num = dbl(bits(num) + (int)(g() % 5) - 2);
    } else if (i % 3 == 0 && !plain) {
      num = dbl((uint64_t)(g() % 2048) << 52 | frac());
    } else {
      num = dbl((uint64_t)(1023 + (int)(g() % 60) - 40) << 52 | (g() & kFrac));
    }
    if (g() & 1) num = -num;
    if (!std::isfinite(num)) continue;
    const double q0 = num * -(1.0 / D);
    const uint64_t q = fs::quotient_tabled_bits(bits(q0), bits(num), bits(D));
    if (plain && !(i & 1)) {
      ++want_q;
      got_q += q != 0;
    }
    if (q && q != bits(-(num / D))) {
      std::printf("MISMATCH quotient num=%a D=%a\n", num, D);
      return 1;
    }
  }
  if (got_add * 100 < want_add * 99 || (want_q - got_q) * 100000 > want_q) {
    std::printf("accepted %ld of %ld sums, %ld of %ld quotients\n", got_add, want_add, got_q, want_q);
    return 1;
  }
  std::printf("%ld cases: %ld of %ld sums and %ld of %ld quotients accepted, all equal to FP64\n", n,
              got_add, want_add, got_q, want_q);
  return 0;
}
