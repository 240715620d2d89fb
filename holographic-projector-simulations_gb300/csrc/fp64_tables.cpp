// fp64_tables.cpp -- the tables of the fixed-point FP64 kernel (fp64_fixed.cuh), on the host.
#include "fp64_tables.h"

#include <math.h>

namespace holo {

static const long double kTwoPi = 6.283185307179586476925286766559005768394L;

// cos and sin of 2 pi i / 1024 from the first octant (long double has 64 or 113 bits).
static void circle(int i, long double *cosine, long double *sine) {
  constexpr int n = fixed::kTrigEntries;
  const int quadrant = i / (n / 4), j = i % (n / 4);
  const bool upper = j > n / 8;  // the angle's complement in the quadrant
  const long double a = kTwoPi * (upper ? n / 4 - j : j) / n;
  long double c = upper ? sinl(a) : cosl(a), s = upper ? cosl(a) : sinl(a);
  for (int q = 0; q < quadrant; ++q) {
    const long double t = c;
    c = -s;
    s = t;
  }
  *cosine = c;
  *sine = s;
}

void fill_trig(fixed::TrigEntry *out) {
  for (int i = 0; i < fixed::kTrigEntries; ++i) {
    long double c, s;
    circle(i, &c, &s);
    fixed::TrigEntry &e = out[i];
    e.c = (int64_t)llroundl(c * 0x1p62L);
    e.s = (int64_t)llroundl(s * 0x1p62L);
    e.ch = (float)c;
    e.cl = (float)(c - (long double)e.ch);
    e.sh = (float)s;
    e.sl = (float)(s - (long double)e.sh);
  }
}

void fill_polar(fixed::PolarEntry *out) {
  constexpr int n = fixed::kTrigEntries;
  static_assert(n == 2 * fixed::kPolarHalf, "the same angles");
  for (int i = -fixed::kPolarHalf; i <= fixed::kPolarHalf; ++i) {
    long double c, s;
    circle((i + n) % n, &c, &s);
    const long double a = kTwoPi * i / n;
    fixed::PolarEntry &e = out[i + fixed::kPolarHalf];
    e = {};
    e.c = (double)c;
    e.s = (double)s;
    e.a = (double)a;
    e.cl = (float)(c - (long double)e.c);
    e.sl = (float)(s - (long double)e.s);
    e.al = (float)(a - (long double)e.a);
  }
}

// 2^(e - 52) / 2 pi mod 1 for every exponent: windows of the bits of 1 / 2 pi.
void fill_turns(fixed::TurnWords *out) {
  static const uint32_t inv_two_pi[4] = {0x28BE60DBu, 0x9391054Au, 0x7F09D5F4u, 0x7D4D3770u};
  for (int e = fixed::kTurnLow; e <= fixed::kTurnHigh; ++e)
    for (int w = 0; w < 4; ++w) {
      uint32_t v = 0;
      for (int b = 0; b < 32; ++b) {
        const int at = 32 * w + b + e - 52;  // bit of weight 2^-(at + 1)
        const uint32_t bit = at >= 0 && at < 128 ? inv_two_pi[at / 32] >> (31 - at % 32) & 1u : 0u;
        v = v << 1 | bit;
      }
      out[e - fixed::kTurnLow].k[w] = v;
    }
}

}  // namespace holo
