// fp64_fixed.cuh -- the per-pair arithmetic of HOLO_FP64 on the integer and FP32 pipes.
//
// GB300 executes 1.7 FP64 lane operations per clock and SM against ~60 integer and 128 FP32 ones,
// so all of a term (cuda/superposition.cu:35-51) but the difference, the sum of squares and
// the two roundings of the phase runs outside the FP64 pipe:
//   - the distance, the correctly rounded square root, from an FP32 estimate, one integer
//     Newton step and the exact remainder;
//   - the phase in turns, a 53 x 117 bit product with 1 / 2 pi, as a 64-bit fraction;
//   - sine and cosine from a table of 1024 angles and a rotation by the rest in float-float
//     arithmetic, as 62-bit fractions (error below 2^-55);
//   - amplitude / distance and the products as 64-bit fixed-point numbers, summed exactly.
// Everything up to the phase is bit for bit what FP64 instructions give.  The functions are host
// code too (tests compile them), except where they call the MUFU estimate of 1 / sqrt.
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define HOLO_HD __host__ __device__ __forceinline__
#else
#define HOLO_HD inline
#endif

namespace holo {
namespace fixed {

HOLO_HD uint32_t mulhi32(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
  return __umulhi(a, b);
#else
  return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
HOLO_HD int64_t mulhi64(int64_t a, int64_t b) {
#ifdef __CUDA_ARCH__
  return __mul64hi(a, b);
#else
  return (int64_t)(((__int128)a * b) >> 64);
#endif
}
HOLO_HD float as_float(uint32_t b) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(b);
#else
  float f;
  memcpy(&f, &b, 4);
  return f;
#endif
}
HOLO_HD uint32_t as_bits(float f) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(f);
#else
  uint32_t b;
  memcpy(&b, &f, 4);
  return b;
#endif
}
HOLO_HD int round_int(float x) {
#ifdef __CUDA_ARCH__
  return __float2int_rn(x);
#else
  return (int)lrintf(x);
#endif
}
// Each operation rounded on its own.
HOLO_HD float fmul(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fmul_rn(a, b);
#else
  return a * b;
#endif
}
HOLO_HD float fadd(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fadd_rn(a, b);
#else
  return a + b;
#endif
}

// Distance as an integer and its reciprocal's FP32 parts: distance = d 2^(q - 52), d in
// [2^52, 2^53]; 1 / sqrt(x) = y0 + yl to 2^-45 for the x in [1, 4) that d is the root of.
struct Root {
  uint64_t d;
  int q;
  float y0, yl;
};

// Correctly rounded square root of s = hi:lo (a normal positive double).  y0_of: an estimate of
// 1 / sqrt of a float in [1, 4), good to 2^-21.
template <typename F>
HOLO_HD Root root(uint32_t hi, uint32_t lo, F y0_of) {
  Root r;
  const int e = (int)(hi >> 20) - 1023, odd = e & 1;
  r.q = e >> 1;
  // x = x_hi + x_lo in [1, 4): the top 23 bits of the fraction and the 29 below them
  const float xh = as_float((((hi << 3) | (lo >> 29)) & 0x7fffffu) | (uint32_t)(127 + odd) << 23);
  const float xl = fmul((float)(int)(lo & 0x1fffffffu), odd ? 0x1p-51f : 0x1p-52f);
  const float y0 = y0_of(xh);
  // t = 1 - x y0^2 to 2^-46, 1 / sqrt(x) = y0 (1 + t / 2 + 3 t^2 / 8)
  const float p = fmul(y0, y0), pe = fmaf(y0, y0, -p);
  const float t = fmaf(-xl, p, fmaf(-xh, pe, fmaf(-xh, p, 1.f)));
  r.y0 = y0;
  r.yl = fmul(y0, fmul(t, fmaf(0.375f, t, 0.5f)));
  // sqrt(x) = x / sqrt(x) = gh + gl, as an integer in units of 2^-50 off by less than 2^9
  const float gh = fmul(xh, y0);
  const float gl = fmaf(xh, r.yl, fmaf(xl, y0, fmaf(xh, y0, -gh)));
  const int64_t g = ((int64_t)round_int(fmul(gh, 0x1p29f)) << 21) + round_int(fmul(gl, 0x1p50f));
  // remainder x - g^2 in units of 2^-100: it fits 64 bits, so the low 64 bits are enough
  const uint32_t g0 = (uint32_t)g, g1 = (uint32_t)((uint64_t)g >> 32);
  const uint64_t sq = (uint64_t)g0 * g0 + ((uint64_t)(2u * g0 * g1) << 32);
  const int64_t rem = (int64_t)(((uint64_t)((lo << odd) << 16) << 32) - sq);
  // Newton step in units of 2^-52, and what it leaves in units of 2^-104 (small again: mod 2^64)
  const int step = round_int(fmul((float)(int)(rem >> 32), fmul(y0, 0x1p-17f)));
  int64_t d = 4 * g + step;
  const int64_t left = (int64_t)(16 * (uint64_t)rem - (uint64_t)((int64_t)step * (8 * g + step)));
  // nearest: -d < left <= d
  if (left > d) ++d;
  else if (left + d <= 0) --d;
  r.d = (uint64_t)d;
  return r;
}

// Words of 2^(e - 52) / 2 pi mod 1, weights 2^-32, 2^-64, 2^-96 and 2^-128.
struct TurnWords {
  uint32_t k[4];
};
constexpr int kTurnLow = -20, kTurnHigh = 43;  // exponents of the phases the table covers
constexpr int kTurnEntries = kTurnHigh - kTurnLow + 1;

// A normal double hi:lo (its exponent's words k) in turns mod 1, in units of 2^-64.
HOLO_HD uint64_t turns(uint32_t hi, uint32_t lo, const uint32_t k0, const uint32_t k1,
                       const uint32_t k2, const uint32_t k3) {
  const uint32_t m1 = (hi & 0xfffffu) | 0x100000u, m0 = lo;
  uint64_t t = ((uint64_t)(m0 * k0 + m1 * k1) << 32) + (uint64_t)m0 * k1 + (uint64_t)m1 * k2;
  t += (uint64_t)mulhi32(m0, k2) + mulhi32(m1, k3);
  return (int32_t)hi < 0 ? 0 - t : t;
}

// One of 1024 angles: cosine and sine in units of 2^-62 and as float-float pairs.
struct TrigEntry {
  int64_t c, s;
  float ch, cl, sh, sl;
};
constexpr int kTrigBits = 10, kTrigEntries = 1 << kTrigBits;

// corr = ah bh + ... of two float-float products a b + c d with |a b| >= |c d|, as (h, l).
HOLO_HD void dot2(float ah, float al, float bh, float bl, float ch, float cl, float dh, float dl,
                  float *h, float *l) {
  const float p = fmul(ah, bh), pe = fmaf(al, bh, fmaf(ah, bl, fmaf(ah, bh, -p)));
  const float r = fmul(ch, dh), re = fmaf(cl, dh, fmaf(ch, dl, fmaf(ch, dh, -r)));
  const float s = fadd(p, r), bb = fadd(s, -p);
  const float e = fadd(fadd(p, -fadd(s, -bb)), fadd(r, -bb));
  *h = s;
  *l = fadd(e, fadd(pe, re));
}

// h + l (|h| < 2^-8, |l| < 2^-30) in units of 2^-62: h's multiple of 2^-30 from the bits of a sum
// whose last place that is, the rest by a conversion.
HOLO_HD int64_t to_62(float h, float l) {
  const float big = 0x1.8p-7f;  // last place 2^-30
  const float u = fadd(h, big);
  const int i1 = (int)(as_bits(u) - as_bits(big));
  const float rest = fadd(fadd(h, -fadd(u, -big)), l);
  return ((int64_t)i1 << 32) + ((int64_t)round_int(fmul(rest, 0x1p60f)) << 2);
}

// cos and sin of 2 pi t / 2^64 in units of 2^-62; entry: of index (t + 2^53) >> 54 (mod 1024).
HOLO_HD uint32_t trig_index(uint64_t t) {
  return (uint32_t)((t + (1ull << (63 - kTrigBits))) >> (64 - kTrigBits));
}
HOLO_HD void cos_sin(uint64_t t, uint32_t index, const TrigEntry &E, int64_t *c, int64_t *s) {
  // delta = 2 pi (t - index 2^54) / 2^64, |delta| <= 2 pi / 2048: g = ga 2^30 + gb
  const int64_t g = (int64_t)(t - ((uint64_t)index << (64 - kTrigBits)));
  const float ga = (float)(int)(g >> 30), gb = fmul((float)(int)(g & 0x3fffffff), 0x1p-30f);
  // 2 pi 2^-34 as a float-float pair
  const float k = 0x1.921fb6p-32f, kl = -0x1.777a5cp-57f;
  const float dh0 = fmul(ga, k);
  const float dl0 = fmaf(gb, k, fmaf(ga, kl, fmaf(ga, k, -dh0)));
  const float dh = fadd(dh0, dl0), dl = fadd(dl0, -fadd(dh, -dh0));
  // z = delta^2, 1 - cos = z / 2 - z^2 / 24 + z^3 / 720
  const float zh = fmul(dh, dh), zl = fmaf(fadd(dh, dh), dl, fmaf(dh, dh, -zh)), zz = fmul(zh, zh);
  const float ch = fmul(0.5f, zh), cl = fmaf(zz, fmaf(zh, 1.f / 720.f, -1.f / 24.f), fmul(0.5f, zl));
  // sin = delta - delta v, v = z / 6 - z^2 / 120
  const float sixth = 0x1.555556p-3f, sixth_l = -0x1.555556p-28f;
  const float vh = fmul(zh, sixth);
  const float vl = fmaf(-zz, 1.f / 120.f,
                        fmaf(zl, sixth, fmaf(zh, sixth_l, fmaf(zh, sixth, -vh))));
  const float wh = fmul(dh, vh), wl = fmaf(dl, vh, fmaf(dh, vl, fmaf(dh, vh, -wh)));
  const float sh = fadd(dh, -wh), sl = fadd(fadd(fadd(dh, -sh), -wh), fadd(dl, -wl));
  float h, l;
  // cos(a + delta) = cos a - (sin a sin delta + cos a (1 - cos delta))
  dot2(E.sh, E.sl, sh, sl, E.ch, E.cl, ch, cl, &h, &l);
  *c = E.c - to_62(h, l);
  // sin(a + delta) = sin a + (cos a sin delta - sin a (1 - cos delta))
  dot2(E.ch, E.cl, sh, sl, -E.sh, -E.sl, ch, cl, &h, &l);
  *s = E.s + to_62(h, l);
}

// 1 / sqrt(x) of the rounded root d (distance = d 2^(q - 52)) in units of 2^-62: 2^(-q) times it is
// 1 / distance.  One Newton step on the FP32 estimate with the exact residual 1 - d y.
HOLO_HD int64_t reciprocal(const Root &r) {
  const int64_t y = ((int64_t)round_int(fmul(r.y0, 0x1p29f)) << 23) +
                    ((int64_t)round_int(fmul(r.yl, 0x1p50f)) << 2);  // units of 2^-52
  const uint32_t y0 = (uint32_t)y, y1 = (uint32_t)((uint64_t)y >> 32);
  const uint32_t d0 = (uint32_t)r.d, d1 = (uint32_t)(r.d >> 32);
  const uint64_t low = (uint64_t)d0 * y0 + ((uint64_t)(d0 * y1 + d1 * y0) << 32);
  const int64_t res = (int64_t)(0 - low);  // 2^104 - d y, fits 64 bits
  return (y << 10) + round_int(fmul((float)(int)(res >> 32), fmul(r.y0, 0x1p-10f)));
}

// One of 1025 angles a = 2 pi i / 1024, i = -512 .. 512: cosine, sine and angle as a double and
// what that leaves.
struct PolarEntry {
  double c, s, a;
  float cl, sl, al, none[3];
};
constexpr int kPolarHalf = 512, kPolarEntries = 2 * kPolarHalf + 1;

HOLO_HD uint64_t double_bits(double x) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t b;
  memcpy(&b, &x, 8);
  return b;
#endif
}
HOLO_HD double as_double(uint64_t b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)b);
#else
  double x;
  memcpy(&x, &b, 8);
  return x;
#endif
}

// x of exponent field e below or equal to `top`, divided by 2^(top - 1023), cut to FP32.
HOLO_HD float cut_float(uint64_t bits, int e, int top) {
  const uint32_t sign = (uint32_t)(bits >> 32) & 0x80000000u;
  const uint32_t mant = (uint32_t)(bits >> 29) & 0x7fffffu;
  return as_float(top - e > 100 ? sign : sign | (uint32_t)(e - top + 127) << 23 | mant);
}

// Modulus and angle of x + i y: a table angle near the FP32 estimate, the point turned back by
// it (the cancelling component to 2^-60), the small angle left by its series; the modulus as the
// rounded root of the rounded sum of squares.  24 FP64 operations instead of the ~90 of a hypot
// and an atan2.
// False, and nothing written, for what is not well inside the exponent range (zeros, infinities,
// NaN, components more than 2^500 apart).  angle_of(y, x): atan2 to 2^-16; inverse_of: 1 / x to 2^-20; y0_of: as in root().
template <typename A, typename R, typename Q>
HOLO_HD bool polar(double x, double y, const PolarEntry *table, A angle_of, R inverse_of, Q y0_of,
                   double *modulus, double *angle) {
  const uint64_t bx = double_bits(x), by = double_bits(y);
  const int ex = (int)(bx >> 52) & 0x7ff, ey = (int)(by >> 52) & 0x7ff;
  const int top = ex > ey ? ex : ey, low = ex > ey ? ey : ex;
  if (top <= 500 || top >= 1500 || low + 500 < top) return false;
  const uint64_t shift = (uint64_t)(int64_t)(top - 1023) << 52;
  const double xn = as_double(bx - shift), yn = as_double(by - shift);
  const float fx = cut_float(bx, ex, top), fy = cut_float(by, ey, top);
  const int index = round_int(fmul(angle_of(fy, fx), (float)(kPolarHalf / 3.14159265358979)));
  const PolarEntry &E = table[index + kPolarHalf];
  const double p = xn * E.s, pe = fma(xn, E.s, -p);
  const double across = (fma(yn, E.c, -p) - pe) + (double)fmaf(fy, E.cl, -fmul(fx, E.sl));
  const double along = fma(xn, E.c, yn * E.s);
  double inv = (double)inverse_of((float)along);
  inv = fma(fma(-along, inv, 1.0), inv, inv);
  const double t0 = across * inv, t = fma(fma(-along, t0, across), inv, t0);  // |t| < 2^-8
  const double t2 = t * t, series = fma(t * t2, fma(t2, 0.2, -1.0 / 3.0), t);
  *angle = E.a + (series + (double)E.al);
  const double big = ex > ey ? xn : yn, small = ex > ey ? yn : xn;
  const uint64_t sum = double_bits(fma(big, big, small * small));
  const Root r = root((uint32_t)(sum >> 32), (uint32_t)sum, y0_of);
  *modulus = as_double(r.d + ((uint64_t)(uint32_t)(r.q + top - 1) << 52));
  return true;
}

}  // namespace fixed
}  // namespace holo
