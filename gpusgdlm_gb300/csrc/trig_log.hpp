// FP64 logarithm, sine and cosine by table, for the samplers of FP64 draws.  Plain C++
// beside the loads and bit operations, so that the host can measure the errors of the same
// operations (tests/trig_log_check.cpp).
//
// FP64 is the narrow pipe of this GPU: a warp's log() costs about 30 FMA slots,
// sincospi() about 26, and a FP64 draw takes one of each per two normals and three
// logarithms per gamma.  Table-driven reductions (P. T. P. Tang, "Table-driven
// implementation of the logarithm function in IEEE floating-point arithmetic", ACM
// TOMS 16, 1990, and the same idea with the angle-addition formulas) leave short
// polynomials: 15 and 14 FMA slots, the uniforms' bits taken by integer operations.
//   log: x = 2^k m, m in [3/4, 3/2), m = (1 + f) / inv with inv from 256 intervals,
//     log x = k log 2 + log(1 / inv) + log1p(f).  inv is a multiple of 2^-9 (1 for the two
//     intervals beside 1, so that log is accurate relative to its size there): |f| <= 2^-8
//     and f is exact wherever the sum is small.  The constants are in two parts, the upper
//     ones multiples of 2^-42, so that their sum is exact; f is added to it with its
//     rounding error kept (T. J. Dekker, "A floating-point technique for extending the
//     available precision", 1971).  Error at most 0.517 ulp: the last addition's half, and
//     f^7 / 8 <= 2^-59 of the polynomial in the interval above 1 (log(): 0.54 ulp).  Without
//     f's rounding error and with inv of 53 bits, 12 slots, it was 1.09 ulp beside 1.
//     10 000 draws, the sampler, with log() and sincospi() / 12 slots / 15: m = 100 1084 /
//     576 / 616 us, m = 400 5.88 / 3.3 / 3.49 ms.
//   sin, cos of 2 pi u: the nearest of 1024 angles plus a rest of at most pi / 1024.
//     Absolute error below 1.12e-16 (sincospi(): 1.29e-16).
// The table is 25 KB and read through L1.
//   [0, 2048): cos, sin of 2 pi i / 1024; [2048, 3072): inv, upper and lower part of
//   log(1 / inv), 0; [3072, 3140): upper and lower part of -k log 2, k = 0 .. 33.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#if defined(__CUDACC__)
#define SGDLM_TAB_HD __host__ __device__ __forceinline__
#else
#define SGDLM_TAB_HD inline
#endif

namespace sgdlm {

constexpr int kLogIntervals = 256;
constexpr int kTabLog = 2048, kTabLn2 = kTabLog + 4 * kLogIntervals, kTabSize = kTabLn2 + 2 * 34;
constexpr double kLn2Hi = 0x1.62e42fefa38p-1;  // log 2 rounded to a multiple of 2^-42

inline std::vector<double> trig_log_table() {
  std::vector<double> t(kTabSize, 0.0);
  const long double pi = acosl(-1.0L), grid = ldexpl(1.0L, 42);
  const long double ln2 = logl(2.0L), ln2_hi = kLn2Hi;
  for (int i = 0; i < 1024; ++i) {
    const long double a = 2.0L * pi * i / 1024.0L;
    t[2 * i] = i % 512 == 256 ? 0.0 : (double)cosl(a);
    t[2 * i + 1] = i % 512 == 0 ? 0.0 : (double)sinl(a);
  }
  for (int j = 0; j < kLogIntervals; ++j) {
    long double c = 1.0L + (j + 0.5L) / kLogIntervals;
    if (j >= kLogIntervals / 2) c *= 0.5L;
    if (j == 0 || j == kLogIntervals - 1) c = 1.0L;
    const double inv = (double)(roundl(512.0L / c) / 512.0L);
    const long double l = -logl((long double)inv), hi = roundl(l * grid) / grid;
    double *e = &t[kTabLog + 4 * j];
    e[0] = inv;
    e[1] = (double)hi;
    e[2] = (double)(l - hi);
  }
  for (int k = 0; k < 34; ++k) {
    t[kTabLn2 + 2 * k] = (double)(-k * ln2_hi);
    t[kTabLn2 + 2 * k + 1] = (double)(-k * (ln2 - ln2_hi));
  }
  return t;
}

struct TabPair {
  double x, y;
};
SGDLM_TAB_HD TabPair tab_pair(const double *p) {  // 16-byte aligned
#if defined(__CUDA_ARCH__)
  const double2 v = __ldg(reinterpret_cast<const double2 *>(p));
  return TabPair{v.x, v.y};
#else
  return TabPair{p[0], p[1]};
#endif
}
SGDLM_TAB_HD double tab_value(const double *p) {
#if defined(__CUDA_ARCH__)
  return __ldg(p);
#else
  return *p;
#endif
}
SGDLM_TAB_HD double double_of(uint64_t b) {
#if defined(__CUDA_ARCH__)
  return __longlong_as_double((long long)b);
#else
  double v;
  std::memcpy(&v, &b, sizeof v);
  return v;
#endif
}
SGDLM_TAB_HD uint64_t bits_of(double v) {
#if defined(__CUDA_ARCH__)
  return (uint64_t)__double_as_longlong(v);
#else
  uint64_t b;
  std::memcpy(&b, &v, sizeof b);
  return b;
#endif
}
SGDLM_TAB_HD int leading_zeros(uint64_t v) {
#if defined(__CUDA_ARCH__)
  return __clzll((long long)v);
#else
  return __builtin_clzll(v);
#endif
}

// log1p(f) + log(1 / inv_j) + (khi + klo) for mantissa bits `frac` (52 bits) of a
// value in [1, 2); the value is halved in the upper half of the intervals.
SGDLM_TAB_HD double log_reduced(uint64_t frac, const double *tab, double khi, double klo) {
  const int j = (int)(frac >> 44);
  const uint64_t ex = j >= kLogIntervals / 2 ? 0x3FEull : 0x3FFull;
  const double m = double_of((ex << 52) | frac);
  const TabPair t0 = tab_pair(tab + kTabLog + 4 * j);
  const double lo = tab_value(tab + kTabLog + 4 * j + 2);
  const double f = fma(m, t0.x, -1.0);
  double q = 1.0 / 7.0;
  q = fma(q, f, -1.0 / 6.0);
  q = fma(q, f, 1.0 / 5.0);
  q = fma(q, f, -1.0 / 4.0);
  q = fma(q, f, 1.0 / 3.0);
  q = fma(q, f, -1.0 / 2.0);
  // base + f = s + e (|base| >= |f|, or base = 0)
  const double base = khi + t0.y, s = base + f, e = (base - s) + f;
  return s + (e + fma(f * f, q, klo + lo));
}
// log((a + 1/2) 2^-32)
SGDLM_TAB_HD double log_uniform(uint32_t a, const double *tab) {
  const uint64_t v = 2ull * a + 1ull;  // u = v 2^-33
  const int lz = leading_zeros(v);
  const uint64_t frac = (v << lz >> 11) & 0x000FFFFFFFFFFFFFull;
  // u = 2^(30 - lz) (1 + frac), the exponent one higher where the mantissa is halved
  const int k = lz - 30 - (int)(frac >> 51);
  const TabPair kk = tab_pair(tab + kTabLn2 + 2 * k);
  return log_reduced(frac, tab, kk.x, kk.y);
}
// log(x) for any x (the library's for zero, subnormal, negative and non-finite ones)
SGDLM_TAB_HD double log_table(double x, const double *tab) {
  const uint64_t b = bits_of(x);
  const int ex = (int)(b >> 52);
  if (ex < 1 || ex > 2046) return log(x);
  const uint64_t frac = b & 0x000FFFFFFFFFFFFFull;
  const double k = (double)(ex - 1023 + (int)(frac >> 51));
  const double lo = tab_value(tab + kTabLn2 + 3);  // of -log 2
  return log_reduced(frac, tab, k * kLn2Hi, -k * lo);
}
// sin and cos of 2 pi (b + 1/2) 2^-32
SGDLM_TAB_HD void sincos_uniform(uint32_t b, const double *tab, double &s, double &c) {
  const uint64_t v = 2ull * b + 1ull;  // the angle in units of 2 pi 2^-33
  const uint32_t i = (uint32_t)((v + (1u << 22)) >> 23);
  const int64_t d = (int64_t)v - ((int64_t)i << 23);  // |d| <= 2^22
  const TabPair t0 = tab_pair(tab + 2 * (i & 1023u));
  // d as a double: added into the low bits of 1.5 2^52
  const double x = (double_of((uint64_t)(0x4338000000000000ll + d)) - 0x1.8p52) *
                   7.3145903963357981e-10;  // 2 pi 2^-33
  const double t = x * x;
  const double sx = fma(t * x, fma(t, 1.0 / 120.0, -1.0 / 6.0), x);
  const double cm = t * fma(t, 1.0 / 24.0, -0.5);
  c = t0.x + fma(-t0.y, sx, t0.x * cm);
  s = t0.y + fma(t0.x, sx, t0.y * cm);
}

}  // namespace sgdlm
