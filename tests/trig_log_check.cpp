// Test harness: the FP64 logarithm, sine and cosine of gpusgdlm_gb300/csrc/trig_log.hpp on
// the host, with their errors against long double.
#include "../gpusgdlm_gb300/csrc/trig_log.hpp"

namespace {
const std::vector<double> &table() {
  static const std::vector<double> t = sgdlm::trig_log_table();
  return t;
}
double ulps(double got, long double want) {
  int ex;
  frexpl(want, &ex);
  return (double)(fabsl((long double)got - want) / ldexpl(1.0L, ex - 53));
}
}  // namespace

extern "C" {
// err[i]: error of log((a_i + 1/2) 2^-32) in units of the last place
void check_log_uniform(long n, const uint32_t *a, double *err) {
  for (long i = 0; i < n; ++i) {
    const long double v = 2.0L * a[i] + 1.0L, one = ldexpl(1.0L, 33);
    const long double want = v > 0.5L * one ? log1pl((v - one) / one) : logl(v / one);
    err[i] = ulps(sgdlm::log_uniform(a[i], table().data()), want);
  }
}
void check_log(long n, const double *x, double *err) {
  for (long i = 0; i < n; ++i) {
    const long double want = logl((long double)x[i]);
    err[i] = want == 0.0L ? fabs(sgdlm::log_table(x[i], table().data()))
                          : ulps(sgdlm::log_table(x[i], table().data()), want);
  }
}
void values_log(long n, const double *x, double *y) {
  for (long i = 0; i < n; ++i) y[i] = sgdlm::log_table(x[i], table().data());
}
// err[i]: the larger absolute error of sin and cos of 2 pi (b_i + 1/2) 2^-32
void check_sincos(long n, const uint32_t *b, double *err) {
  const long double two_pi = 2.0L * acosl(-1.0L);
  for (long i = 0; i < n; ++i) {
    double s, c;
    sgdlm::sincos_uniform(b[i], table().data(), s, c);
    // the angle reduced to an eighth of the circle, where the functions are exact to the
    // long double's last place
    const uint64_t v = 2ull * b[i] + 1ull;
    const int oct = (int)((v + (1ull << 29)) >> 30);  // nearest multiple of pi / 4 (exact rest)
    const long double r = two_pi * ldexpl((long double)((int64_t)v - ((int64_t)oct << 30)), -33);
    const long double h = sqrtl(0.5L), cr = cosl(r), sr = sinl(r);
    const long double co[8] = {1, h, 0, -h, -1, -h, 0, h}, si[8] = {0, h, 1, h, 0, -h, -1, -h};
    const long double wc = co[oct % 8] * cr - si[oct % 8] * sr, ws = si[oct % 8] * cr + co[oct % 8] * sr;
    const double es = (double)fabsl(s - ws), ec = (double)fabsl(c - wc);
    err[i] = es > ec ? es : ec;
  }
}
}
