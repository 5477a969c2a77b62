// Host build of the fixed-point arithmetic (scale-dg-kernel-extraction_gb300/
// csrc/sdg_fix.cuh), compiled with g++ by test_fix_host.py.  Checks the
// conversions on both sides, what the range check takes, and that one row of
// an even-odd line sum (products q u, pair sums, coefficients, two lift terms)
// agrees with long double to 46 units of 2^-61 of the row's bound and is nearer
// to it, over many rows, than the same row in double.
//
// The 46 units (a row's pair coefficients add up to at most 1/2): an aligned
// value is off by at most one of 2^-59, four units, a pair sum by eight, so the
// weighted sum by four; a face at a quarter scale by 16, two faces by 32,
// weighted by 16; a coefficient by half of 2^-60 against sums of 2^60, two units
// a term; the dropped low limbs by half a unit a term; the last shift by one:
// 4 + 16 + 20 + 5 + 1 for n <= 10.  The products q u themselves are doubles, as
// in FP64 arithmetic: the exact sum starts from them.
#include <cmath>
#include <cstdio>
#include <random>

#include "sdg_fix.cuh"

using namespace sdg;

static std::mt19937_64 rng(20261205);
static double uni(double a, double b) { return std::uniform_real_distribution<double>(a, b)(rng); }
static double pow2(int e) { return std::ldexp(1.0, e); }

static int fail(const char* what, double x) {
  std::printf("FAIL %s %a\n", what, x);
  return 1;
}

static int conversions() {
  for (int t = 0; t < 1000000; t++) {
    const double f = uni(-1, 1) * pow2((int)(rng() % 300) - 150);
    const int32_t E = fix_value_exp(f) + ((int32_t)(rng() % 80) << 20);
    if (!fix_in_range(E)) return fail("range", f);
    const long double want = std::ldexp((long double)f, 59 - fix_line_exp(E));
    const int64_t got = fix_align(f, E);
    if (std::fabs((long double)got - want) > 1.0L || std::fabs((long double)got) > std::ldexp(1.0L, 59))
      return fail("align", f);
    const int32_t Eg = fix_face_exp(f) + ((int32_t)(rng() % 80) << 20);
    const long double wg = std::ldexp((long double)f, 57 - fix_line_exp(Eg));
    const int64_t ig = fix_align_face(f, Eg);
    if (std::fabs((long double)ig - wg) > 1.0L || std::fabs((long double)ig) > std::ldexp(1.0L, 59))
      return fail("face", f);
    const int64_t y = (int64_t)(rng() >> (1 + rng() % 62)) * ((rng() & 1) ? 1 : -1);
    const int e = (int)(rng() % 1000) - 500;
    const long double wy = std::ldexp((long double)y, e);
    // a negative value is complemented: one unit beside the rounding
    if (std::fabs((long double)fix_to_double(y, e) - wy) >
        std::ldexp(std::fabs(wy), -53) + std::ldexp(1.0L, e))
      return fail("to_double", (double)y);
  }
  const int64_t one = 1;
  const int64_t edge[] = {0, 1, -1, 2, one << 31, one << 32, (one << 32) - 1, -(one << 33) + 1,
                          (one << 53) + 1, -((one << 62) + 511), (one << 62) - 1, INT64_MAX,
                          INT64_MAX - 600, -INT64_MAX, (one << 54) - 1, 1023, -2048};
  for (int64_t y : edge)
    if (std::fabs((long double)fix_to_double(y, -7) - std::ldexp((long double)y, -7)) >
        std::ldexp(std::fabs((long double)y), -60) + std::ldexp(1.0L, -7))
      return fail("edge", (double)y);
  // infinities, NaN and values near the ends of the range are refused
  const double out[] = {(double)INFINITY, -(double)INFINITY, (double)NAN, 1e300, pow2(701),
                        0.0, -0.0, 4e-310, 1e-300, pow2(-702)};
  for (double x : out)
    if (fix_in_range(fix_value_exp(x)) || (std::fabs(x) > 1.0 && fix_in_range(fix_face_exp(4 * x))))
      return fail("taken", x);
  // zeros and subnormals align to at most one unit on any line that is taken
  const int32_t low = fix_value_exp(pow2(-701));
  if (!fix_in_range(low)) return fail("low", 0.0);
  const double none[] = {0.0, -0.0, 4e-310};
  for (double x : none)
    if (std::abs(fix_align(x, low)) > 1 || std::abs(fix_align_face(x, low)) > 1)
      return fail("zero", x);
  return 0;
}

int main() {
  if (conversions()) return 1;
  double worst = 0.0, sum_fix = 0.0, sum_dbl = 0.0;
  const int trials = 150000;
  for (int trial = 0; trial < trials; trial++) {
    const int N = 2 + trial % 15, H = N / 2, n = H + 2;
    const double qs = pow2((int)(rng() % 200) - 100), us = pow2((int)(rng() % 40) - 20);
    const double rough = (trial % 3 == 0) ? 1.0 : (trial % 3 == 1) ? 1e-3 : 0.5;
    const double decay = (trial % 3 == 2) ? uni(0.0, 3.0) : 0.0;  // a steep profile along the line
    double q[16], u[16], c[10], most = 0.0;
    for (int l = 0; l < N; l++) {
      q[l] = qs * (0.5 + rough * uni(-1, 1)) * std::exp(-decay * l);
      u[l] = us * (0.7 + rough * uni(-1, 1));
    }
    const double gm = qs * us * rough * uni(-4, 4), gp = qs * us * rough * uni(-4, 4);
    for (int k = 0; k < n; k++) {
      c[k] = (k == H && !(N & 1)) ? 0.0 : uni(-30, 30);
      most += (k == H ? 1.0 : 2.0) * std::fabs(c[k]);
    }
    int k2;
    std::frexp(most * (1.0 + 1e-8), &k2);
    int32_t E = std::max(0, std::max(fix_face_exp(gm), fix_face_exp(gp)));
    double f[16];
    for (int l = 0; l < N; l++) {
      f[l] = q[l] * u[l];
      E = std::max(E, fix_value_exp(f[l]));
    }
    if (!fix_in_range(E)) return fail("row range", q[0]);
    const int B = fix_line_exp(E);
    const bool even = (trial / 15) & 1;
    auto C = [&](int k) { return fix_coef((int64_t)std::llround(std::ldexp((long double)c[k], 60 - k2))); };
    const int64_t im = fix_align_face(gm, E), ip = fix_align_face(gp, E);
    fixacc a;
    fix_mul(a, C(H + 1), fix_split(even ? im - ip : im + ip));
    long double want = (long double)c[H + 1] * 0.25L * (even ? (long double)gm - gp : (long double)gm + gp);
    double dbl = c[H + 1] * 0.25 * (even ? gm - gp : gm + gp);
    for (int l = 0; l < H; l++) {
      const int64_t f1 = fix_align(f[l], E), f2 = fix_align(f[N - 1 - l], E);
      fix_fma(a, C(l), fix_split(even ? f1 + f2 : f1 - f2));
      const long double w1 = f[l], w2 = f[N - 1 - l];
      want += (long double)c[l] * (even ? w1 + w2 : w1 - w2);
      const double p2 = q[N - 1 - l] * u[N - 1 - l];
      dbl = std::fma(c[l], std::fma(q[l], u[l], even ? p2 : -p2), dbl);
    }
    if (N & 1) {
      fix_fma(a, C(H), fix_split(fix_align(f[H], E)));
      want += (long double)c[H] * f[H];
      dbl = std::fma(c[H], q[H] * u[H], dbl);
    }
    const long double got = fix_to_double(fix_sum(a), k2 + B - 61);
    const long double unit = std::ldexp(1.0L, k2 + B);
    // the double nearest to the result adds half an ulp of the result
    const long double err = std::fabs(got - want) - std::ldexp(std::fabs(want), -53);
    worst = std::max(worst, (double)(err / unit) * pow2(61));
    sum_fix += std::pow((double)((got - want) / unit), 2);
    sum_dbl += std::pow((double)((dbl - want) / unit), 2);
  }
  std::printf("worst %.2f units of 2^-61; rms error in the row's bound: fixed %.3e, double %.3e\n",
              worst, std::sqrt(sum_fix / trials), std::sqrt(sum_dbl / trials));
  return (worst <= 46.0 && sum_fix <= sum_dbl) ? 0 : 1;
}
