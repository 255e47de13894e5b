// Host check of the stage arithmetic (cato_physics.cuh): the same source as the device code,
// compiled for the host with the device intrinsics spelled out below.  Each family compares a
// routine that leaves work out, or does it on the integer pipe, with the general form it stands
// for, bit for bit (any NaN equals any NaN).
//
// usage: physics_check <cases per family and range>
// Prints one line per family ("<family> tested <n> bad <n>") and exits 1 on any mismatch.
#include <cfloat>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <type_traits>

#include <cuda_runtime.h>

// the runtime header's host spelling of the qualifiers
#undef __noinline__
#define __noinline__ __attribute__((__noinline__))
#undef __forceinline__
#define __forceinline__ inline

using std::isfinite;
using std::isnan;
using std::max;
using std::min;
using std::signbit;

template <typename T, typename U> static T bit_cast(U u) {
  static_assert(sizeof(T) == sizeof(U), "");
  T t;
  std::memcpy(&t, &u, sizeof t);
  return t;
}
static inline double __longlong_as_double(long long x) { return bit_cast<double>(x); }
static inline long long __double_as_longlong(double x) { return bit_cast<long long>(x); }
static inline float __uint_as_float(unsigned x) { return bit_cast<float>(x); }
static inline unsigned __float_as_uint(float x) { return bit_cast<unsigned>(x); }
static inline int __double2hiint(double x) { return (int)(bit_cast<uint64_t>(x) >> 32); }
static inline int __double2loint(double x) { return (int)(uint32_t)bit_cast<uint64_t>(x); }
static inline double __hiloint2double(int h, int l) {
  return bit_cast<double>(((uint64_t)(uint32_t)h << 32) | (uint32_t)l);
}
static inline unsigned __funnelshift_l(unsigned lo, unsigned hi, unsigned s) {
  return (unsigned)(((((uint64_t)hi << 32) | lo) << (s & 31)) >> 32);
}
static inline double __dadd_rn(double a, double b) { return a + b; }
static inline double __dsub_rn(double a, double b) { return a - b; }
static inline double __dmul_rn(double a, double b) { return a * b; }
static inline float __fadd_rn(float a, float b) { return a + b; }
static inline float __fsub_rn(float a, float b) { return a - b; }
static inline float __fmul_rn(float a, float b) { return a * b; }
static inline float __fdiv_rn(float a, float b) { return a / b; }
static inline float __fdividef(float a, float b) { return a / b; }
static inline float __fmaf_rn(float a, float b, float c) { return fmaf(a, b, c); }
static inline float __int2float_rn(int a) { return (float)a; }
static inline float rsqrtf(float a) { return (float)(1.0 / std::sqrt((double)a)); }

#include "../fvleg_2d_gb300/csrc/cato_physics.cuh"

using namespace cato;

static std::mt19937_64 rng(20261205);
static unsigned long long tested, bad;
static int fail = 0;

static double unit() { return (double)(rng() >> 11) * 0x1p-53; }
// +-2^e for e in [lo, hi], one in four a power of two
static double any_of(double lo, double hi) {
  double e = lo + unit() * (hi - lo);
  if (rng() % 4 == 0) e = std::floor(e);
  const double m = std::exp2(e);
  return (rng() & 1) ? m : -m;
}
static const double kSpecial[] = {0.0,     -0.0,    1.0,     -1.0,     INFINITY, -INFINITY, NAN,
                                  DBL_MAX, -DBL_MAX, DBL_MIN, 4.9e-324, 1e-16,    -1e-16,    1e-30,
                                  1e30,    2.220446049250313e-16};
static double special() { return kSpecial[rng() % (sizeof kSpecial / sizeof *kSpecial)]; }

static bool same(double a, double b) {
  return (isnan(a) && isnan(b)) || bit_cast<uint64_t>(a) == bit_cast<uint64_t>(b);
}
static void report(const char* family) {
  printf("%s tested %llu bad %llu\n", family, tested, bad);
  fail |= bad != 0;
  tested = bad = 0;
}

// ranges of the reconstruction families: magnitudes 2^lo .. 2^hi; kind 0 values, 1 relative
// differences around a base value, 2 values and zeros, 3 values and special values
static const struct {
  int kind, lo, hi;
} kRanges[] = {{0, -4, 4},    {1, -50, -1}, {0, -30, 30},  {2, -20, 20},   {2, -52, 30},
               {0, -52, 58}, {2, -52, 58}, {0, -100, 100}, {3, -52, 58}, {2, -56, 2}};
template <int N> static void stencil(int kind, int lo, int hi, double (&q)[N]) {
  const double base = any_of(-3, 3);
  for (double& x : q) {
    if (kind == 1) x = base * (1.0 + any_of(lo, hi));
    else if (kind == 2 && rng() % 3 == 0) x = (rng() & 1) ? 0.0 : -0.0;
    else if (kind == 3 && rng() % 2 == 0) x = special();
    else x = any_of(lo, hi);
  }
}

// the MLP edge values that leave out what cannot decide, against all of the limiter's terms
template <int ORDER> static void check_mlp(long n) {
  for (const auto& r : kRanges)
    for (long i = 0; i < n; ++i) {
      double q[10];
      stencil(r.kind, r.lo, r.hi, q);
      const EdgePair a = recon_mlp_f64<ORDER>(q[0], q[1], q[2], q[3], q[4], q[5], q[6], q[7], q[8],
                                              q[9]);
      const EdgePair b = recon_mlp_any<ORDER>(q[0], q[1], q[2], q[3], q[4], q[5], q[6], q[7], q[8],
                                              q[9]);
      ++tested;
      if (same(a.L, b.L) && same(a.R, b.R)) continue;
      if (bad++ < 3) {
        printf("mlp%d", ORDER);
        for (double x : q) printf(" %.17g", x);
        printf(": %.17g %.17g, general form %.17g %.17g\n", a.L, a.R, b.L, b.R);
      }
    }
}

// the Roe pressure sensor that divides only where the pressures are far apart, in every type
static void check_roe_sensor(long n) {
  for (const auto& r : kRanges)
    for (long i = 0; i < n; ++i) {
      double q[2];
      stencil(r.kind, std::max(r.lo, -60), std::min(r.hi, 60), q);
      if (r.kind == 1) q[1] = std::copysign(q[1], q[0]);
      const float f[2] = {(float)q[0], (float)q[1]};
      ++tested;
      const bool ok = roe_sensor<double>(q[0], q[1]) == roe_sensor_slow<double>(q[0], q[1]) &&
                      roe_sensor<float>(f[0], f[1]) == roe_sensor_slow<float>(f[0], f[1]) &&
                      roe_sensor<df>(df(q[0]), df(q[1])) == roe_sensor_slow<df>(df(q[0]), df(q[1]));
      if (!ok && bad++ < 3) printf("roe_sensor %.17g %.17g\n", q[0], q[1]);
    }
}

// the TVD2 edge values that divide only where the ratio itself is needed
static void check_tvd2(long n) {
  for (const auto& r : kRanges)
    for (long i = 0; i < n; ++i) {
      double q[4];
      stencil(r.kind, r.lo, r.hi, q);
      const int lim = (int)(i % 3);
      const EdgePair a = recon_tvd2_f64(lim, q[0], q[1], q[2], q[3]);
      EdgePair b;
      recon_tvd2<double>(lim, q[0], q[1], q[2], q[3], b.L, b.R);
      ++tested;
      if (same(a.L, b.L) && same(a.R, b.R)) continue;
      if (bad++ < 3)
        printf("tvd2 limiter %d %.17g %.17g %.17g %.17g: %.17g %.17g, general form %.17g %.17g\n", lim,
               q[0], q[1], q[2], q[3], a.L, a.R, b.L, b.R);
    }
}

// a bit pattern: the exponents 0 to 2047 in turn, either sign, and significands at random, near
// either end, or with few bits set
static uint64_t pattern(long i) {
  constexpr uint64_t frac = 0x000fffffffffffffULL;
  uint64_t m = rng() & frac;
  switch (rng() % 5) {
    case 0: m &= 0xfff; break;
    case 1: m = frac - (m & 0xfff); break;
    case 2: m = (rng() & 1) ? 0 : frac; break;
    case 3: m = (1ULL << (rng() % 52)) | (1ULL << (rng() % 52)); break;
    default: break;
  }
  return ((rng() & 1) << 63) | ((uint64_t)(i & 2047) << 52) | m;
}

static void check_sums(long n, bool one) {
  for (long i = 0; i < 10 * n; ++i) {
    uint64_t u = pattern(i);
    if (one && i % 2) u = (u & 0x000fffffffffffffULL) | ((uint64_t)(988 + i / 2 % 40) << 52);
    const double x = bit_cast<double>(u), y = one ? 1.0 + x : x + 1e-16;
    bool ok;
    const uint64_t r = one ? intdiv::one_plus_bits(u, ok) : intdiv::add_1em16_bits(u, ok);
    if (!ok) continue;
    ++tested;
    if (r == bit_cast<uint64_t>(y)) continue;
    if (bad++ < 3) printf("%a: %a, sum %a\n", x, bit_cast<double>(r), y);
  }
}

static void check_to_df(long n) {
  for (long i = 0; i < 10 * n; ++i) {
    const double d = bit_cast<double>(pattern(i));
    const df a = to_df(d), b = to_df_any(d);
    ++tested;
    if (same(a.hi, b.hi) && same(a.lo, b.lo)) continue;
    if (bad++ < 3) printf("to_df %a: %a %a, general form %a %a\n", d, a.hi, a.lo, b.hi, b.lo);
  }
}

// exact but for denormals, which become zeros
static void check_f2d(long n) {
  for (long i = 0; i < 10 * n; ++i) {
    uint32_t u = (uint32_t)rng();
    if (i % 4 == 1) u = (u & 0x80000000u) | ((uint32_t)(i / 4 % 256) << 23);
    if (i % 4 == 2) u |= 0x007fffffu;
    if (i % 4 == 3) u = (u & 0x80000007u) + ((uint32_t)(rng() % 4 * 85) << 23);
    const float f = bit_cast<float>(u);
    const double d = std::fabs(f) < FLT_MIN ? std::copysign(0.0, f) : (double)f;
    ++tested;
    if (!same(f2d_int(f), d) && bad++ < 3) printf("f2d_int %a: %a\n", f, f2d_int(f));
  }
}

// normal operands with a normal quotient (one just below the normal range can round into it)
static void check_div_normal(long n) {
  auto normal = [](double x) { return std::isnormal(x); };
  auto in_range = [](double q) { return q >= 2.0 * DBL_MIN && q <= DBL_MAX; };
  for (long i = 0; i < 5 * n; ++i) {
    double x[4];
    for (double& v : x) v = bit_cast<double>(pattern((long)(rng() % 2048)));
    if (i % 2)
      for (double& v : x) {
        int e;
        v = std::ldexp(std::frexp(v, &e), (int)(rng() % 60) - 30);
      }
    if (!normal(x[0]) || !normal(x[1]) || !normal(x[2]) || !normal(x[3])) continue;
    const double q = std::fabs(x[0] / x[1]), p = std::fabs(x[2] / x[3]);
    if (!in_range(q) || !in_range(p)) continue;
    const D2 two = div_normal2(x[0], x[1], x[2], x[3]);
    ++tested;
    const bool ok = same(div_normal(x[0], x[1]), q) && same(two.x, q) && same(two.y, p);
    if (!ok && bad++ < 3) printf("div_normal %a / %a, %a / %a\n", x[0], x[1], x[2], x[3]);
  }
}

int main(int argc, char** argv) {
  const long n = argc > 1 ? atol(argv[1]) : 400000;
  check_mlp<3>(n);
  report("mlp3");
  check_mlp<5>(n);
  report("mlp5");
  check_roe_sensor(n);
  report("roe_sensor");
  check_tvd2(n);
  report("tvd2");
  check_sums(n, false);
  report("add_1em16");
  check_sums(n, true);
  report("one_plus");
  check_to_df(n);
  report("to_df");
  check_f2d(n);
  report("f2d_int");
  check_div_normal(n);
  report("div_normal");
  return fail;
}
