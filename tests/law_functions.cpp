// log_two and exp_two of dnl_math.cuh on the CPU, as they are written, against
// 113-bit values: the largest errors in ulp of x^y for x in 1e-18..100, y in
// 0..3, and of log x (test_law_functions.py).
#include <math.h>
#include <string.h>

#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <quadmath.h>

static inline uint64_t bits(double x)
{
  uint64_t u;
  memcpy(&u, &x, 8);
  return u;
}
static inline double from(uint64_t u)
{
  double x;
  memcpy(&x, &u, 8);
  return x;
}
static inline int __double2hiint(double x) { return (int)(bits(x) >> 32); }
static inline int __double2loint(double x) { return (int)bits(x); }
static inline double __hiloint2double(int hi, int lo) { return from(((uint64_t)(uint32_t)hi << 32) | (uint32_t)lo); }
static inline double __longlong_as_double(long long v) { return from((uint64_t)v); }
static inline double __dadd_rn(double a, double b) { return a + b; }
#define __device__
#define __forceinline__ inline
#include LAW_SOURCE

int main(int argc, char **argv)
{
  const long n = atol(argv[1]);
  uint64_t s = 88172645463325252ull;
  auto uniform = [&]() { // xorshift
    s ^= s << 13;
    s ^= s >> 7;
    s ^= s << 17;
    return (double)(s >> 11) * 0x1p-53;
  };
  double worstPow = 0, worstLog = 0;
  for (long k = 0; k < n; k++)
  {
    const double x = exp(log(1e-18) + uniform() * (log(100.0) - log(1e-18))), y = 3.0 * uniform();
    const TwoDoubles l = log_two(x);
    const double e = y * l.hi, p = exp_two(e, fma(y, l.lo, fma(y, l.hi, -e)));
    const __float128 lx = logq((__float128)x), q = expq(y * lx);
    const double ulpP = nextafter(p, INFINITY) - p, ulpL = nextafter(fabs(l.hi), INFINITY) - fabs(l.hi);
    worstPow = std::max(worstPow, (double)fabsq(q - p) / ulpP);
    worstLog = std::max(worstLog, (double)fabsq(lx - l.hi) / ulpL);
  }
  printf("%.4f %.4f\n", worstPow, worstLog);
}
