// CPU check of minifs_b200/csrc/mfg_quot.cuh, the file itself compiled for the
// host with the C library's fma, against the division: the ends of every
// window crossed with the significands where rounding goes wrong, then
// pseudo-random pairs.  Usage: quotient_check N SEED; prints the count of
// wrong quotients, of wrong reciprocals, and of operands on the wrong side of
// a window.
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#define __device__
#define __forceinline__ inline
static uint64_t bits(double d) {
  uint64_t u;
  memcpy(&u, &d, 8);
  return u;
}
static double number(uint64_t u) {
  double d;
  memcpy(&d, &u, 8);
  return d;
}
static int __double2hiint(double d) { return (int)(uint32_t)(bits(d) >> 32); }
static int __double2loint(double d) { return (int)(uint32_t)bits(d); }
static double __hiloint2double(int hi, int lo) {
  return number((uint64_t)(uint32_t)hi << 32 | (uint32_t)lo);
}
static double __dmul_rn(double a, double b) { return a * b; }
static double __fma_rn(double a, double b, double c) { return fma(a, b, c); }
#include "mfg_quot.cuh"

static long long wrong_q, wrong_r, wrong_side;

static bool within(double v, int far) {  // a normal number of an exponent in [-far, far]
  const int e = (int)(bits(v) >> 52 & 0x7FF);
  return e >= 1023 - far && e <= 1023 + far;
}

static void quotient(double a, double b, double near, double y, int bad, bool b_in) {
  const double q = mfg::quot_near(a, b, near, y, bad);
  if ((bad >= 0) != ((a == 0.0 || within(a, 500)) && b_in))
    wrong_side++;
  else if (bad >= 0 && bits(q) != bits(a / b))
    wrong_q++;
}

// a over b as the sweeps' diagonal, a triangle's mean, and the flux's density,
// whose reciprocal starts from one that is off by the factor 1 + off
static void check(double a, double b, double off) {
  quotient(a, b, 1.0 / b, 1.0 / b, mfg::outside_exp(b, 523, 1523), within(b, 500));
  quotient(a, 3.0, 1.0 / 3.0, 1.0 / 3.0, 0, true);
  double near = 0.0;
  int bad = 0;
  const double y = mfg::rcp_rn_from(b, 1.0 / b * (1.0 + off), near, bad);
  const bool ones = (bits(b) & 0xFFFFFFFFFFFFFull) == 0xFFFFFFFFFFFFFull;
  if ((bad >= 0) != (within(b, 500) && !ones)) wrong_side++;
  if (bad < 0) return;
  if (bits(y) != bits(1.0 / b)) wrong_r++;
  quotient(a, b, near, y, 0, true);
}

static uint64_t splitmix64(uint64_t *x) {
  uint64_t z = (*x += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

int main(int argc, char **argv) {
  const long long n = argc > 1 ? atoll(argv[1]) : 1000000;
  uint64_t x = argc > 2 ? strtoull(argv[2], nullptr, 10) : 1;
  const int exps[] = {0,   1,   522,  523,  524,  903,  904,  905, 1022,
                      1023, 1024, 1141, 1142, 1143, 1522, 1523, 1524, 2046, 2047};
  uint64_t mant[] = {0, 1, 0xFFFFFFFFFFFFFull, 0xFFFFFFFFFFFFEull, 0x8000000000000ull, 0, 0};
  for (auto &m : mant)
    if (&m >= mant + 5) m = splitmix64(&x) & 0xFFFFFFFFFFFFFull;
  for (int ea : exps)
    for (int eb : exps)
      for (uint64_t ma : mant)
        for (uint64_t mb : mant)
          for (int s = 0; s < 4; s++)
            check(number((uint64_t)(s & 1) << 63 | (uint64_t)ea << 52 | ma),
                  number((uint64_t)(s >> 1) << 63 | (uint64_t)eb << 52 | mb),
                  s & 1 ? 0x1.fp-19 : -0x1.fp-19);
  for (long long i = 0; i < n; i++) {
    const uint64_t r = splitmix64(&x), e = splitmix64(&x), t = splitmix64(&x), o = splitmix64(&x);
    const uint64_t ea = 1023 - 600 + e % 1201;
    const uint64_t eb = (i & 1) ? 1023 - 130 + (e >> 32) % 261 : 1023 - 600 + (e >> 32) % 1201;
    uint64_t mb = t & 0xFFFFFFFFFFFFFull;
    if ((i & 6) == 6) mb = 0xFFFFFFFFFFFFFull - (i >> 3 & 1);
    check(number((r >> 63) << 63 | ea << 52 | (r & 0xFFFFFFFFFFFFFull)),
          number((t >> 63) << 63 | eb << 52 | mb), ((double)(o >> 11) * 0x1p-53 - 0.5) * 0x1.fcp-18);
  }
  printf("%lld %lld %lld\n", wrong_q, wrong_r, wrong_side);
  return 0;
}
