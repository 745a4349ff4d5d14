// fpi::fifth_powers against long double powl: every binade, the force law's
// velocity range and the neighbours of powers of two, with the host's seeds
// and with seeds moved by up to +-8 ulp (more than the device's approximations
// are off).  The root is held to 2^-58 of its value, its square to 2^-57: half an
// ulp of rounding, 2^-5 and 2^-4 of one more.
// fpi::sqrt_many and fpi::div_many against the host, special operands among
// the others.
#include <cmath>
#include <cstdio>
#include <cstdint>
#include <cstring>
#include <random>
static uint64_t state = 88172645463325252ull;
static bool noise = false;
static float seed_noise(float r) {
  if (!noise) return r;
  state ^= state << 13; state ^= state >> 7; state ^= state << 17;
  uint32_t u;
  memcpy(&u, &r, 4);
  u += (uint32_t)((int32_t)(state % 17) - 8);
  memcpy(&r, &u, 4);
  return r;
}
#define FPI_HOST_SEED_HOOK seed_noise
#include "../../sdem_gb300/csrc/fp64_int.cuh"

static double off(double got, long double want) {
  const double w = (double)want;
  return (double)(fabsl(got - want) / (std::nextafter(w, INFINITY) - w));
}
static bool same(double a, double b) { return (a != a && b != b) || fpi::bits(a) == fpi::bits(b); }

int main() {
  std::mt19937_64 g(7);
  long bad = 0;
  double m2 = 0, m4 = 0;
  for (int round = 0; round < 2; round++) {
    noise = round == 1;
    for (long i = 0; i < 1500000; i++) {
      double x;
      if (i % 3 == 0) x = fpi::from_bits(((uint64_t)(1 + g() % 2046) << 52) | (g() & fpi::kMant));
      else if (i % 3 == 1) x = 0.01 * std::exp((g() % 1000000) * 1e-6 * 9);
      else x = fpi::from_bits(fpi::bits(std::ldexp(1.0, (int)(g() % 61) - 30)) + g() % 9 - 4);
      double a, b;
      fpi::fifth_powers(x, a, b);
      const double e2 = off(a, powl((long double)x, (long double)0.2)), e4 = off(b, powl((long double)x, (long double)0.4));
      if (e2 > m2) m2 = e2;
      if (e4 > m4) m4 = e4;
    }
  }
  std::printf("x^0.2 %.4f ulp, x^0.4 %.4f ulp\n", m2, m4);
  if (!(m2 <= 0.5 + 1.0 / 32) || !(m4 <= 0.5 + 1.0 / 16)) bad++;
  double a, b;
  fpi::fifth_powers(INFINITY, a, b);
  if (a != INFINITY || b != INFINITY) bad++;
  noise = false;
  const double sp[] = {0.0, -0.0, 1.0, -3.0, INFINITY, -INFINITY, NAN, 4.9e-324, 1e-310, 1.7e308, 2.5e-300};
  for (long i = 0; i < 200000; i++) {
    auto pick = [&]() { return g() % 4 ? fpi::from_bits(((uint64_t)(900 + g() % 250) << 52) | (g() & fpi::kMant)) : sp[g() % 11]; };
    const double x[4] = {pick(), pick(), pick(), pick()}, y = pick(), q3[3] = {x[0], x[1], x[2]};
    double r[4], q[3];
    fpi::sqrt_many(x, r);
    fpi::div_many(q3, fpi::divisor(y), q);
    for (int k = 0; k < 4; k++) bad += !same(r[k], std::sqrt(x[k]));
    for (int k = 0; k < 3; k++) bad += !same(q[k], q3[k] / y);
  }
  std::printf("%ld wrong\n", bad);
  return bad != 0;
}
