// Host check of fc3dgpu_ieee64.cuh: division, square root and comparisons
// against the compiler's, on random and structured operands, with the FP32
// seeds off by argv[1] units of the last place (the device's approximations
// are not exact).  Prints the number of mismatches.
#include <cmath>
#include <cstdio>
#include <cstdlib>

#include "fc3dgpu_ieee64.cuh"
using namespace fc3dgpu;

static uint64_t state[2] = {123456789, 987654321};
static uint64_t rnd() {
  uint64_t a = state[0], b = state[1];
  state[0] = b;
  a ^= a << 23;
  state[1] = a ^ b ^ (a >> 17) ^ (b >> 26);
  return state[1] + b;
}
static bool differ(double x, double y) { return ie_bits(x) != ie_bits(y) && !(x != x && y != y); }

static long check(double x, double y) {
  long bad = differ(ie_div(x, y), x / y) + differ(ie_sqrt(x), std::sqrt(x));
  double q0, q1;
  ie_div2(x, y, ie_den(y), q0, q1);
  bad += differ(q0, x / y) + differ(q1, y / y);
  bad += (ie_lt(x, y) != (x < y)) + (ie_le(x, y) != (x <= y)) + (ie_positive(x) != (x > 0)) + (ie_nan(x) != (x != x));
  const double a = ie_abs(x), b = ie_abs(y);
  bad += (ie_lt_pos(a, b) != (a < b)) + (ie_le_pos(a, b) != (a <= b));
  if (a >= 1.2e-38 && a < 3e38) bad += !(std::fabs((double)ie_float(x) - a) <= a * 1.2e-7);
  return bad;
}

int main(int argc, char** argv) {
  ie_host_seed_ulps = std::atoi(argv[1]);
  const long n = std::atol(argv[2]);
  long bad = 0;
  const double edge[] = {0.0, -0.0, 1.0, -1.0, INFINITY, -INFINITY, NAN, -NAN, 5e-324, -5e-324, 2.2250738585072014e-308,
                         1.7976931348623157e308, 1e-310, 2.0, 0.5, 3.0, 0x1.fffffffffffffp0, 0x1.0000000000001p0};
  for (double a : edge)
    for (double b : edge) bad += check(a, b);
  for (long i = 0; i < n; i++) {
    uint64_t a = rnd(), b = rnd();
    const int k = i & 15;
    if (k == 1) a &= 0xfff0000000000000ull;
    if (k == 2) b &= 0xfff0000000000000ull;
    if (k == 3) a |= 0xfffffffffffffull;
    if (k == 4) b |= 0xfffffffffffffull;
    if (k == 5) b = (b & 0xfff0000000000000ull) | (rnd() & 0xff);
    if (k == 7) b = ((a & 0xfffffffffffffull) | (b & 0xfff0000000000000ull)) + rnd() % 5 - 2;
    if (k >= 8) {
      a = (a & 0x800fffffffffffffull) | ((1003 + rnd() % 40) << 52);
      b = (b & 0x800fffffffffffffull) | ((1003 + rnd() % 40) << 52);
    }
    bad += check(ie_double(a), ie_double(b));
    double z = ie_double((b & 0xfffffffffffffull) | ((1000 + rnd() % 50) << 52));  // next to a square
    z = ie_double(ie_bits(z * z) + rnd() % 5 - 2);
    bad += differ(ie_sqrt(z), std::sqrt(z));
  }
  std::printf("%ld\n", bad);
  return 0;
}
