/* Host check of the integer-arithmetic FP64 operations (p3x_intfp64.cuh is
 * plain integer code on the host too): disagreements of the division with
 * IEEE division over N operand pairs of one family. */
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#include "p3x_intfp64.cuh"

using namespace p3x::dev;

static std::mt19937_64 g(20240);
static double range(int lo, int hi) {
  return d_from_bits((g() & 0x800fffffffffffffull) | (uint64_t(1023 + lo + int(g() % uint64_t(hi - lo + 1))) << 52));
}
static double edge() {
  const uint64_t m = (g() & 1) ? 0xfffffffffffffull - g() % 4 : g() % 4;
  return d_from_bits((uint64_t(1003 + g() % 40) << 52) | m);
}

static long check_div(int family, long n) {
  long bad = 0;
  for (long i = 0; i < n; ++i) {
    double a = 0, b = 1;
    switch (family) {
      case 0: a = range(-300, 300); b = range(-300, 300); break; /* ordinary */
      case 1: a = edge(); b = edge(); break;                     /* significands near 1 and 2 */
      case 2: b = range(-10, 10); a = range(-10, 10) * b; break; /* quotients near a double */
      case 3: a = double(g() % 100000); b = double(1 + g() % 1000); break;
      case 4: a = d_from_bits(g()); b = d_from_bits(g()); break; /* any bits: inf, NaN, subnormal, overflow */
      case 5: a = (g() & 1) ? 0.0 : -0.0; b = range(-300, 300); break;
      case 6: a = range(-1022, -960); b = range(40, 70); break;  /* quotients around the smallest normal */
      case 7: b = range(-3, 3); a = d_from_bits(d_bits(b) + g() % 16); break;
    }
    const double got = ddiv_int(a, b), want = a / b;
    if (d_bits(got) != d_bits(want) && !(std::isnan(got) && std::isnan(want))) ++bad;
  }
  return bad;
}

int main(int argc, char** argv) {
  std::printf("%ld\n", check_div(std::atoi(argv[1]), std::atol(argv[2])));
  return 0;
}
