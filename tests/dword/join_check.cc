// Host check of dw_join_int in csrc/dword.cuh (compiled and run by tests/test_dword_join.py): the bits
// of hi + lo for the pairs dw_from_double makes, at one binary exponent (the argument): significands
// at random, at the halves and carries of hi's rounding, next to a power of two, and both signs.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#include "dword.cuh"

static unsigned long long bits(double v) {
  unsigned long long u;
  std::memcpy(&u, &v, 8);
  return u;
}

int main(int, char** argv) {
  const int lo_e = std::atoi(argv[1]), hi_e = std::atoi(argv[2]);
  std::mt19937_64 g(7);
  long bad = 0, n = 0;
  const auto check = [&](double v) {
    const sg::dw q = sg::dw_from_double(v);
    const double want = (double)q.hi + (double)q.lo, got = sg::dw_join_int(q);
    ++n;
    if (want != want ? got == got : bits(want) != bits(got)) ++bad;
  };
  const unsigned long long top = 0xFFFFFFFFFFFFFull;
  for (int e = lo_e; e <= hi_e; ++e)
    for (int k = 0; k < 400; ++k) {
      unsigned long long m = g() & top;
      if (k % 5 == 1) m = (m & ~0x1FFFFFFFull) | 0x10000000ull;         // half of hi's last place
      if (k % 5 == 2) m = (m & ~0x1FFFFFFFull) | (0x10000000ull + (k & 2 ? 1 : -1));
      if (k % 5 == 3) m = (g() & top) >> (12 + g() % 40);               // just above a power of two
      if (k % 5 == 4) m = top - ((g() & top) >> (20 + g() % 32));       // just below one
      const double v = std::ldexp(1.0 + std::ldexp((double)m, -52), e);
      check(v);
      check(-v);
    }
  check(0.0);
  check(-0.0);
  check(INFINITY);
  check(-INFINITY);
  check(NAN);
  std::printf("%ld of %ld differ\n", bad, n);
  return bad != 0;
}
