// Check of the kernels' own FP64 reciprocal and quotient, of the conversions of the preconditioner's
// factors and of the device's double-word reciprocal against CUDA's operations (compiled and run by
// tests/test_quotient.py). One line per check: its name and the worst error in units in the last place
// of the plain operation's result, or the number of results that are not the same bits.
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "sayram_ops.cuh"

using sg::dw;
typedef unsigned long long u64;

struct Out {
  double rcp, rcp_plain, div, div_plain, wide;
  float nar, nar_plain, fdiv;
  dw rd;
};
__global__ void k_check(int n, const double* a, const double* b, Out* o) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  Out r;
  r.rcp = sg::rcp64(b[k]);
  r.rcp_plain = 1.0 / b[k];
  r.div = sg::div64(a[k], b[k]);
  r.div_plain = a[k] / b[k];
  r.nar = sg::narrow(fabs(b[k]));
  r.nar_plain = __double2float_rz(fabs(b[k]));
  r.wide = sg::widen<double>(r.nar);
  r.rd = sg::dw_rcp(sg::dw_from_double(b[k]));
  o[k] = r;
}

static u64 bits(double v) { u64 u; memcpy(&u, &v, 8); return u; }
static double frombits(u64 u) { double v; memcpy(&v, &u, 8); return v; }
static bool same(double x, double y) { return (std::isnan(x) && std::isnan(y)) || (x == y && (x == 0.0 || bits(x) == bits(y))); }
// distance of two doubles in units in the last place; 1e300 where they are not comparable. Zeros are alike.
static double ulps(double x, double y) {
  if (x == y || same(x, y)) return 0.0;
  if (std::isnan(x) || std::isnan(y) || std::isinf(x) || std::isinf(y) || std::signbit(x) != std::signbit(y)) return 1e300;
  const long long d = (long long)bits(x) - (long long)bits(y);
  return (double)(d < 0 ? -d : d);
}

int main() {
  std::vector<double> A, B;
  auto put = [&](double a, double b) { A.push_back(a); B.push_back(b); };
  std::mt19937_64 g(2024);
  const double special[] = {0.0, INFINITY, NAN, 4.9406564584124654e-324, 1e-310, 2.2250738585072009e-308,
                            2.2250738585072014e-308, 1.7976931348623157e308, 1.0, 1.5, 3.0};
  std::vector<double> edge;
  for (double v : special)
    for (int s = 0; s < 2; ++s) edge.push_back(s ? -v : v);
  for (int e : {0, 1, 2, 3, 4, 1022, 1023, 1024, 2041, 2042, 2043, 2044, 2046})  // around the branches, both ends of a binade
    for (u64 m : {0ull, 1ull, 0x8000000000000ull, 0xfffffffffffffull})
      for (u64 s : {0ull, 1ull}) edge.push_back(frombits(s << 63 | (u64)e << 52 | m));
  for (double a : edge)
    for (double b : edge) put(a, b);
  for (int e = 0; e < 2047; ++e)  // every exponent of the divisor, powers of two among them
    for (int k = 0; k < 400; ++k) {
      const u64 m = k == 0 ? 0 : g() >> 12, s = g() & 1;
      const int ea = k % 2 ? (int)(g() % 2047) : std::min(2046, std::max(0, e + (int)(g() % 41) - 20));
      put(frombits((g() & 1) << 63 | (u64)ea << 52 | g() >> 12), frombits(s << 63 | (u64)e << 52 | m));
    }
  const int n = (int)A.size();
  double *da, *db;
  Out* dout;
  std::vector<Out> o(n);
  if (cudaMalloc(&da, 8 * (size_t)n) || cudaMalloc(&db, 8 * (size_t)n) || cudaMalloc(&dout, sizeof(Out) * (size_t)n)) return 2;
  cudaMemcpy(da, A.data(), 8 * (size_t)n, cudaMemcpyHostToDevice);
  cudaMemcpy(db, B.data(), 8 * (size_t)n, cudaMemcpyHostToDevice);
  k_check<<<(n + 255) / 256, 256>>>(n, da, db, dout);
  if (cudaMemcpy(o.data(), dout, sizeof(Out) * (size_t)n, cudaMemcpyDeviceToHost)) return 3;
  double rcp = 0, div = 0, rd = 0;
  long long special_rcp = 0, special_div = 0, nar = 0, wid = 0;
  for (int k = 0; k < n; ++k) {
    const Out& r = o[k];
    const int e = (int)(bits(B[k]) >> 52) & 0x7ff;
    rcp = std::fmax(rcp, ulps(r.rcp, r.rcp_plain));
    div = std::fmax(div, ulps(r.div, r.div_plain));
    if ((e < 3 || e > 2042) && !same(r.rcp, r.rcp_plain)) ++special_rcp;
    if ((e < 3 || e > 2042 || !std::isfinite(A[k])) && !same(r.div, r.div_plain)) ++special_div;
    const double b = std::fabs(B[k]);
    if (b < 3.0e38) {  // factors are at most a few units; FP32's subnormals count as 0
      const float want = b < 1.1754943508222875e-38 ? 0.0f : r.nar_plain;
      if (r.nar != want) ++nar;
      if (r.wide != (double)want) ++wid;
    }
    if (b > 1e-24 && b < 1e24) {  // relative error of the double-word reciprocal in units of 2^-48
      const long double y = (long double)sg::dw_to_double(sg::dw_from_double(B[k]));
      rd = std::fmax(rd, (double)(fabsl(((long double)r.rd.hi + (long double)r.rd.lo) * y - 1.0L) * 281474976710656.0L));
    }
  }
  std::printf("rcp64_ulp %g\ndiv64_ulp %g\nrcp64_special %lld\ndiv64_special %lld\nnarrow %lld\nwiden %lld\ndw_rcp %.3f\n", rcp,
              div, special_rcp, special_div, nar, wid, rd);
  return 0;
}
