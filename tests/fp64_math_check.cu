// fp64_math_check.cu -- MathF64's quotients, reciprocals and roots (hydro_math.cuh) against
// CUDA's operators, and its fifth roots against the host's long double powl.
// Prints one line per function: name, pairs compared, pairs that differ, largest
// difference in units of the last place.  Built with -fmad=false, as the FP64 units.
#include <cmath>
#include <cstdio>
#include <vector>
#include "../emma_b200/csrc/hydro_math.cuh"

using emma::MathF64;

constexpr int kBlocks = 1480, kThreads = 256, kPerThread = 400, kRoots = 1 << 18;
enum { RCP, RCP_ONES, ROOT2, QUOT, QUOT_ONES, DIV_Y, DIV_YY, OVER_G1, COUNT };  // _ONES: divisors of all-ones mantissa

// 64 bits from the upper halves of two steps of a linear congruence (D. Knuth's MMIX)
__device__ unsigned long long bits64(unsigned long long &s) {
  s = s * 6364136223846793005ULL + 1442695040888963407ULL;
  const unsigned long long hi = s >> 32;
  s = s * 6364136223846793005ULL + 1442695040888963407ULL;
  return (hi << 32) | (s >> 32);
}

// +-m 2^e, |e| <= emax; every eighth mantissa all ones, a few bits above a power of two, or
// a few below the next one
__device__ double draw(unsigned long long &s, int emax) {
  unsigned long long m = bits64(s) & 0xfffffffffffffULL;
  const int k = (int)(bits64(s) % 24);
  if (k == 0) m = 0xfffffffffffffULL;
  if (k == 1) m &= 0xfULL;
  if (k == 2) m |= 0xffffffffffff0ULL;
  const unsigned long long e = 1023 - emax + bits64(s) % (2 * emax + 1);
  return __longlong_as_double((long long)((e << 52) | m | (bits64(s) & 0x8000000000000000ULL)));
}

__device__ void compare(double x, double ref, unsigned long long &differ, unsigned long long &ulp) {
  const long long d = __double_as_longlong(x) - __double_as_longlong(ref);
  const unsigned long long u = (unsigned long long)(d < 0 ? -d : d);
  if (u != 0) differ++;
  if (u > ulp) ulp = u;
}

__global__ void operators(int emax, unsigned long long *differ, unsigned long long *ulp) {
  unsigned long long s = (blockIdx.x * (unsigned long long)kThreads + threadIdx.x) * 7919ULL + emax;
  unsigned long long n[COUNT] = {}, u[COUNT] = {};
  for (int i = 0; i < kPerThread; i++) {
    const double a = draw(s, emax), b = draw(s, emax), y = 1. / b;
    const bool ones = (__double_as_longlong(b) & 0xfffffffffffffLL) == 0xfffffffffffffLL;
    compare(MathF64::rcp(b), y, n[RCP + ones], u[RCP + ones]);
    // a root's argument: anything, or a few places from a square, whose root is nearly a number
    const double q = fabs(b), sq = __longlong_as_double(__double_as_longlong(q * q) + (long long)(bits64(s) % 9) - 4);
    const double x = (i & 1) ? sq : fabs(a);
    compare(MathF64::root2(x), sqrt(x), n[ROOT2], u[ROOT2]);
    compare(MathF64::quot(a, b), a / b, n[QUOT + ones], u[QUOT + ones]);
    compare(MathF64::div_y(a, b, y), a / b, n[DIV_Y], u[DIV_Y]);
    compare(MathF64::div_yy(a, b, y), a / (b * b), n[DIV_YY], u[DIV_YY]);
    compare(MathF64::over_g1(a), a / (emma::kGam - 1.), n[OVER_G1], u[OVER_G1]);
  }
  for (int k = 0; k < COUNT; k++) {
    atomicAdd(differ + k, n[k]);
    atomicMax(ulp + k, u[k]);
  }
}

__global__ void fifth_roots(double *out) {  // x, root5, its reciprocal, root5_near
  const int i = blockIdx.x * kThreads + threadIdx.x;
  if (i >= kRoots) return;
  unsigned long long s = i * 104729ULL;
  const double x = fabs(draw(s, 100));
  double iy;
  const double y = MathF64::root5(x, iy);
  out[4 * i] = x;
  out[4 * i + 1] = y;
  out[4 * i + 2] = iy;
  out[4 * i + 3] = MathF64::root5_near(x, y * (1. + (double)((int)(bits64(s) % 9) - 4) * 2.220446049250313e-16));
}

#define CK(e)                                                  \
  if (cudaError_t err = (e)) {                                 \
    std::fprintf(stderr, "%s\n", cudaGetErrorString(err));     \
    return 1;                                                  \
  }

int main() {
  unsigned long long *d, n[COUNT] = {}, u[COUNT] = {};
  CK(cudaMalloc(&d, sizeof(n) + sizeof(u)));
  CK(cudaMemset(d, 0, sizeof(n) + sizeof(u)));
  // exponents that leave every product, quotient and residual normal (div_yy: 3 emax + 53 + 2 < 1022)
  const int emax[] = {1, 20, 100, 300};
  for (int e : emax) operators<<<kBlocks, kThreads>>>(e, d, d + COUNT);
  CK(cudaGetLastError());
  CK(cudaMemcpy(n, d, sizeof(n), cudaMemcpyDeviceToHost));
  CK(cudaMemcpy(u, d + COUNT, sizeof(u), cudaMemcpyDeviceToHost));
  const char *name[COUNT] = {"rcp", "rcp_ones", "root2", "quot", "quot_ones", "div_y", "div_yy", "over_g1"};
  const double pairs = 4. * kBlocks * kThreads * kPerThread;
  for (int k = 0; k < COUNT; k++) std::printf("%s %.0f %llu %llu\n", name[k], pairs, n[k], u[k]);

  double *r;
  CK(cudaMalloc(&r, sizeof(double) * 4 * kRoots));
  fifth_roots<<<(kRoots + kThreads - 1) / kThreads, kThreads>>>(r);
  CK(cudaGetLastError());
  std::vector<double> h(4 * kRoots);
  CK(cudaMemcpy(h.data(), r, sizeof(double) * 4 * kRoots, cudaMemcpyDeviceToHost));
  // distance from the exact power in units of the double's last place
  auto off = [](double x, long double exact) {
    return (double)(fabsl((long double)x - exact) / (long double)(std::nextafter(std::fabs(x), INFINITY) - std::fabs(x)));
  };
  double most[3] = {};
  unsigned long long miss[3] = {};
  for (int i = 0; i < kRoots; i++) {
    const long double p = powl((long double)h[4 * i], (long double)0.2);  // the double nearest 1/5
    const long double want[3] = {p, 1.L / (long double)h[4 * i + 1], p};
    for (int k = 0; k < 3; k++) {
      const double e = off(h[4 * i + 1 + k], want[k]);
      if (e > most[k]) most[k] = e;
      if (h[4 * i + 1 + k] != (double)want[k]) miss[k]++;
    }
  }
  const char *rname[3] = {"root5", "root5_rcp", "root5_near"};
  for (int k = 0; k < 3; k++) std::printf("%s %d %llu %.4f\n", rname[k], kRoots, miss[k], most[k]);
  return 0;
}
