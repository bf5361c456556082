// Device check of the arithmetic that replaces correctly rounded or converting
// FP64 instructions (psph_common.cuh) and of the training sigmoid (psph_mlp.cuh):
// against long double on the host, the device's own sqrt and the casts, over
// random arguments of every exponent, range edges, exact squares, powers of two
// and their neighbours, and special values. One line per function: arguments,
// largest error in ulp or mismatches. Exits non-zero where a stated bound does
// not hold.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>
#include <vector>

#include "psph_common.cuh"
#include "psph_mlp.cuh"

using namespace psph;
typedef unsigned long long u64;

static double from_bits(u64 b) {
  double x;
  memcpy(&x, &b, sizeof x);
  return x;
}
static u64 bits(double x) {
  u64 b;
  memcpy(&b, &x, sizeof b);
  return b;
}
// the distance between neighbouring doubles (floats) at the magnitude of x
static long double ulp(long double x, int digits) {
  int e;
  frexpl(x, &e);
  return ldexpl(1.0L, e - digits);
}

enum { RCP, RCP2, RSQRT, SQRT, SQRT_ANY, SQRT_LIB, ABOVE, NEGATIVE, D2F };
__global__ void eval(int f, const double* x, double* y, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double a = x[i];
  switch (f) {
    case RCP: y[i] = rcp_newton(a); break;
    case RCP2: y[i] = rcp_refined(a); break;
    case RSQRT: y[i] = rsqrt_newton(a); break;
    case SQRT: y[i] = sqrt_newton(a); break;
    case SQRT_ANY: y[i] = sqrt_any(a); break;
    case SQRT_LIB: y[i] = sqrt(a); break;
    case ABOVE: y[i] = above(a, 2.0) ? 1.0 : 0.0; break;
    case NEGATIVE: y[i] = negative(a) ? 1.0 : 0.0; break;
    default: y[i] = (double)d2f_bits(a);
  }
}
__global__ void eval_i2d(const int* c, double* y, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = i2d_small(c[i]);
}
__global__ void eval_f2d(const float* c, double* y, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = f2d_bits(c[i]);
}
__global__ void eval_sigm(const float* z, float* y, float* den, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  y[i] = sigm_row(z[i]);
  den[i] = 1.f + expf(-z[i]);
}
__global__ void eval_cell(GridDev g, const double* x, int* got, int* want, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  got[i] = cell_floor(g, 0, x[i]);
  want[i] = (int)floor((x[i] - g.blpf[0]) / g.cell_size[0]);
}

static int failures = 0;
static void must(bool ok, const char* what) {
  if (ok) return;
  printf("FAILED %s\n", what);
  ++failures;
}
template <class T>
static T* to_device(const std::vector<T>& v) {
  T* d = nullptr;
  must(cudaMalloc(&d, v.size() * sizeof(T)) == cudaSuccess, "cudaMalloc");
  must(cudaMemcpy(d, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice) == cudaSuccess, "copy");
  return d;
}
template <class T>
static std::vector<T> to_host(T* d, size_t n) {
  std::vector<T> v(n);
  must(cudaMemcpy(v.data(), d, n * sizeof(T), cudaMemcpyDeviceToHost) == cudaSuccess, "copy back");
  cudaFree(d);
  return v;
}
static std::vector<double> run(int f, const std::vector<double>& x) {
  double *dx = to_device(x), *dy = to_device(x);
  const int n = (int)x.size();
  eval<<<(n + 255) / 256, 256>>>(f, dx, dy, n);
  must(cudaDeviceSynchronize() == cudaSuccess, "launch");
  cudaFree(dx);
  return to_host(dy, x.size());
}

// positive doubles with exponents in [lo, hi): random, near one, powers of two and
// their neighbours, exact squares
static std::vector<double> positives(int lo, int hi, int n) {
  std::mt19937_64 rng(7 * lo + hi);
  std::vector<double> v;
  for (int k = 0; k < n; ++k) {
    const u64 e = (u64)(1023 + lo + (int)(rng() % (u64)(hi - lo)));
    v.push_back(from_bits(e << 52 | (rng() & 0xfffffffffffffull)));
    v.push_back(from_bits((u64)(1022 + (int)(rng() % 3)) << 52 | (rng() & 0xfffffffffffffull)));
    const double q = (double)(1 + rng() % (1u << 26));
    v.push_back(q * q);
  }
  for (int e = lo; e < hi; ++e)
    for (u64 m : {0ull, 1ull, 2ull, 0x8000000000000ull, 0xffffffffffffeull, 0xfffffffffffffull})
      v.push_back(from_bits((u64)(1023 + e) << 52 | m));
  return v;
}

template <class F>
static void ulp_check(const char* name, int f, const std::vector<double>& x, double bound, F&& exact) {
  const std::vector<double> y = run(f, x);
  long double worst = 0.0L;
  double at = 0.0;
  for (size_t k = 0; k < x.size(); ++k) {
    const long double r = exact((long double)x[k]);
    const long double e = std::isfinite(y[k]) ? fabsl((long double)y[k] - r) / ulp(r, 53) : 1e9L;
    if (e > worst) worst = e, at = x[k];
  }
  printf("%-12s %9zu arguments, largest error %.4f ulp (%.17g), bound %.2f\n", name, x.size(), (double)worst, at, bound);
  must(worst <= (long double)bound, name);
}

int main() {
  const int n = 600000;
  const auto full = positives(-1022, 1022, n), roots = positives(-1006, 1024, n);
  ulp_check("rcp_newton", RCP, full, 0.55, [](long double x) { return 1.0L / x; });
  ulp_check("rsqrt_newton", RSQRT, roots, 1.05, [](long double x) { return 1.0L / sqrtl(x); });
  ulp_check("sqrt_newton", SQRT, roots, 1.05, [](long double x) { return sqrtl(x); });
  ulp_check("sqrt_any", SQRT_ANY, roots, 1.05, [](long double x) { return sqrtl(x); });
  {  // correctly rounded: the host's division
    const auto y = run(RCP2, full);
    long long bad = 0;
    for (size_t k = 0; k < full.size(); ++k) bad += y[k] != 1.0 / full[k];
    printf("rcp_refined  %9zu arguments, %lld not correctly rounded\n", full.size(), bad);
    must(bad == 0, "rcp_refined");
  }
  const double inf = std::numeric_limits<double>::infinity(), nan = std::numeric_limits<double>::quiet_NaN();
  {  // outside the roots' range
    const std::vector<double> s = {0.0, 1e-310, 1e-304, inf, nan, -nan};
    const auto q = run(SQRT, s), r = run(RSQRT, s);
    for (int k = 0; k < 3; ++k) must(q[k] == 0.0 && r[k] == 0.0, "no separation");
    must(q[3] == inf && std::isnan(r[3]), "an infinite separation");
    for (int k = 4; k < 6; ++k) must(std::isnan(q[k]) && std::isnan(r[k]), "NaN stays NaN");
    std::vector<double> w = {0.0, -0.0, 1e-310, 5e-324, 1e-304, inf, nan, -1.0, -inf, -nan, -1e-310};
    for (int e = -1022; e < -1006; ++e) w.push_back(ldexp(1.37, e));
    const auto a = run(SQRT_ANY, w), b = run(SQRT_LIB, w);
    for (size_t k = 0; k < w.size(); ++k)
      must(bits(a[k]) == bits(b[k]) || (std::isnan(a[k]) && std::isnan(b[k])), "sqrt_any outside the range");
    // reciprocals of what lies outside: never a wrong finite number
    const std::vector<double> z = {0.0, inf, nan, -nan, 1e-310, ldexp(1.0, 1023)};
    for (int f : {RCP, RCP2}) {
      const auto c = run(f, z);
      for (size_t k = 0; k < 5; ++k) must(!std::isfinite(c[k]) || (c[k] == 0.0 && std::isinf(z[k])), "reciprocal outside");
      must(fabs(c[5]) <= ldexp(1.0, -1023), "reciprocal of 2^1023");
    }
  }
  {  // comparisons
    const std::vector<double> s = {0.0, 1.0, 2.0, nextafter(2.0, 3.0), 3.0, 1e300, inf, nan, -nan};
    const auto a = run(ABOVE, s);
    for (size_t k = 0; k < s.size(); ++k) must((a[k] != 0.0) == (s[k] > 2.0), "above");
    const std::vector<double> t = {0.0, 1.0, -1.0, 5e-324, -5e-324, inf, -inf, -1e300};
    const auto b = run(NEGATIVE, t);
    for (size_t k = 0; k < t.size(); ++k) must((b[k] != 0.0) == (t[k] < 0.0), "negative");
    printf("comparisons  %9zu arguments\n", s.size() + t.size());
  }
  {  // truncation to FP32
    std::vector<double> x = positives(-126, 127, n / 4);
    for (size_t k = 0; k < x.size(); k += 2) x[k] = -x[k];
    const auto y = run(D2F, x);
    long long bad = 0;
    for (size_t k = 0; k < x.size(); ++k)
      bad += !(fabs(y[k]) <= fabs(x[k]) && fabs(y[k]) > fabs(x[k]) * (1.0 - ldexp(1.0, -23)) && (y[k] < 0) == (x[k] < 0));
    printf("d2f_bits     %9zu arguments, %lld not truncated\n", x.size(), bad);
    must(bad == 0, "d2f_bits");
  }
  std::mt19937_64 rng(99);
  {  // integers and floats as doubles
    std::vector<int> c = {0, 1, 2, 3, 2147483647, 2147483646};
    for (int b = 1; b < 31; ++b)
      for (int d = -1; d <= 1; ++d) c.push_back((1 << b) + d);
    for (int k = 0; k < n; ++k) c.push_back((int)(rng() & 0x7fffffff) >> (rng() % 31));
    int* dc = to_device(c);
    double* dy = to_device(std::vector<double>(c.size()));
    eval_i2d<<<((int)c.size() + 255) / 256, 256>>>(dc, dy, (int)c.size());
    const auto y = to_host(dy, c.size());
    long long bad = 0;
    for (size_t k = 0; k < c.size(); ++k) bad += bits(y[k]) != bits((double)c[k]);
    cudaFree(dc);
    printf("i2d_small    %9zu arguments, %lld mismatches\n", c.size(), bad);
    must(bad == 0, "i2d_small");
    std::vector<float> f;
    for (int k = 0; k < 4 * n; ++k) {
      const unsigned u = (unsigned)rng();
      float v;
      memcpy(&v, &u, 4);
      f.push_back(v);
    }
    for (float v : {0.f, -0.f, 1.f, -1.f, (float)inf, -(float)inf, (float)nan, std::numeric_limits<float>::min(),
                    std::numeric_limits<float>::denorm_min(), std::numeric_limits<float>::max()})
      f.push_back(v);
    float* df = to_device(f);
    dy = to_device(std::vector<double>(f.size()));
    eval_f2d<<<((int)f.size() + 255) / 256, 256>>>(df, dy, (int)f.size());
    const auto z = to_host(dy, f.size());
    bad = 0;
    for (size_t k = 0; k < f.size(); ++k)
      bad += std::isnan(f[k]) ? !std::isnan(z[k]) : bits(z[k]) != bits((double)f[k]);
    cudaFree(df);
    printf("f2d_bits     %9zu arguments, %lld mismatches\n", f.size(), bad);
    must(bad == 0, "f2d_bits");
  }
  {  // the training sigmoid: the reciprocal of its own 1 + exp(-z)
    std::vector<float> z;
    for (int k = 0; k < n; ++k) {
      z.push_back((float)((rng() >> 11) * 0x1p-53 * 180.0 - 86.0));
      z.push_back((float)((rng() >> 11) * 0x1p-53 * 16.0 - 8.0));
    }
    float *dz = to_device(z), *dy = to_device(z), *dd = to_device(z);
    eval_sigm<<<((int)z.size() + 255) / 256, 256>>>(dz, dy, dd, (int)z.size());
    const auto y = to_host(dy, z.size()), d = to_host(dd, z.size());
    long double worst = 0.0L;
    for (size_t k = 0; k < z.size(); ++k) {
      const long double r = 1.0L / (long double)d[k];
      worst = std::max(worst, fabsl((long double)y[k] - r) / ulp(r, 24));
    }
    printf("sigm_row     %9zu arguments, largest error %.7f ulp, bound 0.500001\n", z.size(), (double)worst);
    must(worst <= 0.500001L, "sigm_row");
    cudaFree(dz);
    const std::vector<float> s = {-88.f, -1000.f, -(float)inf, (float)inf, 1000.f, (float)nan};
    dz = to_device(s), dy = to_device(s), dd = to_device(s);
    eval_sigm<<<1, 256>>>(dz, dy, dd, (int)s.size());
    const auto t = to_host(dy, s.size());
    must(t[0] == 0.f && t[1] == 0.f && t[2] == 0.f && t[3] == 1.f && t[4] == 1.f && std::isnan(t[5]), "sigm_row's ends");
    cudaFree(dz);
    cudaFree(dd);
  }
  {  // a coordinate's cell: ListGenerate's FP64 floor, on and beside every cell face
    long long bad = 0, total = 0;
    struct Axis { double lo, size; int cells; };
    for (const Axis& a : {Axis{0.0, 0.0241, 400}, Axis{-0.0137, 0.013, 1023}, Axis{1234.567, 1e-3, 4000},
                          Axis{-3.0e-4, 3.25e-5, 50}, Axis{-987654.0, 0.37, 20000}, Axis{0.0, 1.0 / 3.0, 100}}) {
      GridDev g;
      memset(&g, 0, sizeof g);
      g.blpf[0] = a.lo;
      g.cell_size[0] = a.size;
      g.inv_cell_size32[0] = (float)(1.0 / a.size);
      g.blpf32[0] = (float)a.lo;
      std::vector<double> x = {0.0, -0.0, inf, -inf, nan, 1e300, -1e300, 5e-324};
      for (int c = -3; c <= a.cells + 3; ++c) {
        double at = a.lo + c * a.size;
        x.push_back(at);
        double up = at, down = at;
        for (int s = 0; s < 6; ++s) {
          x.push_back(up = nextafter(up, inf));
          x.push_back(down = nextafter(down, -inf));
        }
        for (double s : {1e-9, 1e-8, 1e-7, 1e-6, 1e-5, 1e-4}) {
          x.push_back(at + s * a.size);
          x.push_back(at - s * a.size);
        }
      }
      for (int k = 0; k < n / 4; ++k) x.push_back(a.lo + ((rng() >> 11) * 0x1p-53 * (a.cells + 6) - 3) * a.size);
      double* dx = to_device(x);
      int *dg = to_device(std::vector<int>(x.size())), *dw = to_device(std::vector<int>(x.size()));
      eval_cell<<<((int)x.size() + 255) / 256, 256>>>(g, dx, dg, dw, (int)x.size());
      const auto got = to_host(dg, x.size()), want = to_host(dw, x.size());
      cudaFree(dx);
      for (size_t k = 0; k < x.size(); ++k) bad += got[k] != want[k];
      total += (long long)x.size();
    }
    printf("cell_floor   %9lld arguments, %lld mismatches\n", total, bad);
    must(bad == 0, "cell_floor");
  }
  printf("failures %d\n", failures);
  return failures ? 1 : 0;
}
