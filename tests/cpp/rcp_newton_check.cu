// Reciprocals of random numbers by the secular solver's Newton steps against
// correctly rounded ones: prints the largest distance in units of the last place
// over the range the function states, then its results at 0, a subnormal and
// infinity.
#include <stdio.h>
#include <string.h>

#include <cmath>
#include <limits>
#include <random>
#include <vector>

#include "dc_secular.cuh"

__global__ void rcp_kernel(const double* x, double* r, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) r[i] = nrgb::rcp_newton(x[i]);
}

static long long bits(double x) {
  long long b;
  memcpy(&b, &x, sizeof b);
  return b;
}

int main() {
  const int per = 4000, n = 2001 * per + 3;
  std::vector<double> x(n), r(n);
  std::mt19937_64 g(1);
  std::uniform_real_distribution<double> u(1.0, 2.0);
  int k = 0;
  for (int e = -1000; e <= 1000; ++e)
    for (int i = 0; i < per; ++i) {
      // the binade's ends, and numbers between them
      double m = i == 0 ? 1.0 : i == 1 ? std::nextafter(2.0, 1.0) : i == 2 ? std::nextafter(1.0, 2.0) : u(g);
      if (e == 1000) m = 1.0;
      x[k++] = std::ldexp((i & 1) ? -m : m, e);
    }
  x[k++] = 0.0;
  x[k++] = std::numeric_limits<double>::denorm_min() * 12345;
  x[k++] = INFINITY;
  double *dx = nullptr, *dr = nullptr;
  if (cudaMalloc(&dx, n * sizeof(double)) != cudaSuccess || cudaMalloc(&dr, n * sizeof(double)) != cudaSuccess ||
      cudaMemcpy(dx, x.data(), n * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess)
    return 1;
  rcp_kernel<<<(n + 255) / 256, 256>>>(dx, dr, n);
  if (cudaMemcpy(r.data(), dr, n * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
  long long worst = 0;
  for (int i = 0; i < n - 3; ++i) {
    const long long d = std::llabs(bits(r[i]) - bits(1.0 / x[i]));
    if (d > worst || r[i] != r[i]) worst = r[i] != r[i] ? 1ll << 62 : d;
  }
  printf("%lld %d %d %d\n", worst, std::isnan(r[n - 3]), std::isnan(r[n - 2]), std::isnan(r[n - 1]));
  return 0;
}
