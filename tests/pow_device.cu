// The fixed-point power on the device (its own wide products and tables)
// against the same header's host build, bit for bit, on the operands that the
// fixed-point path takes.
//
// usage: pow_device N SEED -> "cases=<n> different=<n>"
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "../meshcfd_gb300/csrc/mcfd_pow.cuh"

static unsigned long long g_state;
static double uniform() {
  unsigned long long z = (g_state += 0x9e3779b97f4a7c15ull);
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return (double)((z ^ (z >> 31)) >> 11) * 0x1p-53;
}

__global__ void k_pow(int n, const double* __restrict__ x, const double* __restrict__ y, double* __restrict__ r) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) r[i] = mcfd::pow_rn(x[i], y[i]);
}

int main(int argc, char** argv) {
  const int n = argc > 1 ? std::atoi(argv[1]) : 100000;
  g_state = argc > 2 ? std::strtoull(argv[2], nullptr, 10) : 1;
  const double fixed[] = {1.4, 1.0 / (1.4 - 1.0), 1.4 / (1.4 - 1.0), 1.5, 0.4, 5.0 / 3.0, -1.0, 2.0, 64.0, 0x1p-40};
  std::vector<double> x(n), y(n), r(n);
  for (int i = 0; i < n; ++i) {
    y[i] = i % 3 == 0 ? fixed[(i / 3) % 10] : (uniform() - 0.5) * (i % 3 == 1 ? 16.0 : 128.0);
    if (std::fabs(y[i]) < 0x1p-40) y[i] = 1.0;
    double span = i % 4 == 0 ? 0.001 : i % 4 == 1 ? 1.0 : i % 4 == 2 ? 20.0 : 1000.0;
    span = std::fmin(span, 1000.0 / (std::fabs(y[i]) + 1.0));  // results stay in the normal range
    x[i] = i % 97 == 0 ? 1.0 : std::exp2((2.0 * uniform() - 1.0) * span);
  }
  double *dx, *dy, *dr;
  const size_t bytes = n * sizeof(double);
  if (cudaMalloc((void**)&dx, bytes) != cudaSuccess || cudaMalloc((void**)&dy, bytes) != cudaSuccess ||
      cudaMalloc((void**)&dr, bytes) != cudaSuccess)
    return 1;
  cudaMemcpy(dx, x.data(), bytes, cudaMemcpyHostToDevice);
  cudaMemcpy(dy, y.data(), bytes, cudaMemcpyHostToDevice);
  k_pow<<<(n + 255) / 256, 256>>>(n, dx, dy, dr);
  if (cudaMemcpy(r.data(), dr, bytes, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
  int different = 0;
  for (int i = 0; i < n; ++i) {
    const double h = mcfd::pow_rn(x[i], y[i]);
    if (std::memcmp(&h, &r[i], sizeof(h)) != 0 && different++ < 5)
      std::printf("%a ^ %a: device %a, host %a\n", x[i], y[i], r[i], h);
  }
  std::printf("cases=%d different=%d\n", n, different);
  return different ? 1 : 0;
}
