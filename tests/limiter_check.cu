// The reverse mode's limiter function (limiter_value, mcfd_device.cuh) against
// the forward quotient bit for bit, and its slope against long double on the
// host, over ratios from tiny to past the cap.
//
// usage: limiter_check N -> "cases=<n> values=<differing> slope=<worst relative error / eps>"
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../meshcfd_gb300/csrc/mcfd_device.cuh"

using namespace mcfd;

template <int L>
__global__ void k_limiter(int n, const double* __restrict__ r, double* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double slope;
  out[3 * i] = limiter_value<L>(r[i], &slope);
  out[3 * i + 1] = slope;
  // ratio r: an increment of 1 towards an extreme r away; the forward takes the
  // minimum with 1, which an overflowing inf / inf does not lower
  const double f = limiter_face_factor<L>(0.0, 1.0, 0.0, r[i], 1e-14);
  out[3 * i + 2] = icmp::lt_nonneg(f, 1.0) ? f : 1.0;
}

int main(int argc, char** argv) {
  const int n = argc > 1 ? std::atoi(argv[1]) : 100000;
  std::vector<double> r(n), out(3 * (size_t)n);
  unsigned long long state = 5;
  for (int i = 0; i < n; ++i) {
    state = state * 6364136223846793005ull + 1442695040888963407ull;
    const double u = (double)(state >> 11) * 0x1p-53;
    r[i] = i % 3 == 0 ? 3.0 * u : i % 3 == 1 ? u : std::exp2(-60.0 * u);
  }
  r[0] = 0.0, r[1] = 1.0, r[2] = 2.0, r[3] = 1e300, r[4] = std::nextafter(1.0, 0.0), r[5] = std::nextafter(2.0, 0.0);
  double *dr, *dout;
  if (cudaMalloc((void**)&dr, n * sizeof(double)) != cudaSuccess ||
      cudaMalloc((void**)&dout, out.size() * sizeof(double)) != cudaSuccess)
    return 1;
  cudaMemcpy(dr, r.data(), n * sizeof(double), cudaMemcpyHostToDevice);
  int values = 0;
  double worst = 0.0;
  for (int L = 0; L < 4; ++L) {
    const int b = (n + 255) / 256;
    if (L == 0) k_limiter<0><<<b, 256>>>(n, dr, dout);
    if (L == 1) k_limiter<1><<<b, 256>>>(n, dr, dout);
    if (L == 2) k_limiter<2><<<b, 256>>>(n, dr, dout);
    if (L == 3) k_limiter<3><<<b, 256>>>(n, dr, dout);
    if (cudaMemcpy(out.data(), dout, out.size() * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    for (int i = 0; i < n; ++i) {
      if (out[3 * i] != out[3 * i + 2] && values++ < 5)
        std::printf("limiter %d at %a: %a, forward %a\n", L, r[i], out[3 * i], out[3 * i + 2]);
      const long double x = r[i], D = x * x + x + 2.0L + 1e-12L, N = x * x + 2.0L * x + 1e-12L;
      long double s = 0.0L;
      if (L <= 1) s = r[i] < 1.0;
      else if (L == 2) s = r[i] > 0.0 && r[i] < 1.0 ? 2.0L / ((1.0L + x) * (1.0L + x)) : 0.0L;
      else if (out[3 * i + 2] < 1.0)  // on the side of the cap that the forward takes
        s = ((2.0L * x + 2.0L) * D - N * (2.0L * x + 1.0L)) / (D * D);
      if (out[3 * i + 1] != 0.0 || s != 0.0L)
        worst = std::fmax(worst, (double)(fabsl((long double)out[3 * i + 1] - s) / fmaxl(fabsl(s), 1e-300L)) * 0x1p52);
    }
  }
  std::printf("cases=%d values=%d slope=%.2f\n", n, values, worst);
  return values ? 1 : 0;
}
