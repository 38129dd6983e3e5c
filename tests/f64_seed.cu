// The approximate reciprocal that the FP64 face quotients start from, over all of
// its inputs: every upper significand field at both ends of the lower word (the
// seed reads the upper 32 bits only, checked on a third lower word).  Prints the
// largest e = |1 - b y| and the smallest ratio of what a field's denominators
// b = 2 (1 - n) have, n, to what exact quotients ask for, e/2 + 2^52 e^4
// (fv_f64.cuh), over the fields the guard lets pass.
#include <cmath>
#include <cstdio>
#include <vector>

#include "fv_f64.cuh"

__global__ void seed_errors(double* err, int* bad)
{
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  const double b0 = __hiloint2double(1023 << 20 | m, 0), b1 = __hiloint2double(1023 << 20 | m, -1);
  const double y = dn::rcp_seed(b0);
  if (dn::rcp_seed(b1) != y || dn::rcp_seed(__hiloint2double(1023 << 20 | m, m * 40503)) != y) atomicOr(bad, 1);
  const double e = fmax(fabs(fma(-b0, y, 1.0)), fabs(fma(-b1, y, 1.0)));
  dn::Guard g;
  g.den(b1);
  err[m] = g.any() ? -e : e;
}

int main()
{
  constexpr int n = 1 << 20;
  double* err;
  int* bad;
  if (cudaMalloc(&err, n * sizeof(double)) != cudaSuccess || cudaMalloc(&bad, sizeof(int)) != cudaSuccess) return 2;
  cudaMemset(bad, 0, sizeof(int));
  seed_errors<<<n / 256, 256>>>(err, bad);
  std::vector<double> h(n);
  int b = 0;
  if (cudaMemcpy(h.data(), err, n * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  if (cudaMemcpy(&b, bad, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  double top = 0, room = 1e300;
  for (int m = 0; m < n; ++m) {
    const double e = std::fabs(h[m]);
    top = std::fmax(top, e);
    if (h[m] >= 0) room = std::fmin(room, std::ldexp(n - 1 - m, -21) / (e / 2 + std::ldexp(e * e * e * e, 52)));
  }
  std::printf("%.17g %.17g\n", top, room);
  return b;
}
