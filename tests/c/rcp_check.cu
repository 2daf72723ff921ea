// Reciprocals of rcp_d (clblm_fpconv.cuh) against the device's correctly
// rounded division, both by the GPU: random significands and those next to
// powers of two, over the exponents of AL2 + x^2 (2^-60 to 2^40) and beyond.
#include <cuda_runtime.h>

#include <cstdio>
#include <random>
#include <vector>

#include "clblm_fpconv.cuh"

using namespace clblm;

__global__ void k_check(const double* x, int n, unsigned long long* worst) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const long long a = __double_as_longlong(rcp_d(x[i])), b = __double_as_longlong(1.0 / x[i]);
  atomicMax(worst, (unsigned long long)(a > b ? a - b : b - a));
}

int main() {
  std::mt19937_64 g(11);
  std::uniform_real_distribution<double> u(1., 2.);
  std::vector<double> x;
  for (int e = -200; e <= 200; ++e) {
    for (int k = 0; k < 5000; ++k) x.push_back(std::ldexp(u(g), e));
    double lo = std::ldexp(1., e), hi = std::ldexp(2., e);
    for (int k = 0; k < 50; ++k) {
      x.push_back(lo);
      lo = std::nextafter(lo, 1e300);
      hi = std::nextafter(hi, 0.);
      x.push_back(hi);
    }
  }
  const int n = (int)x.size();
  double* d = nullptr;
  unsigned long long *w = nullptr, worst = ~0ull;
  bool ok = cudaMalloc(&d, sizeof(double) * n) == cudaSuccess && cudaMalloc(&w, 8) == cudaSuccess &&
            cudaMemcpy(d, x.data(), sizeof(double) * n, cudaMemcpyHostToDevice) == cudaSuccess &&
            cudaMemset(w, 0, 8) == cudaSuccess;
  if (ok) {
    k_check<<<(n + 255) / 256, 256>>>(d, n, w);
    ok = cudaGetLastError() == cudaSuccess && cudaMemcpy(&worst, w, 8, cudaMemcpyDeviceToHost) == cudaSuccess;
  }
  printf("reciprocals %d, units in the last place apart at most %llu%s\n", n, worst, ok ? "" : " (CUDA error)");
  return !(ok && worst <= 1);
}
