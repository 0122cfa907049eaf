// Largest relative errors of the FP64 reciprocal square roots over two binades (every exponent behaves as one of
// them): prints those of the approximation instruction, rsqrt_any<1> and rsqrt_any<2>, and fails on CUDA errors.
#include <cstdio>
#include <vector>

#include "kernels.cuh"

__global__ void k_errors(long long n, double* out) {
  double m[3] = {0, 0, 0};
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    // 1 <= x < 4, the low bits of the significand varied too
    const double x = 1.0 + 3.0 * ((double)i + 0.5) / (double)n;
    const double r = 1.0 / sqrt(x);
    const double y[3] = {xfmm::rsqrt_approx64(x), xfmm::rsqrt_any<1>(x), xfmm::rsqrt_any<2>(x)};
    for (int k = 0; k < 3; k++) m[k] = fmax(m[k], fabs(y[k] - r) / r);
  }
  for (int k = 0; k < 3; k++) out[3 * (blockIdx.x * blockDim.x + threadIdx.x) + k] = m[k];
}

int main() {
  constexpr int BLOCKS = 592, THREADS = 256;
  std::vector<double> h(3 * BLOCKS * THREADS);
  double* d = nullptr;
  if (cudaMalloc(&d, h.size() * sizeof(double)) != cudaSuccess) return 1;
  k_errors<<<BLOCKS, THREADS>>>(1ll << 28, d);
  if (cudaMemcpy(h.data(), d, h.size() * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  double m[3] = {0, 0, 0};
  for (size_t i = 0; i < h.size(); i++) m[i % 3] = h[i] > m[i % 3] ? h[i] : m[i % 3];
  printf("%.6e %.6e %.6e\n", m[0], m[1], m[2]);
  return 0;
}
