// rsqrt64 (csrc/wide.cuh) on every high word of [1, 4), with the low words at
// their ends and a few between, and at other exponents: prints the largest
// |1 - x y^2| of the SFU's estimate y and the largest relative error of rsqrt64.
#include <cstdint>
#include <cstdio>

#include "../../galactic-tides_gb300/csrc/wide.cuh"

__device__ void keep_most(unsigned long long *at, double v) {
  atomicMax(at, static_cast<unsigned long long>(__double_as_longlong(fabs(v))));
}

__global__ void k_check(unsigned long long *most) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;  // below 2^21
  const uint32_t lows[4] = {0u, 0x80000001u, 0xfffffffeu, 0xffffffffu};
  double e_most = 0.0, r_most = 0.0;
  for (int shift = -900; shift <= 900; shift += 300)
    for (uint32_t low : lows) {
      const double x = __hiloint2double(static_cast<int>((1023u << 20) + k + (static_cast<uint32_t>(shift) << 20)),
                                        static_cast<int>(low));
      // 1 - x v^2, exact up to 2^-104: v^2 = t + tl
      auto deficit = [&](double v) {
        const double t = v * v, tl = fma(v, v, -t);
        return fma(-x, tl, fma(-x, t, 1.0));
      };
      e_most = fmax(e_most, fabs(deficit(gtc::rsqrt64_estimate(x))));
      r_most = fmax(r_most, 0.5 * fabs(deficit(gtc::rsqrt64(x))));
    }
  keep_most(most, e_most);
  keep_most(most + 1, r_most);
}

int main() {
  unsigned long long *most = nullptr, host[2] = {};
  if (cudaMalloc(&most, sizeof host) != cudaSuccess) return 2;
  cudaMemset(most, 0, sizeof host);
  k_check<<<(1u << 21) / 256, 256>>>(most);
  const cudaError_t e = cudaDeviceSynchronize();
  cudaMemcpy(host, most, sizeof host, cudaMemcpyDeviceToHost);
  double v[2];
  static_assert(sizeof v == sizeof host);
  __builtin_memcpy(v, host, sizeof v);
  std::printf("estimate %.6e result %.6e status %s\n", v[0], v[1], cudaGetErrorString(e));
  cudaFree(most);
  return e == cudaSuccess ? 0 : 1;
}
