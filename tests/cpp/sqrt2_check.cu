// Compares the packed square root of csrc/f32x2.cuh with sqrtf for every
// float from 1e-30 to the largest finite one; prints the number that differ.
#include <cstdio>

#include "../../granular_gpu_gb300/csrc/f32x2.cuh"

__global__ void k_compare(unsigned first, unsigned last, unsigned long long* differ) {
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  unsigned long long bad = 0;
  for (unsigned long long b = first + blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; b <= last; b += stride) {
    const float x = __uint_as_float((unsigned)b);
    float lo, hi;
    gg::unpack2(gg::sqrt2(gg::pack2(x, x)), lo, hi);
    const unsigned want = __float_as_uint(sqrtf(x));
    bad += __float_as_uint(lo) != want || __float_as_uint(hi) != want;
  }
  if (bad) atomicAdd(differ, bad);
}

int main() {
  unsigned long long* d = nullptr;
  unsigned long long bad = 0;
  if (cudaMalloc((void**)&d, sizeof(*d)) != cudaSuccess || cudaMemset(d, 0, sizeof(*d)) != cudaSuccess) return 2;
  k_compare<<<1216, 256>>>(0x0da24260u, 0x7f7fffffu, d);  // 1e-30f ... FLT_MAX
  if (cudaMemcpy(&bad, d, sizeof(bad), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  cudaFree(d);
  std::printf("differ: %llu\n", bad);
  return bad != 0;
}
