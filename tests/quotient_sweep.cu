// The softmax's quotients against the division they stand for, for test_gpu_steps.py: 2^26 weights up to 1 over sums from 1 on.
#include "../megabake_b200/csrc/device_common.cuh"

__device__ unsigned scrambled(unsigned x) {  // a bijection of 32-bit words
  x = (x ^ (x >> 16)) * 0x21F0AAADu;
  x = (x ^ (x >> 15)) * 0x735A2D97u;
  return x ^ (x >> 15);
}

// Weights of every exponent down to the least normal number, with zero and one among them; sums below 2^20, a quarter of them
// within 64 units in the last place of a power of two, where a rounded reciprocal is worst.
__global__ void sweep(unsigned* counts) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x, a = scrambled(i), b = scrambled(~i);
  float weight = __uint_as_float((1u + a % 126u) << 23 | (a >> 9));
  if ((i & 255u) == 0) weight = (i & 256u) ? 1.f : 0.f;
  unsigned mantissa = b >> 9;
  if ((b & 3u) == 0) mantissa = (b & 4u) ? (mantissa & 63u) : 0x7FFFFFu - (mantissa & 63u);
  const float sum = __uint_as_float((127u + (b >> 3) % 20u) << 23 | mantissa);
  if (!mk::quotient_fits(weight)) {
    atomicAdd(counts + 2, 1u);
    return;
  }
  const float mine = mk::quotient(weight, sum, 1.0f / sum), exact = weight / sum;
  if (__float_as_uint(mine) != __float_as_uint(exact)) atomicAdd(counts + 1, 1u);
  else if ((threadIdx.x & 31u) == 0) atomicAdd(counts, 1u);
}

extern "C" int quotient_sweep(unsigned* counts) {
  unsigned* device = nullptr;
  if (cudaMalloc(&device, 3 * sizeof(unsigned)) != cudaSuccess || cudaMemset(device, 0, 3 * sizeof(unsigned)) != cudaSuccess) return 1;
  sweep<<<1 << 18, 256>>>(device);
  const cudaError_t done = cudaMemcpy(counts, device, 3 * sizeof(unsigned), cudaMemcpyDeviceToHost);
  cudaFree(device);
  return done == cudaSuccess ? 0 : 2;
}
