// The epilogues' SiLU against the division it stands for, for test_gpu_steps.py: every bf16 pattern once.
#include "../megabake_b200/csrc/device_common.cuh"

__global__ void sweep(unsigned* same, unsigned* differ) {
  const unsigned bits = blockIdx.x * blockDim.x + threadIdx.x;  // 65536 threads
  const float x = __uint_as_float(bits << 16);
  if (!(fabsf(x) < 80.f)) return;
  const float mine = mk::silu_inner(x), exact = mk::silu(x);
  const bool equal = __float_as_uint(mine) == __float_as_uint(exact) || (mine == 0.f && exact == 0.f);
  atomicAdd(equal ? same : differ, 1u);
}

// The activation that is rounded to bf16: the same bf16, and not a number where the other is none.
__global__ void sweep_rounded(unsigned* same, unsigned* differ) {
  const float x = __uint_as_float((blockIdx.x * blockDim.x + threadIdx.x) << 16);
  const __nv_bfloat16 mine = __float2bfloat16_rn(mk::silu_to_bf16(x)), exact = __float2bfloat16_rn(mk::silu(x));
  const bool equal = __bfloat16_as_ushort(mine) == __bfloat16_as_ushort(exact) || (__hisnan(mine) && __hisnan(exact));
  atomicAdd(equal ? same : differ, 1u);
}

template <typename Kernel>
static int count(Kernel kernel, unsigned* counts) {
  unsigned* device = nullptr;
  if (cudaMalloc(&device, 2 * sizeof(unsigned)) != cudaSuccess || cudaMemset(device, 0, 2 * sizeof(unsigned)) != cudaSuccess) return 1;
  kernel<<<256, 256>>>(device, device + 1);
  const cudaError_t done = cudaMemcpy(counts, device, 2 * sizeof(unsigned), cudaMemcpyDeviceToHost);
  cudaFree(device);
  return done == cudaSuccess ? 0 : 2;
}

extern "C" int silu_sweep(unsigned* counts) { return count(sweep, counts); }
extern "C" int silu_rounded_sweep(unsigned* counts) { return count(sweep_rounded, counts); }
