// Every float bit pattern x, for each number s of fluid neighbours (0 to 4): the
// fast-math division x / s by a run-time s, as apply_projection_at divides the
// divergence (src/fluid.cu:240), against the product x * __fdividef(1, s) that the
// projection's tiles compute by the flags and beside walls. Built with the
// reference's Release flags (--use_fast_math), as the library is.
//
// Prints one line per s: "<s> <inputs whose results differ> <first such input,
// hex>"; a NaN from both counts as the same result.
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>

__global__ void k_compare(int s, unsigned long long* mismatches, unsigned int* first) {
  const float rs = __fdividef(1.0f, (float)s);
  unsigned long long local = 0;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < (1ull << 32);
       t += stride) {
    const float x = __uint_as_float((unsigned int)t);
    const float a = x / (float)s;
    const float b = __fmul_rn(x, rs);
    if (!(__float_as_uint(a) == __float_as_uint(b) || (a != a && b != b))) {
      local++;
      atomicMin(first, (unsigned int)t);
    }
  }
  if (local) atomicAdd(mismatches, local);
}

int main() {
  unsigned long long* d_count = nullptr;
  unsigned int* d_first = nullptr;
  int sms = 0;
  if (cudaMalloc(&d_count, sizeof(*d_count)) != cudaSuccess ||
      cudaMalloc(&d_first, sizeof(*d_first)) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, 0) != cudaSuccess)
    return 1;
  for (int s = 0; s <= 4; s++) {
    unsigned long long count = 0;
    unsigned int first = 0xffffffffu;
    cudaMemcpy(d_count, &count, sizeof(count), cudaMemcpyHostToDevice);
    cudaMemcpy(d_first, &first, sizeof(first), cudaMemcpyHostToDevice);
    k_compare<<<sms * 8, 256>>>(s, d_count, d_first);
    const cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess) {
      fprintf(stderr, "kernel: %s\n", cudaGetErrorString(e));
      return 1;
    }
    cudaMemcpy(&count, d_count, sizeof(count), cudaMemcpyDeviceToHost);
    cudaMemcpy(&first, d_first, sizeof(first), cudaMemcpyDeviceToHost);
    printf("%d %llu %08x\n", s, count, first);
  }
  cudaFree(d_count);
  cudaFree(d_first);
  return 0;
}
