// Every gate that takes the shorter division of SwiGLU: prints how many of them there are, and how many give other bits.
#include <cstdio>

#include "act.cuh"

__device__ unsigned long long taken, other;

__global__ void gates() {
  unsigned long long t = 0, o = 0;
  for (unsigned long long i = blockIdx.x * 256ull + threadIdx.x; i < 1ull << 32; i += gridDim.x * 256ull) {
    const float g = __uint_as_float((unsigned)i);
    if (!logos::silu_plain(g)) continue;
    ++t;
    o += __float_as_uint(logos::silu_f(g)) != __float_as_uint(logos::silu_markstein(g));
  }
  atomicAdd(&taken, t);
  atomicAdd(&other, o);
}

int main() {
  gates<<<2048, 256>>>();
  unsigned long long t = 0, o = 0;
  if (cudaMemcpyFromSymbol(&t, taken, sizeof(t)) != cudaSuccess || cudaMemcpyFromSymbol(&o, other, sizeof(o)) != cudaSuccess) return 1;
  printf("%llu %llu\n", t, o);
  return 0;
}
