// Waits for barriers that nothing completes, until the limit of csrc/ptx.cuh ends them: prints a line
// "<form> <milliseconds> <gave up>" for the form with a limit of its own, for the one with a limit shared by several
// waits, and for the one that waits for other CTAs' pushes.  Barriers that are ready come first: those waits must not give up.
#include "ptx.cuh"

#include <cstdio>

using namespace logos::ptx;

__global__ void wait_limit(int form, int* out) {
  __shared__ uint64_t open_bar, done_bar;
  if (threadIdx.x == 0) {
    mbar_init(&open_bar, 1);
    mbar_init(&done_bar, 1);
    fence_barrier_init();
    mbar_arrive(&done_bar);
  }
  __syncthreads();
  const uint32_t open_a = smem_u32(&open_bar), done_a = smem_u32(&done_bar);
  if (form == 0) {
    const bool ready = mbar_wait(&done_bar, 0);
    const bool ok = mbar_wait(&open_bar, 0);
    if (threadIdx.x == 0) out[0] = ready && !ok;
  } else if (form == 2) {
    const bool ready = mbar_wait_cluster(&done_bar, 0);
    const bool ok = mbar_wait_cluster(&open_bar, 0);
    if (threadIdx.x == 0) out[0] = ready && !ok;
  } else {
    uint32_t since = wait_start();
    mbar_wait2(done_a, 0, done_a, 0, &since);
    const bool ready = since != WAIT_OVER;
    mbar_wait3(done_a, 0, open_a, 0, done_a, 0, &since);
    mbar_wait(open_a, 0, &since);   // the limit is over: returns after a poll
    if (threadIdx.x == 0) out[0] = ready && since == WAIT_OVER;
  }
}

int main() {
  int *out = nullptr, gave_up = 0;
  if (cudaMalloc(&out, sizeof(int)) != cudaSuccess) return 2;
  for (int form = 0; form < 3; ++form) {
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    cudaMemset(out, 0, sizeof(int));
    cudaEventRecord(a);
    wait_limit<<<1, 32>>>(form, out);
    cudaEventRecord(b);
    if (cudaDeviceSynchronize() != cudaSuccess) return 3;
    float ms = 0.f;
    cudaEventElapsedTime(&ms, a, b);
    cudaMemcpy(&gave_up, out, sizeof(int), cudaMemcpyDeviceToHost);
    printf("%d %.1f %d\n", form, ms, gave_up);
  }
  return 0;
}
