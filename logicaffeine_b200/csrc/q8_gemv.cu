// Q8 GEMV: y[n] = sum_kb s[n,kb] * sum_{k in kb} q[n,k] * x[k].
//
// HBM-bound: 1.125 bytes of weights per multiply-add, so the kernel is a coalesced stream that must
// not stop while the products are computed.  Every warp owns a ring of three 2 KiB stages of weights
// (with their scales) in shared memory and fills it itself with asynchronous copies: a lane copies
// the bytes that it will use, so nothing wider than the warp ever waits, and an SM keeps up to 100 KiB
// in flight whatever its warps compute.  int8 -> f32 uses the 2^23 mantissa trick (one byte-permute
// and one subtract), the half-block dot product is scaled by its block's f32 scale in registers, and
// the row sum is a warp-shuffle reduction.  x lives in shared memory, laid out so that the four
// 128-bit reads a lane needs are bank-conflict free; a warp takes two rows at a time, because a row at
// a time needs four bytes of x for a byte of weights from the same port.
#include "ops.cuh"

#include <algorithm>

namespace logos {

namespace {

constexpr int GEMV_DEPTH = 3;                     // stages of a warp's ring
constexpr int GEMV_WARPS = 24, GEMV_FEW_WARPS = 16;  // a CTA has; one CTA fills an SM
constexpr int GEMV_STAGE = 2048 + 64 * 4;         // 128 chunks of 16 weights, 64 scales
constexpr int GEMV_SMEM = 227 * 1024;

// byte `sel` of the bias-flipped word -> exact float value of the int8
__device__ __forceinline__ float byte_to_f32(uint32_t w_xor80, uint32_t selector) {
  // 0x4B0000bb = 2^23 + bb ; bb = q + 128
  uint32_t bits = __byte_perm(w_xor80, 0x4B000000u, selector);
  return __uint_as_float(bits) - 8388736.0f;
}

__device__ __forceinline__ float dot4(uint32_t w, float4 x, float acc) {
  uint32_t u = w ^ 0x80808080u;
  acc = fmaf(byte_to_f32(u, 0x7650), x.x, acc);
  acc = fmaf(byte_to_f32(u, 0x7651), x.y, acc);
  acc = fmaf(byte_to_f32(u, 0x7652), x.z, acc);
  acc = fmaf(byte_to_f32(u, 0x7653), x.w, acc);
  return acc;
}

// xs4 layout: chunk c (16 floats) is split into 4 float4; float4 j of chunk c
// sits at index (c/32)*128 + j*32 + (c%32), so the 32 lanes of a warp reading
// the same j of consecutive chunks touch consecutive 16-byte slots.
__device__ __forceinline__ int xs4_index(int chunk, int j) { return (chunk >> 5) * 128 + j * 32 + (chunk & 31); }

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}

// A warp takes R neighbouring rows (a group); groups go round the CTAs first, so that a small matrix still
// uses every SM.  The ring runs on from one group to the next.  Measured before (eight loads a lane in flight in
// registers, four CTAs an SM) -> now: 152064 x 5120 197 -> 148 us (5.9 TB/s), 151936 x 896 72 -> 38 us,
// 27648 x 5120 43 -> 33 us, 5120 x 27648 154 -> 45 us, 300 x 16384 13.6 -> 8.4 us.  Four rows at a time
// measured 166 us on the first, one row 164 us.
template <int R, bool X_IN_SMEM>
__global__ void __launch_bounds__(GEMV_WARPS * 32, 1)
q8_gemv_kernel(const int8_t* __restrict__ q, const float* __restrict__ s, const float* __restrict__ x,
               float* __restrict__ y, int64_t n, int64_t k, bool early) {
  constexpr int U = 4 / R;   // chunks of a row that a lane has in a stage
  extern __shared__ float4 xs4[];
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5, warps = blockDim.x >> 5;
  const int chunks = (int)(k >> 4);  // 16-element chunks per row
  const int kb = (int)(k >> 5);
  const int xchunks = X_IN_SMEM ? (chunks + 31) / 32 * 32 : 0;
  uint8_t* ring = reinterpret_cast<uint8_t*>(xs4 + xchunks * 4) + warp * (GEMV_DEPTH * GEMV_STAGE);
  const uint32_t ring_a = (uint32_t)__cvta_generic_to_shared(ring);
  // In a caller's scope the weights are read before the previous kernel of the stream has finished (the scope promises
  // that nothing in it writes them); x and y wait for it.
  if (!early) pdl_wait();
  pdl_trigger();
  const int64_t groups = (n + R - 1) / R, step = (int64_t)gridDim.x * warps;
  int64_t lg = blockIdx.x + (int64_t)gridDim.x * warp;   // the load cursor
  int lc = 0, lslot = 0;
  // the next stage; a row past the end repeats the last one.  Always a commit group, so that the waits count right
  auto load = [&]() {
    if (lg < groups) {
      const uint32_t at = ring_a + lslot * GEMV_STAGE;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int64_t row = min(lg * R + r, n - 1);
        const int8_t* qr = q + row * k;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int c = lc + 32 * u + lane;
          if (c < chunks) cp_async16(at + (r * U + u) * 512 + lane * 16, qr + (int64_t)c * 16);
        }
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int i = lane + 32 * h, r = i / (16 * U), blk = (lc >> 1) + i % (16 * U);
        if (blk < kb) cp_async4(at + 2048 + i * 4, s + min(lg * R + r, n - 1) * kb + blk);
      }
      lc += 32 * U;
      if (lc >= chunks) {
        lc = 0;
        lg += step;
      }
      lslot = lslot + 1 == GEMV_DEPTH ? 0 : lslot + 1;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int i = 0; i < GEMV_DEPTH - 1; ++i) load();
  if (early) pdl_wait();
  if (X_IN_SMEM) {
    const float4* xg = reinterpret_cast<const float4*>(x);
    for (int i = tid; i < chunks * 4; i += blockDim.x) xs4[xs4_index(i >> 2, i & 3)] = __ldcg(xg + i);
    __syncthreads();
  }
  int slot = 0;
  for (int64_t g = blockIdx.x + (int64_t)gridDim.x * warp; g < groups; g += step) {
    float acc[R];
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = 0.f;
    for (int c0 = 0; c0 < chunks; c0 += 32 * U) {
      __syncwarp();   // every lane is done with the stage that the next load overwrites
      load();
      asm volatile("cp.async.wait_group %0;" ::"n"(GEMV_DEPTH - 1) : "memory");
      __syncwarp();
      const uint8_t* st = ring + slot * GEMV_STAGE;
      slot = slot + 1 == GEMV_DEPTH ? 0 : slot + 1;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int c = c0 + 32 * u + lane;
        if (c < chunks) {
          uint4 w[R];
          float p[R];
#pragma unroll
          for (int r = 0; r < R; ++r) {
            w[r] = *reinterpret_cast<const uint4*>(st + (r * U + u) * 512 + lane * 16);
            p[r] = 0.f;
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float4 xv = X_IN_SMEM ? xs4[xs4_index(c, j)] : __ldcg(reinterpret_cast<const float4*>(x) + (int64_t)c * 4 + j);
#pragma unroll
            for (int r = 0; r < R; ++r) p[r] = dot4(j == 0 ? w[r].x : j == 1 ? w[r].y : j == 2 ? w[r].z : w[r].w, xv, p[r]);
          }
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const float sc = *reinterpret_cast<const float*>(st + 2048 + (r * 16 * U + 16 * u + (lane >> 1)) * 4);
            acc[r] = fmaf(sc, p[r], acc[r]);
          }
        }
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], o);
      if (lane == 0 && g * R + r < n) y[g * R + r] = acc[r];
    }
  }
}


}  // namespace

logos_status_t launch_q8_gemv(const int8_t* q, const float* s, const float* x, float* y, int64_t n, int64_t k,
                              int device, cudaStream_t st) {
  if (n == 0) return LOGOS_OK;
  if (k == 0) {
    LOGOS_CUDA_TRY(cudaMemsetAsync(y, 0, sizeof(float) * n, st));
    return LOGOS_OK;
  }
  // two rows a warp unless that would leave more than half of the warps without any; the larger CTA where x fits
  // beside its rings (K up to 16384), past K = 30208 x stays in global memory
  const int64_t sms = sm_count(device);
  const int rows = n <= sms * GEMV_WARPS ? 1 : 2;
  const int64_t groups = (n + rows - 1) / rows;
  const int64_t xb = (k / 16 + 31) / 32 * 128 * (int64_t)sizeof(float4);
  auto ring = [](int warps) { return (int64_t)warps * GEMV_DEPTH * GEMV_STAGE; };
  const int warps = ring(GEMV_WARPS) + xb <= GEMV_SMEM ? GEMV_WARPS : GEMV_FEW_WARPS;
  const bool in_smem = ring(warps) + xb <= GEMV_SMEM;
  auto kern = rows == 2 ? (in_smem ? q8_gemv_kernel<2, true> : q8_gemv_kernel<2, false>)
                        : (in_smem ? q8_gemv_kernel<1, true> : q8_gemv_kernel<1, false>);
  LOGOS_TRY(allow_smem(reinterpret_cast<const void*>(kern), device, GEMV_SMEM));
  LOGOS_CUDA_TRY(launch_kernel(kern, dim3((unsigned)std::min(groups, sms)), dim3(warps * 32), (size_t)(ring(warps) + (in_smem ? xb : 0)),
                               st, q, s, x, y, n, k, pdl_early()));
  count_launch(LK_GEMV);
  return check_launch("q8_gemv_kernel");
}

}  // namespace logos

using namespace logos;

extern "C" logos_status_t logos_q8_gemv(logos_handle_t q, logos_handle_t s, logos_handle_t x, logos_handle_t y,
                                        int64_t n, int64_t k, void* stream_or_null) {
  return guarded([&]() -> logos_status_t {
    if (n < 0 || k < 0) return fail(LOGOS_OUT_OF_BOUNDS, "logos_q8_gemv: negative extent");
    if (k % 32) return fail(LOGOS_OUT_OF_BOUNDS, "logos_q8_gemv: K=%lld is not a multiple of the block size 32", (long long)k);
    int8_t* qp; float* sp; float* xp; float* yp;
    int32_t dev = 0;
    LOGOS_TRY(buf_ptr<int8_t>(q, n * k, "q", &qp, &dev));
    LOGOS_TRY(buf_ptr<float>(s, n * (k / 32), "s", &sp));
    LOGOS_TRY(buf_ptr<float>(x, k, "x", &xp));
    LOGOS_TRY(buf_ptr<float>(y, n, "y", &yp));
    LOGOS_CUDA_TRY(cudaSetDevice(dev));
    const cudaStream_t st = as_stream(stream_or_null);
    OrderedScope ordered(st);
    return launch_q8_gemv(qp, sp, xp, yp, n, k, dev, st);
  });
}
