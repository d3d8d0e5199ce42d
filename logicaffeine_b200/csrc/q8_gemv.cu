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

__device__ __forceinline__ float4 four_f32(uint32_t w) {
  const uint32_t u = w ^ 0x80808080u;
  return make_float4(byte_to_f32(u, 0x7650), byte_to_f32(u, 0x7651), byte_to_f32(u, 0x7652), byte_to_f32(u, 0x7653));
}
__device__ __forceinline__ float dot4(float4 w, float4 x, float acc) {
  acc = fmaf(w.x, x.x, acc);
  acc = fmaf(w.y, x.y, acc);
  acc = fmaf(w.z, x.z, acc);
  acc = fmaf(w.w, x.w, acc);
  return acc;
}

// four neighbouring values of x, past L1; x is what the previous kernel wrote
__device__ __forceinline__ float4 load_x4(const float* x, int64_t i) { return __ldcg(reinterpret_cast<const float4*>(x) + i); }
__device__ __forceinline__ float4 load_x4(const __nv_bfloat16* x, int64_t i) {
  const uint2 v = __ldcg(reinterpret_cast<const uint2*>(x) + i);
  return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16),
                     __uint_as_float(v.y & 0xffff0000u));
}
// sums of two neighbouring rows' (R = 2) or one row's product with one vector -> results, in T
__device__ __forceinline__ void store_y(float* y, const float*, int, int64_t at, float v) { y[at] = v; }
__device__ __forceinline__ void store_y(__nv_bfloat16* y, const __nv_bfloat16* aux, int epilogue, int64_t at, float v) {
  if (epilogue == EPI_RESIDUAL) v = __fadd_rn(v, __bfloat162float(aux[at]));
  y[at] = __float2bfloat16_rn(v);
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
// M vectors of x at a time (rows of an [M][K] matrix, in T), as the GEMM operators have for a few tokens: a weight is
// converted once for all of them, and their results go through the GEMM's epilogues.
template <int R, bool X_IN_SMEM, int M, typename T, bool STATUS>
__global__ void __launch_bounds__(GEMV_WARPS * 32, 1)
q8_gemv_kernel(const int8_t* __restrict__ q, const float* __restrict__ s, const T* __restrict__ x, T* y, int64_t n, int64_t k, bool early,
               const T* aux, int epilogue, const int* status) {
  constexpr int U = 4 / R;   // chunks of a row that a lane has in a stage
  extern __shared__ float4 xs4[];
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5, warps = blockDim.x >> 5;
  const int chunks = (int)(k >> 4);  // 16-element chunks per row
  const int kb = (int)(k >> 5);
  const int xchunks = X_IN_SMEM ? (chunks + 31) / 32 * 32 : 0;
  uint8_t* ring = reinterpret_cast<uint8_t*>(xs4 + M * xchunks * 4) + warp * (GEMV_DEPTH * GEMV_STAGE);
  const uint32_t ring_a = (uint32_t)__cvta_generic_to_shared(ring);
  // early: the weights are read before the previous kernel of the stream has finished (q8_gemv in a caller's scope, which
  // promises that nothing in it writes them); x and y wait for it.
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
  // The GEMM operators write nothing on top of an earlier failure (STATUS).  A thread of the last warp, which has the least of x
  // to fetch, reads the code for all.  One token 768 x 2176 without it 2.44 us, so 2.52; by thread 0 2.8, by every thread 3.0.
  const bool prior = STATUS && status && tid == (int)blockDim.x - 1 && __ldcg(status) != 0;
  if (X_IN_SMEM) {
#pragma unroll
    for (int v = 0; v < M; ++v)
      for (int i = tid; i < chunks * 4; i += blockDim.x) xs4[v * xchunks * 4 + xs4_index(i >> 2, i & 3)] = load_x4(x + v * k, i);
    if (!STATUS) {
      __syncthreads();
    } else if (__syncthreads_or(prior)) {
      asm volatile("cp.async.wait_all;" ::: "memory");
      return;
    }
  }
  int slot = 0;
  for (int64_t g = blockIdx.x + (int64_t)gridDim.x * warp; g < groups; g += step) {
    float acc[R][M];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int v = 0; v < M; ++v) acc[r][v] = 0.f;
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
          float p[R][M];
#pragma unroll
          for (int r = 0; r < R; ++r) {
            w[r] = *reinterpret_cast<const uint4*>(st + (r * U + u) * 512 + lane * 16);
#pragma unroll
            for (int v = 0; v < M; ++v) p[r][v] = 0.f;
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float4 f[R];
#pragma unroll
            for (int r = 0; r < R; ++r) f[r] = four_f32(j == 0 ? w[r].x : j == 1 ? w[r].y : j == 2 ? w[r].z : w[r].w);
#pragma unroll
            for (int v = 0; v < M; ++v) {
              const float4 xv = X_IN_SMEM ? xs4[v * xchunks * 4 + xs4_index(c, j)] : load_x4(x + v * k, (int64_t)c * 4 + j);
#pragma unroll
              for (int r = 0; r < R; ++r) p[r][v] = dot4(f[r], xv, p[r][v]);
            }
          }
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const float sc = *reinterpret_cast<const float*>(st + 2048 + (r * 16 * U + 16 * u + (lane >> 1)) * 4);
#pragma unroll
            for (int v = 0; v < M; ++v) acc[r][v] = fmaf(sc, p[r][v], acc[r][v]);
          }
        }
      }
    }
#pragma unroll
    for (int v = 0; v < M; ++v) {
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc[r][v] += __shfl_xor_sync(0xffffffffu, acc[r][v], o);
      if (lane != v) continue;
      if (R == 2 && epilogue == EPI_SWIGLU) {   // rows (2j, 2j + 1) are (gate_j, up_j)
        store_y(y, aux, EPI_NONE, v * (n / 2) + g, __fmul_rn(silu_f(acc[0][v]), acc[R - 1][v]));
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r)
          if (g * R + r < n) store_y(y, aux, epilogue, v * n + g * R + r, acc[r][v]);
      }
    }
  }
}


}  // namespace

namespace {

int64_t ring_bytes(int warps) { return (int64_t)warps * GEMV_DEPTH * GEMV_STAGE; }
int64_t x_bytes(int64_t m, int64_t k) { return m * ((k / 16 + 31) / 32 * 128) * (int64_t)sizeof(float4); }

template <int M, typename T, bool STATUS>
logos_status_t launch_m(const int8_t* q, const float* s, const T* x, T* y, int64_t n, int64_t k, bool early, const T* aux, int epilogue,
                        const int* status, int device, cudaStream_t st) {
  // two rows a warp unless that would leave more than half of the warps without any; the larger CTA where x fits
  // beside its rings (K up to 16384 for one vector), past K = 30208 x stays in global memory (one vector only)
  const int64_t sms = sm_count(device);
  const int rows = n <= sms * GEMV_WARPS && epilogue != EPI_SWIGLU ? 1 : 2;
  const int64_t groups = (n + rows - 1) / rows;
  const int64_t xb = x_bytes(M, k);
  const int warps = ring_bytes(GEMV_WARPS) + xb <= GEMV_SMEM ? GEMV_WARPS : GEMV_FEW_WARPS;
  const bool in_smem = ring_bytes(warps) + xb <= GEMV_SMEM;
  auto kern = rows == 2 ? q8_gemv_kernel<2, true, M, T, STATUS> : q8_gemv_kernel<1, true, M, T, STATUS>;
  if constexpr (!STATUS) {
    if (!in_smem) kern = rows == 2 ? q8_gemv_kernel<2, false, M, T, false> : q8_gemv_kernel<1, false, M, T, false>;
  }
  LOGOS_TRY(allow_smem(reinterpret_cast<const void*>(kern), device, GEMV_SMEM));
  LOGOS_CUDA_TRY(launch_kernel(kern, dim3((unsigned)std::min(groups, sms)), dim3(warps * 32), (size_t)(ring_bytes(warps) + (in_smem ? xb : 0)),
                               st, q, s, x, y, n, k, early, aux, epilogue, status));
  count_launch(LK_GEMV);
  return check_launch("q8_gemv_kernel");
}

// The GEMM operators' first kernel waits in a caller's scope too.
template <typename T>
logos_status_t launch_rows(const int8_t* q, const float* s, const T* x, T* y, int64_t m, int64_t n, int64_t k, const T* aux, int epilogue,
                           int device, cudaStream_t st) {
  // Without a word yet no kernel has given up; a capture, which cannot allocate one, goes on without.
  const int* status = kernel_status_ptr(device, false);
  if (!status && !stream_capturing(st)) {
    status = kernel_status_ptr(device);
    if (!status) return fail(LOGOS_ERROR, "q8_gemm: no kernel status word");
  }
  return m == 1 ? launch_m<1, T, true>(q, s, x, y, n, k, false, aux, epilogue, status, device, st)
                : launch_m<2, T, true>(q, s, x, y, n, k, false, aux, epilogue, status, device, st);
}

}  // namespace

logos_status_t launch_q8_gemv(const int8_t* q, const float* s, const float* x, float* y, int64_t n, int64_t k,
                              int device, cudaStream_t st) {
  if (n == 0) return LOGOS_OK;
  if (k == 0) {
    LOGOS_CUDA_TRY(cudaMemsetAsync(y, 0, sizeof(float) * n, st));
    return LOGOS_OK;
  }
  return launch_m<1, float, false>(q, s, x, y, n, k, pdl_early(), nullptr, EPI_NONE, nullptr, device, st);
}

bool gemv_takes(int64_t m, int64_t n, int64_t k) {
  if (m == 2 && n * k > (48ll << 20)) return false;
  return (m == 1 || m == 2) && n >= 1 && k >= 128 && k % 128 == 0 && ring_bytes(GEMV_FEW_WARPS) + x_bytes(m, k) <= GEMV_SMEM;
}

logos_status_t launch_q8_gemv_tokens(const GemmArgs& g, cudaStream_t st) {
  if (g.a_dtype == LOGOS_F32)
    return launch_rows(g.q, g.s, static_cast<const float*>(g.a), static_cast<float*>(g.c), g.m, g.n, g.k, static_cast<const float*>(nullptr),
                       EPI_NONE, g.device, st);
  return launch_rows(g.q, g.s, static_cast<const __nv_bfloat16*>(g.a), static_cast<__nv_bfloat16*>(g.c), g.m, g.n, g.k,
                     static_cast<const __nv_bfloat16*>(g.aux), g.epilogue, g.device, st);
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
