// Q8 GEMM front: C[m,n] = sum_kb s[n,kb] * sum_k A[m,k] * q[n,k].
//
// Dispatch between two kernels:
//   * q8_gemm_tc.cu — the tcgen05 / TMA kernel: K of at least 128, 16-byte aligned operands, and K a
//     multiple of 128 or scales in the tile-major form (the stand-alone operators bring them there);
//   * the SIMT kernel below — anything else, and the on-device cross-check
//     the tests hold the tensor-core kernel against.
// Plus the split-K reduction + epilogue kernel shared by both.
#include "ops.cuh"
#include "q8_gemm_tc.cuh"

#include <algorithm>
#include <atomic>

namespace logos {

namespace {

__device__ __forceinline__ float load_act(const void* a, int dtype, int64_t i, const __half* lo = nullptr) {
  if (dtype == LOGOS_F16) return act_load(reinterpret_cast<const __half*>(a), lo, i);
  if (dtype == LOGOS_BF16) return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(a)[i]);
  return reinterpret_cast<const float*>(a)[i];
}
__device__ __forceinline__ void store_out(void* c, int dtype, int64_t i, float v, const ActOut& planes) {
  if (dtype == LOGOS_ACT_PLANES) act_store(planes, i, v);
  else if (dtype == LOGOS_F16) reinterpret_cast<__half*>(c)[i] = __float2half_rn(v);
  else if (dtype == LOGOS_BF16) reinterpret_cast<__nv_bfloat16*>(c)[i] = __float2bfloat16_rn(v);
  else reinterpret_cast<float*>(c)[i] = v;
}

constexpr int SIMT_TN = 32;  // weight rows per CTA
constexpr int SIMT_TM = 32;  // tokens per CTA

struct SimtArgs {
  const void* a;
  const __half* a_lo;
  int a_dtype;
  int64_t lda;
  const int8_t* q;
  const float* s;
  void* c;
  int c_dtype;
  ActOut c_act;
  int64_t ldc;
  const void* aux;
  float* partials;
  int64_t m, n, k;
  int epilogue, splits;
};
// One tile of the product by 256 threads: lane = weight row inside the tile, warp w owns tokens 4w..4w+3.
__device__ __forceinline__ void simt_tile(const SimtArgs& g, int64_t tile_n, int64_t tile_m, int split, float (&as)[SIMT_TM][33],
                                          float (&qs)[SIMT_TN][33]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t m = g.m, n = g.n, k = g.k, lda = g.lda, ldc = g.ldc;
  const int splits = g.splits;
  const int64_t n0 = tile_n * SIMT_TN, m0 = tile_m * SIMT_TM;
  const int64_t kb_total = k / 32;
  const int64_t kb_per = (kb_total + splits - 1) / splits;
  const int64_t kb_begin = split * kb_per;
  const int64_t kb_end = kb_begin + kb_per < kb_total ? kb_begin + kb_per : kb_total;
  const int64_t row = n0 + lane;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  for (int64_t kb = kb_begin; kb < kb_end; ++kb) {
    for (int i = threadIdx.x; i < SIMT_TM * 32; i += 256) {
      int r = i >> 5, cidx = i & 31;
      as[r][cidx] = (m0 + r < m) ? load_act(g.a, g.a_dtype, (m0 + r) * lda + kb * 32 + cidx, g.a_lo) : 0.f;
      qs[r][cidx] = (n0 + r < n) ? (float)g.q[(n0 + r) * k + kb * 32 + cidx] : 0.f;
    }
    __syncthreads();
    float p[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int kk = 0; kk < 32; ++kk) {
      float qv = qs[lane][kk];
#pragma unroll
      for (int j = 0; j < 4; ++j) p[j] = fmaf(as[warp * 4 + j][kk], qv, p[j]);
    }
    float sc = (row < n) ? g.s[row * kb_total + kb] : 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[j] = fmaf(sc, p[j], acc[j]);
    __syncthreads();
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    int64_t mm = m0 + warp * 4 + j;
    float v = acc[j];
    if (splits > 1) {
      if (mm < m && row < n) g.partials[((int64_t)split * m + mm) * n + row] = v;
      continue;
    }
    if (g.epilogue == EPI_SWIGLU) {
      float other = __shfl_xor_sync(0xffffffffu, v, 1);
      if (!(lane & 1) && mm < m && row + 1 < n) store_out(g.c, g.c_dtype, mm * ldc + (row >> 1), __fmul_rn(silu_f(v), other), g.c_act);
    } else if (mm < m && row < n) {
      if (g.epilogue == EPI_RESIDUAL) v = __fadd_rn(v, load_act(g.aux, g.c_dtype, mm * ldc + row));
      store_out(g.c, g.c_dtype, mm * ldc + row, v, g.c_act);
    }
  }
}

__global__ void __launch_bounds__(256) q8_gemm_simt_kernel(const SimtArgs g) {
  __shared__ float as[SIMT_TM][33];
  __shared__ float qs[SIMT_TN][33];
  simt_tile(g, blockIdx.x, blockIdx.y, blockIdx.z, as, qs);
}

// What the fp16 planes of a call do not hold (see launch_gemm_prep): the preparation stored `call` to *word then, and the
// kernel that comes last computes the product again, epilogue included, instead of what it is for.
struct Misfit {
  const unsigned* word = nullptr;   // null: nothing to look at
  unsigned call = 0;
  SimtArgs product = {};
  int64_t tiles_n = 0, tiles_m = 0;
};
// The whole grid's part.
__device__ __forceinline__ void redo_misfit(const Misfit& f) {
  __shared__ float as[SIMT_TM][33];
  __shared__ float qs[SIMT_TN][33];
  for (int64_t t = blockIdx.x; t < f.tiles_n * f.tiles_m; t += gridDim.x)
    simt_tile(f.product, t % f.tiles_n, t / f.tiles_n, 0, as, qs);
}
// The whole grid's part, unless there is the code of an earlier failure (one thread of a CTA reads it, all take one decision).
__device__ __forceinline__ void redo_unless_failed(const Misfit& f, const int* status) {
  if (!__syncthreads_or(threadIdx.x == 0 && __ldcg(status) != 0)) redo_misfit(f);
}
// Where no other kernel follows the product.
__global__ void __launch_bounds__(256) q8_gemm_misfit_kernel(const Misfit f, const int* status) {
  pdl_wait();
  pdl_trigger();
  if (__ldcg(f.word) == f.call) redo_unless_failed(f, status);
}

// Behind an earlier failure an operator's product does nothing, and its preparation has put NaN where its sums would be: only where
// a result is NaN is the status word looked at.  Read by every CTA, that one sector cost products of few rows and many
// tokens 2 to 10 %; NaN from the product's own kernel a prompt up to 1.7 %, by what the code for it did to the rest.
__device__ __forceinline__ bool unless_failed(float v, const int* status) { return v == v || __ldcg(status) == 0; }

// Sum split-K partials in ascending split order, then apply the epilogue.  The misfit word is loaded beside the
// partials and looked at after them.
template <bool MISFIT>
__global__ void splitk_reduce_kernel(const float* __restrict__ partials, int splits, void* __restrict__ c, int c_dtype,
                                     ActOut c_act, int64_t ldc, const void* __restrict__ aux, int64_t m, int64_t n,
                                     int epilogue, const Misfit f, const int* status) {
  pdl_wait();  // the partials are the previous kernel's output: wait for it, read them past L1
  pdl_trigger();
  const unsigned word = MISFIT ? __ldcg(f.word) : 0u;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool swiglu = epilogue == EPI_SWIGLU;
  const int64_t width = swiglu ? n / 2 : n;
  const bool inside = i < m * width;
  const int64_t mm = inside ? i / width : 0, j = inside ? i - mm * width : 0, at = mm * ldc + j;
  float v = 0.f;
  if (inside) {
    if (swiglu) {
      float g = 0.f, u = 0.f;
      for (int sp = 0; sp < splits; ++sp) {
        const float2 gu = __ldcg(reinterpret_cast<const float2*>(partials + ((int64_t)sp * m + mm) * n + 2 * j));
        g = __fadd_rn(g, gu.x);
        u = __fadd_rn(u, gu.y);
      }
      v = __fmul_rn(silu_f(g), u);
    } else {
      for (int sp = 0; sp < splits; ++sp) v = __fadd_rn(v, __ldcg(partials + ((int64_t)sp * m + mm) * n + j));
      if (epilogue == EPI_RESIDUAL) v = __fadd_rn(v, load_act(aux, c_dtype, at));
    }
  }
  if (MISFIT && word == f.call) redo_unless_failed(f, status);
  else if (inside && unless_failed(v, status)) store_out(c, c_dtype, at, v, c_act);
}

// c = staged sums + residual, bf16; HBM-bound, eight elements a thread.
template <bool MISFIT>
__global__ void __launch_bounds__(256) residual_kernel(const float* __restrict__ sums, const __nv_bfloat16* aux, __nv_bfloat16* c, int64_t count,
                                                       const Misfit f, const int* status) {
  pdl_wait();
  pdl_trigger();
  if (MISFIT && __ldcg(f.word) == f.call) {
    redo_unless_failed(f, status);
    return;
  }
  const int64_t i = ((int64_t)blockIdx.x * 256 + threadIdx.x) * 8;
  const bool vec = i + 8 <= count && !((reinterpret_cast<uintptr_t>(aux) | reinterpret_cast<uintptr_t>(c)) & 15u);
  if (vec) {
    const float4 a = __ldcg(reinterpret_cast<const float4*>(sums + i)), b = __ldcg(reinterpret_cast<const float4*>(sums + i) + 1);
    const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    const uint4 r = *reinterpret_cast<const uint4*>(aux + i);
    const __nv_bfloat16* rh = reinterpret_cast<const __nv_bfloat16*>(&r);
    uint4 o;
    __nv_bfloat16* oh = reinterpret_cast<__nv_bfloat16*>(&o);
#pragma unroll
    for (int j = 0; j < 8; ++j) oh[j] = unless_failed(v[j], status) ? __float2bfloat16_rn(__fadd_rn(v[j], __bfloat162float(rh[j]))) : c[i + j];
    *reinterpret_cast<uint4*>(c + i) = o;
  } else {
    for (int64_t j = i; j < count && j < i + 8; ++j) {
      const float v = __ldcg(sums + j);
      if (unless_failed(v, status)) c[j] = __float2bfloat16_rn(__fadd_rn(v, __bfloat162float(aux[j])));
    }
  }
}

}  // namespace

// K splits: a unit's time is a fixed part (pipeline fill, epilogue: about twelve stage times, measured) plus its K
// stages, and units run in rounds of one per SM.  The split count with the smallest rounds x (fixed + stages);
// ties go to fewer splits (fewer partials to write and fold).  A row tile for each token tile of 64 is a
// unit of its own: with many tokens there are enough.  The split count is also what fixes the order of a
// sum, so that the same shape gives the same bits whatever the kernel's tiles.
// Where the consumer folds the partials as it reads them (`folded`: a decode step's norms and attention) a split costs no
// launch: as few as three stages then, and the fixed part overlaps the predecessor's end, eight stage times.  With the
// other rule / this one, us a step: 0.5B shape at batch 17 844 / 789, 64 1062 / 986; four layers of the 32B shape at batch 1
// 731 / 695, 64 1182 / 1151.
int gemm_pick_splits(int64_t m, int64_t n, int64_t k, int device, bool folded) {
  const int64_t tiles = ((n + 127) / 128) * std::max<int64_t>((m + 63) / 64, 1);
  const int64_t stages = k / 128;
  const int sms = sm_count(device);
  const int64_t least = folded ? 3 : 4;   // stages a split
  if (tiles >= sms || stages < 2 * least) return 1;
  const int64_t fixed = folded ? 8 : 12;
  const int64_t max_splits = std::min<int64_t>(stages / least, 16);
  int best = 1;
  int64_t best_cost = INT64_MAX;
  for (int64_t sp = 1; sp <= max_splits; ++sp) {
    const int64_t rounds = (tiles * sp + sms - 1) / sms;
    const int64_t per = (stages + sp - 1) / sp;
    const int64_t cost = rounds * (fixed + per) * 8 + sp;
    if (cost < best_cost) { best_cost = cost; best = (int)sp; }
  }
  return best;
}

static logos_status_t launch_reduce(const float* partials, int splits, void* c, int c_dtype, ActOut c_act, int64_t ldc,
                                    const void* aux, int64_t m, int64_t n, int epilogue, const Misfit& f, const int* status, cudaStream_t st) {
  int64_t total = (epilogue == EPI_SWIGLU) ? m * (n / 2) : m * n;
  if (total == 0) return LOGOS_OK;
  LOGOS_CUDA_TRY(launch_kernel(f.word ? splitk_reduce_kernel<true> : splitk_reduce_kernel<false>, dim3((unsigned)((total + 255) / 256)),
                               dim3(256), 0, st, partials, splits, c, c_dtype, c_act, ldc, aux, m, n, epilogue, f, status));
  count_launch(LK_ELEMWISE);
  return check_launch("splitk_reduce_kernel");
}

logos_status_t launch_splitk_reduce(const float* partials, int splits, void* c, int c_dtype, ActOut c_act,
                                    int64_t ldc, const void* aux, int64_t m, int64_t n, int epilogue, int device,
                                    cudaStream_t st) {
  const int* status = kernel_status_ptr(device);
  if (!status) return fail(LOGOS_ERROR, "q8_gemm: no kernel status word");
  return launch_reduce(partials, splits, c, c_dtype, c_act, ldc, aux, m, n, epilogue, Misfit(), status, st);
}

static SimtArgs simt_args(const GemmArgs& g) {
  return {g.a, g.a_lo, g.a_dtype, g.lda, g.q, g.s, g.c, g.c_dtype, g.c_act, g.ldc, g.aux, g.partials, g.m, g.n, g.k, g.epilogue, g.splits > 1 ? g.splits : 1};
}

logos_status_t launch_q8_gemm(const GemmArgs& g, cudaStream_t st) {
  if (g.m == 0 || g.n == 0) return LOGOS_OK;
  if (g.k % 32) return fail(LOGOS_OUT_OF_BOUNDS, "q8_gemm: K=%lld is not a multiple of the block size 32", (long long)g.k);
  if (g.epilogue == EPI_SWIGLU && (g.n & 1)) return fail(LOGOS_OUT_OF_BOUNDS, "q8_gemm: swiglu epilogue needs even N");
  if (g.splits > 1 && (!g.partials || g.epilogue != EPI_NONE))
    return fail(LOGOS_ERROR, "q8_gemm: split-K writes raw partials; the caller reduces them");
  if (!g.force_simt && gemm_tc_applicable(g)) return launch_q8_gemm_tc(g, st);
  if (g.q_tiled) return fail(LOGOS_ERROR, "q8_gemm: tile-major weights need the tensor-core kernel, which does not take this call");
  const SimtArgs args = simt_args(g);
  dim3 grid((unsigned)((g.n + SIMT_TN - 1) / SIMT_TN), (unsigned)((g.m + SIMT_TM - 1) / SIMT_TM), (unsigned)args.splits);
  q8_gemm_simt_kernel<<<grid, 256, 0, st>>>(args);
  count_launch(LK_GEMM_SIMT);
  return check_launch("q8_gemm_simt_kernel");
}

}  // namespace logos

using namespace logos;

// The stand-alone operators' way to the tensor-core kernel: activations into fp16 planes (and, where K is not
// a multiple of 128, scales into the tile-major form) by one small kernel, then the product, then the
// fold of the K splits.  The launches are dependent ones: each kernel sets up, and the product fetches its first
// weights, while the one before it finishes.  Nothing here writes weights, and the first kernel lets the product start
// only once what ran before in the stream has ended.
constexpr int64_t STAGED_BYTES = 64ll << 20;   // sums staged at a time, see below: half of L2

static logos_status_t gemm_tensor(GemmArgs g, bool two_planes, cudaStream_t st) {
  const void* src = g.a;
  const int src_dtype = g.a_dtype;
  const int64_t stages = (g.k + 127) / 128;
  const bool retile = g.k % 128 != 0;
  int splits = g.m > 64 ? gemm_many_splits(g.m, g.n, g.k, g.device, false) : gemm_pick_splits(g.m, g.n, g.k, g.device, false);
  auto up = [](int64_t v) { return (v + 255) / 256 * 256; };
  const int64_t lda = stages * 128;
  const int64_t plane_bytes = up(g.m * lda * 2);
  const int64_t scale_bytes = retile ? up((g.n + 127) / 128 * stages * 2048) : 0;
  const int64_t own_bytes = (two_planes ? 2 : 1) * plane_bytes + scale_bytes + (retile ? 256 : 0);
  void* scratch = nullptr;
  // many tokens are worth splitting where there is room for the partial sums
  if (g.m > 64 && splits > 1 && !scratch_try(g.device, 0, own_bytes + splits * g.m * g.n * (int64_t)sizeof(float), st, &scratch)) splits = 1;
  // The product kernel loads a residual row after row, which an SM with several tiles to do waits for every time: with
  // more than 96 tokens, the largest tile of pairs of row tiles, the sums are staged in f32 and a kernel of its own adds the
  // residual, the same bits.  A few such tiles at a time, so that the scratch stays small and the sums in L2.  (Units of
  // 128 or 192 tokens would have the line and the multiple elsewhere; not timed.)
  // Where the product may be done again (below) the residual always is: it must not have been added, `aux` can be `c`.
  int64_t stage_rows = STAGED_BYTES / (g.n * (int64_t)sizeof(float));
  stage_rows = stage_rows >= 96 ? stage_rows / 96 * 96 : retile ? std::max<int64_t>(stage_rows, 1) : 0;
  bool staged = g.epilogue == EPI_RESIDUAL && splits <= 1 && (retile || g.m > 96) && stage_rows > 0;
  const int64_t part_rows = staged ? std::min(g.m, stage_rows) : splits > 1 ? splits * g.m : 0;
  const int64_t part_bytes = part_rows * g.n * (int64_t)sizeof(float);
  if (retile || staged) {
    // neither form is worth failing for: the CUDA-core kernel needs no scratch, and the residual can be added
    // in the product
    if (!scratch_try(g.device, 0, own_bytes + part_bytes, st, &scratch)) {
      if (retile) {
        g.force_simt = 1;
        return launch_q8_gemm(g, st);
      }
      staged = false;
      LOGOS_TRY(scratch_get(g.device, 0, own_bytes, &scratch));
    }
  } else {
    LOGOS_TRY(scratch_get(g.device, 0, own_bytes + part_bytes, &scratch));
  }
  char* at = static_cast<char*>(scratch);
  ActOut planes;
  planes.hi = reinterpret_cast<__half*>(at);
  planes.lo = two_planes ? reinterpret_cast<__half*>(at + plane_bytes) : nullptr;
  planes.mode = two_planes ? LOGOS_F32 : LOGOS_F16;
  at += (two_planes ? 2 : 1) * plane_bytes;
  float* tiled = retile ? reinterpret_cast<float*>(at) : nullptr;
  at += scale_bytes;
  // K that is no multiple of 128 was the CUDA-core kernel's alone, in f32 throughout.  What the planes do not hold is
  // still its, in the call's last kernel: the preparation marks the call by its number (nothing to clear: the word holds
  // another call's otherwise, and a replayed capture that finds its own mark does no more than the product
  // again).  A kernel of its own after every product cost 2 us of 14; the folds load the word beside the partials.
  static std::atomic<unsigned> calls{0};
  unsigned* const misfit = retile ? reinterpret_cast<unsigned*>(at) : nullptr;
  const unsigned call = retile ? ++calls : 0;
  if (retile) at += 256;
  // rows m0 .. m0 + m of the call as the CUDA-core kernel takes them
  auto again = [&, plain = g](int64_t m0, int64_t m) {
    Misfit f;
    if (!retile) return f;
    GemmArgs e = plain;
    e.a = static_cast<const char*>(e.a) + m0 * e.lda * (src_dtype == LOGOS_BF16 ? 2 : 4);
    e.c = static_cast<char*>(e.c) + m0 * e.ldc * (e.c_dtype == LOGOS_BF16 ? 2 : 4);
    if (e.aux) e.aux = static_cast<const __nv_bfloat16*>(e.aux) + m0 * e.ldc;
    e.m = m;
    f.word = misfit;
    f.call = call;
    f.product = simt_args(e);
    f.tiles_n = (e.n + SIMT_TN - 1) / SIMT_TN;
    f.tiles_m = (e.m + SIMT_TM - 1) / SIMT_TM;
    return f;
  };
  const int* status = kernel_status_ptr(g.device);
  if (!status) return fail(LOGOS_ERROR, "q8_gemm: no kernel status word");
  {
    OrderedScope ordered(st);
    LOGOS_TRY(launch_gemm_prep(src, src_dtype, planes, g.m, g.s, tiled, g.n, g.k, misfit, call,
                               part_rows > 0 ? reinterpret_cast<float*>(at) : nullptr, part_rows * g.n, status, st));
  }
  g.lda = lda;
  g.a = planes.hi;
  g.a_lo = planes.lo;
  g.a_dtype = LOGOS_F16;
  if (retile) {
    g.s = tiled;
    g.s_tiled = 1;
  }
  PdlScope pdl(pdl_active() || pdl_enabled());
  if (splits <= 1 && !staged) {
    LOGOS_TRY(launch_q8_gemm(g, st));
    if (!retile) return LOGOS_OK;
    const Misfit f = again(0, g.m);
    const int64_t grid = std::min<int64_t>(f.tiles_n * f.tiles_m, 4ll * sm_count(g.device));
    LOGOS_CUDA_TRY(launch_kernel(q8_gemm_misfit_kernel, dim3((unsigned)grid), dim3(256), 0, st, f, status));
    count_launch(LK_GEMM_SIMT);
    return check_launch("q8_gemm_misfit_kernel");
  }
  GemmArgs gp = g;
  if (staged) {
    gp.c_dtype = LOGOS_F32;
    gp.epilogue = EPI_NONE;
    gp.aux = nullptr;
    gp.c = at;
    for (int64_t m0 = 0; m0 < g.m; m0 += stage_rows) {
      gp.m = std::min(stage_rows, g.m - m0);
      gp.a = planes.hi + m0 * lda;
      gp.a_lo = two_planes ? planes.lo + m0 * lda : nullptr;
      LOGOS_TRY(launch_q8_gemm(gp, st));
      const int64_t count = gp.m * g.n;
      const Misfit f = again(m0, gp.m);
      LOGOS_CUDA_TRY(launch_kernel(f.word ? residual_kernel<true> : residual_kernel<false>, dim3((unsigned)((count + 2047) / 2048)), dim3(256), 0, st,
                                   reinterpret_cast<const float*>(at), reinterpret_cast<const __nv_bfloat16*>(g.aux) + m0 * g.n,
                                   reinterpret_cast<__nv_bfloat16*>(g.c) + m0 * g.n, count, f, status));
      count_launch(LK_ELEMWISE);
      LOGOS_TRY(check_launch("residual_kernel"));
    }
    return LOGOS_OK;
  }
  gp.splits = splits;
  gp.partials = reinterpret_cast<float*>(at);
  gp.epilogue = EPI_NONE;
  gp.c = nullptr;
  gp.c_dtype = LOGOS_F32;
  gp.aux = nullptr;
  LOGOS_TRY(launch_q8_gemm(gp, st));
  return launch_reduce(gp.partials, splits, g.c, g.c_dtype, ActOut(), g.ldc, g.aux, g.m, g.n, g.epilogue, again(0, g.m), status, st);
}

// Whether the operands of a stand-alone call can go to the tensor-core kernel once prepared (the planes and, where
// needed, the scales are scratch of the library's own then).
static bool gemm_tensor_takes(GemmArgs g) {
  g.a_dtype = LOGOS_F16;
  g.a = g.a_lo = nullptr;
  g.lda = (g.k + 127) / 128 * 128;
  g.s_tiled = g.k % 128 != 0;
  return gemm_tc_applicable(g);
}

// A stand-alone product, by the tensor-core kernel where that takes it.
logos_status_t logos::launch_gemm_operator(const GemmArgs& g, cudaStream_t st) {
  if (g.force_simt || !gemm_tensor_takes(g)) return launch_q8_gemm(g, st);
  // A bf16 value is exactly representable in fp16 inside fp16's normal range, so one plane is enough.
  return gemm_tensor(g, g.a_dtype == LOGOS_F32, st);
}
