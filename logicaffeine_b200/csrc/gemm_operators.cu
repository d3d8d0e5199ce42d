// Entry points of the stand-alone Q8 products of several tokens: handles and extents checked, then the GEMV kernel for one
// or two tokens (q8_gemv.cu) or the GEMM (q8_gemm.cu).
#include "ops.cuh"

using namespace logos;

// Whether results go over the activations.  The GEMM has copied those into planes before it writes; of the GEMV kernel some
// CTAs read them while others write already.
static bool over_activations(const GemmArgs& g) {
  const int64_t bytes = g.a_dtype == LOGOS_F32 ? 4 : 2;   // of results too
  const char *a = static_cast<const char*>(g.a), *c = static_cast<const char*>(g.c);
  return c < a + g.m * g.lda * bytes && a < c + g.m * g.ldc * bytes;
}

static logos_status_t launch_product(const GemmArgs& g, cudaStream_t st) {
  if (!g.force_simt && gemv_takes(g.m, g.n, g.k) && !over_activations(g)) {
    OrderedScope ordered(st);
    return launch_q8_gemv_tokens(g, st);
  }
  return launch_gemm_operator(g, st);
}

static logos_status_t gemm_abi(logos_handle_t a, logos_handle_t q, logos_handle_t s, logos_handle_t c, int64_t m,
                               int64_t n, int64_t k, int32_t epilogue, logos_handle_t aux, void* stream,
                               int force_simt) {
  if (m < 0 || n < 0 || k < 0) return fail(LOGOS_OUT_OF_BOUNDS, "logos_q8_gemm: negative extent");
  if (k % 32) return fail(LOGOS_OUT_OF_BOUNDS, "logos_q8_gemm: K=%lld is not a multiple of the block size 32", (long long)k);
  if (epilogue < 0 || epilogue > 2) return fail(LOGOS_ERROR, "logos_q8_gemm: unknown epilogue %d", epilogue);
  if (epilogue == EPI_SWIGLU && (n & 1)) return fail(LOGOS_OUT_OF_BOUNDS, "logos_q8_gemm: swiglu epilogue needs even N");
  int64_t n_out = epilogue == EPI_SWIGLU ? n / 2 : n;
  __nv_bfloat16 *ap, *cp, *xp = nullptr;
  int8_t* qp;
  float* sp;
  int32_t dev = 0;
  LOGOS_TRY(buf_ptr<__nv_bfloat16>(a, m * k, "a", &ap, &dev));
  LOGOS_TRY(buf_ptr<int8_t>(q, n * k, "q", &qp));
  LOGOS_TRY(buf_ptr<float>(s, n * (k / 32), "s", &sp));
  LOGOS_TRY(buf_ptr<__nv_bfloat16>(c, m * n_out, "c", &cp));
  if (epilogue == EPI_RESIDUAL) {
    if (!aux) return fail(LOGOS_NULL_POINTER, "logos_q8_gemm: residual epilogue needs aux");
    LOGOS_TRY(buf_ptr<__nv_bfloat16>(aux, m * n, "aux", &xp));
  }
  LOGOS_CUDA_TRY(cudaSetDevice(dev));
  GemmArgs g;
  g.a = ap; g.a_dtype = LOGOS_BF16; g.lda = k;
  g.q = qp; g.s = sp;
  g.c = cp; g.c_dtype = LOGOS_BF16; g.ldc = n_out;
  g.aux = xp;
  g.m = m; g.n = n; g.k = k;
  g.epilogue = epilogue;
  g.device = dev;
  g.force_simt = force_simt;
  return launch_product(g, as_stream(stream));
}

extern "C" {

// f32 activations, f32 output: the form the decode step uses internally (the
// activations are split into two fp16 planes so the tensor-core product keeps
// f32-class accuracy).
logos_status_t logos_q8_gemm_f32(logos_handle_t a, logos_handle_t q, logos_handle_t s, logos_handle_t c, int64_t m,
                                 int64_t n, int64_t k, void* stream_or_null) {
  return guarded([&]() -> logos_status_t {
    if (m < 0 || n < 0 || k < 0) return fail(LOGOS_OUT_OF_BOUNDS, "logos_q8_gemm_f32: negative extent");
    if (k % 32) return fail(LOGOS_OUT_OF_BOUNDS, "logos_q8_gemm_f32: K=%lld is not a multiple of the block size 32", (long long)k);
    float *ap, *sp, *cp;
    int8_t* qp;
    int32_t dev = 0;
    LOGOS_TRY(buf_ptr<float>(a, m * k, "a", &ap, &dev));
    LOGOS_TRY(buf_ptr<int8_t>(q, n * k, "q", &qp));
    LOGOS_TRY(buf_ptr<float>(s, n * (k / 32), "s", &sp));
    LOGOS_TRY(buf_ptr<float>(c, m * n, "c", &cp));
    LOGOS_CUDA_TRY(cudaSetDevice(dev));
    GemmArgs g;
    g.a = ap; g.a_dtype = LOGOS_F32; g.lda = k;
    g.q = qp; g.s = sp;
    g.c = cp; g.c_dtype = LOGOS_F32; g.ldc = n;
    g.m = m; g.n = n; g.k = k;
    g.device = dev;
    return launch_product(g, as_stream(stream_or_null));
  });
}

logos_status_t logos_q8_gemm(logos_handle_t a, logos_handle_t q, logos_handle_t s, logos_handle_t c, int64_t m,
                             int64_t n, int64_t k, int32_t epilogue, logos_handle_t aux_or_null,
                             void* stream_or_null) {
  return guarded([&]() -> logos_status_t {
    return gemm_abi(a, q, s, c, m, n, k, epilogue, aux_or_null, stream_or_null, 0);
  });
}

// Same contract as logos_q8_gemm, always on the SIMT kernel: the on-device
// cross-check for the tensor-core path.
logos_status_t logos_q8_gemm_simt(logos_handle_t a, logos_handle_t q, logos_handle_t s, logos_handle_t c, int64_t m,
                                  int64_t n, int64_t k, int32_t epilogue, logos_handle_t aux_or_null,
                                  void* stream_or_null) {
  return guarded([&]() -> logos_status_t {
    return gemm_abi(a, q, s, c, m, n, k, epilogue, aux_or_null, stream_or_null, 1);
  });
}

}  // extern "C"
