// What kernels do behind a failure: with a code in the status word, as a wait that gave up leaves it, a launch writes nothing,
// and once the code is cleared the same launch writes its results.  Prints a line "<what> <changed behind the code> <changed after>" for each.
#include "ops.cuh"
#include "ptx.cuh"

#include <cstdio>
#include <cstring>
#include <functional>
#include <vector>

using namespace logos;

#define CHECK(x)                                                       \
  do {                                                                 \
    if (int e_ = (int)(x)) {                                           \
      printf("%s: %d %s\n", #x, e_, last_error_text() ? last_error_text() : ""); \
      return 2;                                                        \
    }                                                                  \
  } while (0)

struct Buf {
  void* p = nullptr;
  size_t bytes = 0;
};
static Buf buf(size_t bytes, int dtype, int kind, int stream, float a, float b) {
  Buf r;
  r.bytes = bytes;
  if (cudaMalloc(&r.p, bytes) != cudaSuccess) return r;
  const int64_t size = dtype == LOGOS_F16 || dtype == LOGOS_BF16 ? 2 : dtype == LOGOS_I8 ? 1 : 4;
  launch_synth_fill(r.p, dtype, kind, 1, stream, 0, (int64_t)bytes / size, a, b, 0, nullptr);
  return r;
}

static int run(const char* what, const std::vector<Buf>& written, const std::function<logos_status_t()>& launch) {
  auto bytes = [&] {
    std::vector<std::vector<char>> v;
    for (const Buf& w : written) {
      v.emplace_back(w.bytes);
      cudaMemcpy(v.back().data(), w.p, w.bytes, cudaMemcpyDeviceToHost);
    }
    return v;
  };
  int* word = kernel_status_ptr(0);
  const int code = 4242;
  const auto before = bytes();
  CHECK(cudaMemcpy(word, &code, sizeof(code), cudaMemcpyHostToDevice));
  CHECK(launch());
  CHECK(cudaDeviceSynchronize());
  const auto behind = bytes();
  int got = 0;
  CHECK(kernel_status_read(0, &got, true));
  if (got != code) return 3;
  CHECK(launch());
  CHECK(cudaDeviceSynchronize());
  const auto after = bytes();
  CHECK(kernel_status_read(0, &got, true));
  if (got != 0) return 4;
  bool all = true;
  for (size_t i = 0; i < after.size(); ++i) all = all && after[i] != before[i];
  printf("%s %d %d\n", what, (int)(behind != before), (int)all);
  return 0;
}

static int attention(int d, int b) {
  const int h_q = 14, h_kv = 2, l_max = 700;
  const int64_t cache = (int64_t)b * h_kv * l_max * d;
  AttnArgs a;
  Buf q = buf(b * h_q * d * 2, LOGOS_F16, 2, 1, 0.f, 1.f), kn = buf(b * h_kv * d * 2, LOGOS_F16, 2, 2, 0.f, 1.f);
  Buf k = buf(cache * 2, LOGOS_F16, 2, 3, 0.f, 1.f), v = buf(cache * 2, LOGOS_F16, 2, 4, 0.f, 1.f);
  Buf rope = buf((size_t)l_max * d * 4, LOGOS_F32, 2, 5, 0.f, 1.f), o = buf(b * h_q * d * 2, LOGOS_F16, 2, 6, 0.f, 1.f);
  Buf seq = buf(b * 4, LOGOS_F32, 2, 7, 0.f, 1.f);
  std::vector<int> lens(b);
  for (int i = 0; i < b; ++i) lens[i] = i * 600 / b;   // an empty sequence among them
  CHECK(cudaMemcpy(seq.p, lens.data(), seq.bytes, cudaMemcpyHostToDevice));
  a.q_f16 = (const __half*)q.p; a.k_new_f16 = a.v_new_f16 = (const __half*)kn.p;
  a.k_cache = (__half*)k.p; a.v_cache = (__half*)v.p; a.rope = (const float*)rope.p; a.rotate_q = 1;
  a.seq_len = (int32_t*)seq.p; a.bump_seq_len = 1; a.o = o.p;
  a.b = b; a.h_q = h_q; a.h_kv = h_kv; a.d = d; a.l_max = l_max; a.scale = 0.1f;
  return run("attention", {o, k, v, seq}, [&] { return launch_gqa_decode_attn(a, nullptr); });
}

static int narrow(int out, int m, int n, int k) {
  NarrowArgs a;
  Buf q = buf((size_t)(n + 127) / 128 * 128 * k, LOGOS_I8, 0, 1, 0.f, 0.f), s = buf((size_t)(n + 127) / 128 * 128 * (k / 32) * 4, LOGOS_F32, 1, 2, 1e-3f, 1e-2f);
  Buf h = buf((size_t)m * k * 4, LOGOS_F32, 2, 3, 0.f, 1.f), gain = buf(k * 4, LOGOS_F32, 1, 4, 1.f, 1.f);
  Buf hi = buf((size_t)m * k * 2, LOGOS_F16, 2, 5, 0.f, 1.f), c = buf((size_t)m * n * 4, LOGOS_F32, 2, 6, 0.f, 1.f);
  Buf phi = buf((size_t)m * n, LOGOS_F16, 2, 7, 0.f, 1.f), plo = buf((size_t)m * n, LOGOS_F16, 2, 8, 0.f, 1.f);
  a.q = (const int8_t*)q.p; a.s = (const float*)s.p; a.m = m; a.n = n; a.k = k;
  a.h_in = (const float*)h.p; a.gain = (const float*)gain.p; a.eps = 1e-6f;
  a.a.hi = a.a.lo = (__half*)hi.p;
  a.out = out; a.c = (float*)c.p; a.planes.hi = (__half*)phi.p; a.planes.lo = (__half*)plo.p;
  if (!narrow_applicable(m, n, k, out != NARROW_RESIDUAL, 0)) return 5;
  return run(out == NARROW_F32 ? "norm" : out == NARROW_SWIGLU ? "norm+swiglu" : "residual",
             out == NARROW_SWIGLU ? std::vector<Buf>{phi, plo} : std::vector<Buf>{c}, [&] { return launch_q8_narrow(a, nullptr); });
}

// A stand-alone product, results in place of the residual where there is one; `form` is what its plan makes of it.
static int product(const char* form, int m, int n, int k, int dtype, int epilogue) {
  const int size = dtype == LOGOS_F32 ? 4 : 2;
  GemmArgs g;
  Buf a = buf((size_t)m * k * size, dtype, 2, 1, 0.f, 1.f), q = buf((size_t)n * k, LOGOS_I8, 0, 2, 0.f, 0.f);
  Buf s = buf((size_t)n * (k / 32) * 4, LOGOS_F32, 1, 3, 1e-3f, 1e-2f), c = buf((size_t)m * n * size, dtype, 2, 4, 0.f, 1.f);
  if (!c.p) return 6;
  g.a = a.p; g.a_dtype = dtype; g.lda = k;
  g.q = (const int8_t*)q.p; g.s = (const float*)s.p;
  g.c = c.p; g.c_dtype = dtype; g.ldc = epilogue == EPI_SWIGLU ? n / 2 : n;
  if (epilogue == EPI_RESIDUAL) g.aux = c.p;
  g.m = m; g.n = n; g.k = k; g.epilogue = epilogue;
  if (int rc = run(form, {c}, [&] { return gemv_takes(m, n, k) ? launch_q8_gemv_tokens(g, nullptr) : launch_gemm_operator(g, nullptr); })) return rc;
  for (const Buf& b : {a, q, s, c}) cudaFree(b.p);
  return 0;
}

int main() {
  if (!kernel_status_ptr(0)) return 1;
  for (int epilogue : {EPI_NONE, EPI_RESIDUAL, EPI_SWIGLU})
    for (int dtype : {LOGOS_F32, LOGOS_BF16}) {
      if (dtype == LOGOS_F32 && epilogue != EPI_NONE) continue;   // (f32 products have no epilogue)
      for (int m : {1, 2})
        if (int rc = product("gemv", m, 1024, 1024, dtype, epilogue)) return rc;
      if (int rc = product("gemm", 40, 37888, 256, dtype, epilogue)) return rc;    // pairs of row tiles
      if (int rc = product("gemm", 384, 18944, 256, dtype, epilogue)) return rc;   // wide units, or a staged residual
      if (int rc = product("gemm", 300, 512, 4096, dtype, epilogue)) return rc;    // K splits
      // K that is no multiple of 128: the kernels behind the product may compute it again
      if (int rc = product("gemm", 5, 512, 160, dtype, epilogue)) return rc;
      if (int rc = product("gemm", 40, 512, 2080, dtype, epilogue)) return rc;
    }
  for (int m : {1, 8, 16})
    for (int out : {NARROW_F32, NARROW_SWIGLU, NARROW_RESIDUAL})
      for (int k : {896, 4864}) {
        if (out != NARROW_RESIDUAL && k > 1024) continue;
        if (int rc = narrow(out, m, 896, k)) return rc;
      }
  for (int d : {64, 128})
    for (int b : {1, 5, 200})   // clusters of up to eight CTAs, and of one
      if (int rc = attention(d, b)) return rc;
  return 0;
}
