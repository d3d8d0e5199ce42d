// Products of csrc/q8_narrow.cu against what must come out bit for bit: a line "<what> <tokens> <columns> <differing>" for each.
#include "ops.cuh"

#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

using namespace logos;

#define CHECK(x)                                                       \
  do {                                                                 \
    if (int e_ = (int)(x)) {                                           \
      printf("%s: %d %s\n", #x, e_, last_error_text() ? last_error_text() : ""); \
      return 2;                                                        \
    }                                                                  \
  } while (0)

template <class T>
static T* dev(const std::vector<T>& v) {
  T* p = nullptr;
  if (cudaMalloc((void**)&p, v.size() * sizeof(T)) != cudaSuccess) return nullptr;
  cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice);
  return p;
}
template <class T>
static std::vector<T> host(const T* p, size_t n) {
  std::vector<T> v(n);
  cudaMemcpy(v.data(), p, n * sizeof(T), cudaMemcpyDeviceToHost);
  return v;
}
static __half* plane(size_t n) { return dev(std::vector<__half>(n, __float2half(0.f))); }

struct Weights {
  int8_t* q = nullptr;
  float* s = nullptr;
};
// n x k, ones on the diagonal
static Weights diagonal(int n, int k) {
  std::vector<int8_t> q((size_t)n * k, 0);
  std::vector<float> s((size_t)n * (k / 32), 1.f);
  for (int i = 0; i < n && i < k; ++i) q[(size_t)i * k + i] = 1;
  Weights w;
  const size_t rows = (size_t)(n + 127) / 128 * 128;
  w.q = dev(std::vector<int8_t>(rows * k));
  w.s = dev(std::vector<float>(rows * (k / 32)));
  launch_q8_retile(dev(q), w.q, n, k, true, 0, nullptr);
  launch_q8_retile_scales(dev(s), w.s, n, k, true, 0, nullptr);
  return w;
}
static unsigned rnd(unsigned* x) { return *x = *x * 1664525u + 1013904223u; }
static const char* name(int mode) { return mode == LOGOS_F32 ? "two planes" : mode == LOGOS_F16 ? "fp16" : "bf16"; }

struct Planes {
  ActOut out;
  size_t n = 0;
  Planes(int mode, size_t elems) : n(elems) {
    out.mode = mode;
    out.hi = plane(n);
    out.lo = mode == LOGOS_F32 ? plane(n) : nullptr;
  }
  // the values that a product sees
  std::vector<float> values() const {
    const auto hi = host(out.hi, n);
    std::vector<float> v(n);
    for (size_t i = 0; i < n; ++i) v[i] = __half2float(hi[i]);
    if (out.lo) {
      const auto lo = host(out.lo, n);
      for (size_t i = 0; i < n; ++i) v[i] += __half2float(lo[i]) * 0x1p-11f;
    }
    return v;
  }
};

// The norm inside a product is the norm kernel's: rows of small whole numbers, whose squares add up exactly in any order, times ones on
// the diagonal, against the planes that the norm kernel makes of the same rows; through SwiGLU, against its kernel's.
static int norm(int m, int k, int mode) {
  std::vector<float> h((size_t)m * k), gain(k);
  unsigned x = 12345u + m + k;
  for (float& v : h) v = (float)((int)(rnd(&x) >> 28) - 8);
  for (float& v : gain) v = 0.5f + (float)(rnd(&x) >> 24) / 256.f;
  float *dh = dev(h), *dg = dev(gain), *c = dev(std::vector<float>((size_t)m * k, 0.f));
  const Planes want(mode, (size_t)m * k), got(mode, (size_t)m * k / 2);
  CHECK(launch_residual_rmsnorm(dh, nullptr, 0, 0, dg, want.out, m, k, 1e-6f, nullptr));
  const Weights w = diagonal(k, k);
  NarrowArgs a;
  a.q = w.q; a.s = w.s; a.m = m; a.n = k; a.k = k; a.h_in = dh; a.gain = dg; a.eps = 1e-6f; a.act_mode = mode; a.out = NARROW_F32; a.c = c;
  CHECK(launch_q8_narrow(a, nullptr));
  a.out = NARROW_SWIGLU; a.planes = got.out;
  CHECK(launch_q8_narrow(a, nullptr));
  CHECK(cudaDeviceSynchronize());
  const auto v = want.values(), cv = host(c, (size_t)m * k);
  int differing = 0;
  for (size_t i = 0; i < v.size(); ++i) differing += cv[i] != v[i];
  printf("norm, %s %d %d %d\n", name(mode), m, k, differing);

  std::vector<float> gate(v.size() / 2), up(v.size() / 2);
  for (size_t i = 0; i < gate.size(); ++i) { gate[i] = v[2 * i]; up[i] = v[2 * i + 1]; }
  float* y = dev(std::vector<float>(gate.size()));
  CHECK(launch_swiglu_f32(dev(gate), dev(up), y, (int64_t)gate.size(), nullptr));
  CHECK(cudaDeviceSynchronize());
  const auto yv = host(y, gate.size()), gv = got.values();
  differing = 0;
  for (size_t i = 0; i < yv.size(); ++i) {
    const float r = mode == LOGOS_BF16 ? __bfloat162float(__float2bfloat16_rn(yv[i])) : yv[i];
    const float hi = __half2float(__float2half_rn(r)), lo = __half2float(__float2half_rn((r - hi) * 2048.f));
    differing += gv[i] != (mode == LOGOS_F32 ? hi + lo * 0x1p-11f : hi);
  }
  printf("norm, SwiGLU, %s %d %d %d\n", name(mode), m, k, differing);
  return 0;
}

// c += a * w with ones on the diagonal: one rounded addition.
static int residual(int m, int n, int k, int mode) {
  // planes as the kernels make them of f32 values: a low part is at most half a last place of its high part, and the two
  // together fit 24 bits, so that their sum is exact wherever it is formed
  Planes a(mode, (size_t)m * k);
  std::vector<__half> hi(a.n), lo(a.n);
  unsigned x = 777u + m + k;
  for (size_t i = 0; i < a.n; ++i) {
    const float f = (float)(int)rnd(&x) / 1073741824.f;
    hi[i] = __float2half_rn(f);
    lo[i] = __float2half_rn((f - __half2float(hi[i])) * 2048.f);
  }
  a.out.hi = dev(hi);
  if (a.out.lo) a.out.lo = dev(lo);
  std::vector<float> h((size_t)m * n);
  for (float& v : h) v = (float)(int)(rnd(&x) >> 8) / 8388608.f - 1.f;
  float* c = dev(h);
  const Weights w = diagonal(n, k);
  NarrowArgs g;
  g.q = w.q; g.s = w.s; g.m = m; g.n = n; g.k = k; g.a = a.out; g.out = NARROW_RESIDUAL; g.c = c;
  CHECK(launch_q8_narrow(g, nullptr));
  CHECK(cudaDeviceSynchronize());
  const auto v = a.values(), cv = host(c, (size_t)m * n);
  int differing = 0;
  for (int t = 0; t < m; ++t)
    for (int i = 0; i < n; ++i) differing += cv[(size_t)t * n + i] != h[(size_t)t * n + i] + (i < k ? v[(size_t)t * k + i] : 0.f);
  printf("residual, %s %d %d %d\n", name(mode), m, k, differing);
  return 0;
}

int main() {
  for (int mode : {LOGOS_F32, LOGOS_F16, LOGOS_BF16})
    for (int m : {1, 4, 8, 16}) {
      for (int k : {128, 896, 1024})
        if (int rc = norm(m, k, mode)) return rc;
      for (int k : {128, 896, 4864})   // a CTA along K, and a cluster of five
        if (int rc = residual(m, 896, k, mode)) return rc;
    }
  return 0;
}
