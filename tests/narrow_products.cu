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
// k x k, the identity
static Weights identity(int k) {
  std::vector<int8_t> q((size_t)k * k, 0);
  std::vector<float> s((size_t)k * (k / 32), 1.f);
  for (int i = 0; i < k; ++i) q[(size_t)i * k + i] = 1;
  Weights w;
  w.q = dev(std::vector<int8_t>((size_t)k * k));
  w.s = dev(std::vector<float>((size_t)k * (k / 32)));
  launch_q8_retile(dev(q), w.q, k, k, true, 0, nullptr);
  launch_q8_retile_scales(dev(s), w.s, k, k, true, 0, nullptr);
  return w;
}

// The norm inside a product is the norm kernel's: rows of small whole numbers, whose squares add up exactly in any order, times the
// identity, against the planes that the norm kernel makes of the same rows.
static int norm(int m, int k) {
  std::vector<float> h((size_t)m * k), gain(k);
  unsigned x = 12345u + m + k;
  for (float& v : h) { x = x * 1664525u + 1013904223u; v = (float)((int)(x >> 28) - 8); }
  for (float& v : gain) { x = x * 1664525u + 1013904223u; v = 0.5f + (float)(x >> 24) / 256.f; }
  float *dh = dev(h), *dg = dev(gain), *c = dev(std::vector<float>((size_t)m * k, 0.f));
  ActOut planes;
  planes.hi = plane((size_t)m * k);
  planes.lo = plane((size_t)m * k);
  CHECK(launch_residual_rmsnorm(dh, nullptr, 0, 0, dg, planes, m, k, 1e-6f, nullptr));
  const Weights w = identity(k);
  NarrowArgs a;
  a.q = w.q; a.s = w.s; a.m = m; a.n = k; a.k = k; a.h_in = dh; a.gain = dg; a.eps = 1e-6f; a.out = NARROW_F32; a.c = c;
  CHECK(launch_q8_narrow(a, nullptr));
  CHECK(cudaDeviceSynchronize());
  const auto hi = host(planes.hi, (size_t)m * k), lo = host(planes.lo, (size_t)m * k);
  const auto got = host(c, (size_t)m * k);
  int differing = 0;
  for (size_t i = 0; i < got.size(); ++i) differing += got[i] != __half2float(hi[i]) + __half2float(lo[i]) * 0x1p-11f;
  printf("norm %d %d %d\n", m, k, differing);
  return 0;
}

int main() {
  for (int m : {1, 4, 8, 16})
    for (int k : {128, 896, 1024})
      if (int rc = norm(m, k)) return rc;
  return 0;
}
