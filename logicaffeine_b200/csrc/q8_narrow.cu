// Q8 products of a small model's decode step: few tokens, matrices that the SMs' shared memories hold, one launch each.
//
//   norm forms:     c[t][n] = sum_k rmsnorm(h[t])[k] * w[n][k]        (f32, or through SwiGLU into activation planes)
//   residual form:  h[t][n] += sum_k a[t][k] * w[n][k]                (o_proj and down_proj)
//
// What bounds it: latency.  A layer of the 0.5B shape is 17 MB of weights, 3 us of HBM time, and a step is a chain of
// these kernels, so each is built around the time from its predecessor's end to its own (an empty kernel in such a
// chain takes 0.77 us, a round of loads from L2 0.4, a cluster barrier 0.3, an instruction of a warp's chain about six cycles):
//   * nothing is left to a kernel of its own: the RMSNorm, SwiGLU, the residual add, the fold of the K splits;
//   * a warp owns 64 columns of K (two Q8 blocks) for all of its CTA's units of 16 rows.  Its weights and scales are copied to
//     shared memory, every lane the bytes that it will use, before the wait for the predecessor; its activations go from
//     global memory straight into the fragments of the MMA, normalised on the way: no staging, and no element is
//     normalised twice in a CTA;
//   * the warps' sums are added through shared memory, K in ascending order.  Where K has more columns than sixteen warps take, a
//     cluster lies along it and its CTAs push their sums into the first one's shared memory.  (Pulled, by 512 threads 16 bytes from
//     each of seven CTAs, they took 8.7 us.)
//   * mma.sync: 64 columns and at most 16 tokens a warp are too little work for an accumulator in tensor memory to
//     pay for its allocation, hand-offs and read-back.
// Measured on a B200, from the wait's return to the last store, 0.5B shape at 8 / 16 tokens (us): qkv 2.4 / 2.9, o_proj 1.5 / 2.0,
// gate/up 4.4 / 5.8, down_proj 2.4 / 3.0 (the rounded norm factor and the status word came later: 0.1 together); a step at batch
// 1 / 8 / 16 477 / 546 / 663 (with norm and GEMM kernels of their own see narrow_layers in llm.cu).
// Of gate/up's time 2.1 / 2.6 us are the products: mma.sync runs at one m16n8k16 in 4.3 cycles an SM.
// Arithmetic as in q8_gemm_tc.cu: int8 -> fp16 exactly, activations in two fp16 planes, a Q8 block's products summed on
// the tensor core (q * lo' first, times 2^-11, then q * hi), then sum += scale * partial in f32.
#include "ops.cuh"
#include "ptx.cuh"

#include <cooperative_groups.h>

#include <algorithm>

namespace logos {

namespace {

using namespace ptx;
namespace cg = cooperative_groups;

constexpr int NW_WARPS = 16, NW_THREADS = NW_WARPS * 32;   // 64 columns a warp
constexpr int NW_UNIT = 16;                          // rows of a unit (MMA M)
constexpr int NW_PIECE = 1024 + NW_UNIT * 8;         // a warp's part of a unit: weights [4][32 lanes] x 8 bytes, scales [16 rows][2]
constexpr int NW_MAX_RANKS = 8;
constexpr int NW_MAX_SMEM = 200 * 1024;

struct NarrowParams {
  const int8_t* q;      // tile-major
  const float* s;
  int n, k, m;
  int units, rt;        // of the matrix, of a CTA
  int ranks;            // CTAs along K
  const float* h_in;    // norm forms
  const float* gain;
  float eps, inv_k;     // inv_k = 1 / k, rounded
  const __half* a_hi;   // residual form
  const __half* a_lo;   // null: one plane
  int act_mode;
  float* c;             // f32 results [m][n], or the residual stream
  ActOut planes;
  int* status;
};

__device__ __forceinline__ uint2 lds_v2(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void cp_async8(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return make_float2(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y)); }
// sum / k, correctly rounded: with the reciprocal's rounded value at hand one step on the quotient's remainder gives that
// (Markstein, IBM J. Res. Dev. 34, 1990).  __fdiv_rn on the kernel's chain: a step of the 0.5B shape at batch 1 473 -> 486 us.
__device__ __forceinline__ float mean(float sum, float k, float inv_k) {
  const float q = __fmul_rn(sum, inv_k);
  return q < INFINITY ? fmaf(fmaf(-q, k, sum), inv_k, q) : q;
}

// Grid: x = unit groups x CTAs along K (a cluster), y = token tiles; a warp for every 64 columns.
// Up to four tokens (TOK = 4) both planes of them are the eight columns of one MMA, hi 0 to 3 and lo 4 to 7: half the MMAs (a
// step of the 0.5B shape at batch 1 498 -> 474 us).
template <int TOK, int OUT>
__global__ void __launch_bounds__(NW_THREADS)
q8_narrow_kernel(const NarrowParams p) {
  constexpr bool NORM = OUT != NARROW_RESIDUAL;
  constexpr bool MERGED = TOK == 4;
  constexpr int NT = MERGED ? 1 : TOK / 8;                      // MMAs side by side, of eight columns
  constexpr int PAIRS = NW_UNIT / 2 * TOK;                      // of a unit: two neighbouring output columns for a token
  constexpr int UNIT_PIECES = NW_WARPS * NW_PIECE;
  constexpr int COLS = 18;                                      // floats between the tokens of a warp's sums
  static_assert(TOK * COLS * 4 <= NW_PIECE, "the sums take the weights' place");
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ float s_ss[NW_WARPS][TOK];
  __shared__ uint64_t s_bar;
  __shared__ int s_prior;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  const int ranks = NORM ? 1 : p.ranks, rank = NORM ? 0 : (int)(blockIdx.x % (unsigned)ranks);
  const int slices = p.k / 64, sl0 = rank * slices / ranks, warps = (rank + 1) * slices / ranks - sl0;
  const int unit0 = (int)(blockIdx.x / (unsigned)ranks) * p.rt, have = min(p.rt, p.units - unit0);
  const int m0 = blockIdx.y * TOK, rows = min(TOK, p.m - m0);
  const int slice = sl0 + warp, col = slice * 64;
  const bool active = warp < warps;
  // pieces [unit][warp], whose place the sums [TOK][COLS] take; then, in the first CTA of a cluster, the others' sums
  const uint32_t piece0 = smem_u32(smem) + warp * NW_PIECE;
  const uint32_t pushed = smem_u32(smem) + p.rt * UNIT_PIECES;
  const int all = have * PAIRS;

  pdl_trigger();
  // A code that an earlier kernel left: nothing is stored on top of it.  One thread reads and the CTA takes one decision; of a
  // cluster the CTA that stores does, and the others push all the same, since it waits for what they push.  Read before the wait
  // for the predecessor, as the kernels of q8_gemm_tc.cu do: all CTAs ask one L2 line for the word, and after the wait that is on
  // the kernel's chain (a step of the 0.5B shape at batch 16 675 -> 688 us; 695 with every thread asking).
  int status = 0;
  if (tid == 0) status = *reinterpret_cast<volatile int*>(p.status);
  // ---- weights, scales, gains: nothing in a step writes them
  float4 gain[4];
  if (active) {
    const int64_t ktiles = p.k / 128, kt = slice >> 1;
    for (int r = 0; r < have; ++r) {
      const int u = unit0 + r;
      const int64_t row0 = ((u >> 3) * ktiles + kt) * 128 + (u & 7) * NW_UNIT;   // of the tile-major array
      const int8_t* q = p.q + (row0 + g) * 128 + (slice & 1) * 64 + t4 * 8;
      const uint32_t dst = piece0 + r * UNIT_PIECES + lane * 8;
#pragma unroll
      for (int i = 0; i < 4; ++i) cp_async8(dst + i * 256, q + (i & 1) * 8 * 128 + (i >> 1) * 32);   // rows g, g + 8 of either block
      if (lane < NW_UNIT) cp_async8(piece0 + r * UNIT_PIECES + 1024 + lane * 8, p.s + (row0 + lane) * 4 + (slice & 1) * 2);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (NORM)
#pragma unroll
      for (int i = 0; i < 4; ++i) gain[i] = __ldg(reinterpret_cast<const float4*>(p.gain + col + (i >> 1) * 32 + t4 * 8) + (i & 1));
  }
  if (!NORM && ranks > 1) {
    if (rank == 0 && tid == 0) {
      mbar_init(&s_bar, 1);
      fence_barrier_init();
      mbar_arrive_expect_tx(&s_bar, (ranks - 1) * all * 8);
    }
    cg::this_cluster().barrier_arrive();   // "this CTA runs, its barrier stands": before anyone pushes into it
  }
  if (tid == 0) s_prior = status;
  pdl_wait();

  // ---- fragments of the activations: a lane has columns 8 t4 .. 8 t4 + 7 of either block, for tokens g + 8 j
  uint4 bh[2][NT], bl[2][NT];
  const bool two = NORM ? p.act_mode == LOGOS_F32 : p.a_lo != nullptr;
  if (NORM) {
    float4 v[NT][4];
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      const int t = MERGED ? g & 3 : g + 8 * j;
      const float* src = p.h_in + (int64_t)(m0 + t) * p.k + col + t4 * 8;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        v[j][i] = active && t < rows ? __ldcg(reinterpret_cast<const float4*>(src + (i >> 1) * 32) + (i & 1)) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      float2 ss = make_float2(0.f, 0.f);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 x = make_float2(v[j][i].x, v[j][i].y), y = make_float2(v[j][i].z, v[j][i].w);
        ss = __ffma2_rn(x, x, ss);
        ss = __ffma2_rn(y, y, ss);
      }
      float t = ss.x + ss.y;
      t += __shfl_xor_sync(0xffffffffu, t, 1);
      t += __shfl_xor_sync(0xffffffffu, t, 2);
      if (t4 == 0 && g + 8 * j < TOK) s_ss[warp][g + 8 * j] = t;
    }
    __syncthreads();
    float ss[NW_WARPS];
#pragma unroll
    for (int w = 0; w < NW_WARPS; ++w) ss[w] = s_ss[w][lane % TOK];
#pragma unroll
    for (int o = NW_WARPS / 2; o > 0; o >>= 1)
#pragma unroll
      for (int w = 0; w < o; ++w) ss[w] += ss[w + o];
    const float inv_all = __frcp_rn(__fsqrt_rn(__fadd_rn(mean(ss[0], (float)p.k, p.inv_k), p.eps)));   // of token `lane`
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      const float i1 = __shfl_sync(0xffffffffu, inv_all, MERGED ? g & 3 : g + 8 * j);
      const float2 inv = make_float2(i1, i1);
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        const float4 x = v[j][2 * b], y = v[j][2 * b + 1];
        const float4 gx = active ? gain[2 * b] : make_float4(0.f, 0.f, 0.f, 0.f), gy = active ? gain[2 * b + 1] : gx;
        float2 n[4] = {__fmul2_rn(__fmul2_rn(make_float2(x.x, x.y), inv), make_float2(gx.x, gx.y)),
                       __fmul2_rn(__fmul2_rn(make_float2(x.z, x.w), inv), make_float2(gx.z, gx.w)),
                       __fmul2_rn(__fmul2_rn(make_float2(y.x, y.y), inv), make_float2(gy.x, gy.y)),
                       __fmul2_rn(__fmul2_rn(make_float2(y.z, y.w), inv), make_float2(gy.z, gy.w))};
        if (p.act_mode == LOGOS_BF16)
#pragma unroll
          for (int i = 0; i < 4; ++i) n[i] = __bfloat1622float2(__floats2bfloat162_rn(n[i].x, n[i].y));
        act_words(n[0], &bh[b][j].x, &bl[b][j].x);
        act_words(n[1], &bh[b][j].y, &bl[b][j].y);
        act_words(n[2], &bh[b][j].z, &bl[b][j].z);
        act_words(n[3], &bh[b][j].w, &bl[b][j].w);
        if (MERGED && g >= 4) bh[b][j] = two ? bl[b][j] : make_uint4(0u, 0u, 0u, 0u);
      }
    }
  } else {
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      const int t = MERGED ? g & 3 : g + 8 * j;
      const int64_t at = (int64_t)(m0 + t) * p.k + col + t4 * 8;
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        if (MERGED) {
          const __half* plane = g < 4 ? p.a_hi : p.a_lo;
          bh[b][j] = active && t < rows && plane ? __ldcg(reinterpret_cast<const uint4*>(plane + at + b * 32)) : zero;
          continue;
        }
        bh[b][j] = active && t < rows ? __ldcg(reinterpret_cast<const uint4*>(p.a_hi + at + b * 32)) : zero;
        bl[b][j] = active && t < rows && two ? __ldcg(reinterpret_cast<const uint4*>(p.a_lo + at + b * 32)) : zero;
      }
    }
  }
  // a thread finishes a pair of output columns for a token: lanes along the columns of a unit
  const int n0 = unit0 * NW_UNIT;
  auto column = [&](int e) { return n0 + e / PAIRS * NW_UNIT + e % 8 * 2; };
  auto token = [&](int e) { return e % PAIRS / 8; };
  float2 h0 = make_float2(0.f, 0.f);   // the residual values of the first, needed last
  if (!NORM && rank == 0 && tid < all && column(tid) < p.n && token(tid) < rows)
    h0 = __ldcg(reinterpret_cast<const float2*>(p.c + (int64_t)(m0 + token(tid)) * p.n + column(tid)));

  // ---- products.  The chains (block, tokens) advance together, since instructions issue in order.
  if (active) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    for (int r = 0; r < have; ++r) {
      const uint32_t piece = piece0 + r * UNIT_PIECES;
      uint2 w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) w[i] = lds_v2(piece + i * 256 + lane * 8);
      const uint2 s0 = lds_v2(piece + 1024 + g * 8), s1 = lds_v2(piece + 1024 + (g + 8) * 8);
      uint32_t a[2][2][4];   // [block][K step]
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        const uint32_t w0[2] = {w[2 * b].x, w[2 * b].y}, w1[2] = {w[2 * b + 1].x, w[2 * b + 1].y};
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          a[b][k][0] = cvt_pair(w0[k], 0x4140);
          a[b][k][1] = cvt_pair(w1[k], 0x4140);
          a[b][k][2] = cvt_pair(w0[k], 0x4342);
          a[b][k][3] = cvt_pair(w1[k], 0x4342);
        }
      }
      float d[2][NT][4];
      auto each = [&](auto f) {
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
          for (int j = 0; j < NT; ++j) f(b, j);
      };
      each([&](int b, int j) { d[b][j][0] = d[b][j][1] = d[b][j][2] = d[b][j][3] = 0.f; });
      if (two && !MERGED) {
        each([&](int b, int j) { mma_f16_16816(d[b][j], a[b][0], bl[b][j].x, bl[b][j].y); });
        each([&](int b, int j) { mma_f16_16816(d[b][j], a[b][1], bl[b][j].z, bl[b][j].w); });
        each([&](int b, int j) {
          for (int x = 0; x < 4; ++x) d[b][j][x] *= 4.8828125e-4f;   // 2^-11
        });
      }
      each([&](int b, int j) { mma_f16_16816(d[b][j], a[b][0], bh[b][j].x, bh[b][j].y); });
      each([&](int b, int j) { mma_f16_16816(d[b][j], a[b][1], bh[b][j].z, bh[b][j].w); });
      __syncwarp();   // every lane has its weights and scales: the sums [token][row] take their place
      float* sums = reinterpret_cast<float*>(smem + r * UNIT_PIECES + warp * NW_PIECE);
      const float sc0[2] = {__uint_as_float(s0.x), __uint_as_float(s0.y)}, sc1[2] = {__uint_as_float(s1.x), __uint_as_float(s1.y)};
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const float* sc = x < 2 ? sc0 : sc1;
          float v = fmaf(sc[1], d[1][j][x], __fmul_rn(sc[0], d[0][j][x]));
          if (MERGED) v = fmaf(__shfl_xor_sync(0xffffffffu, v, 2), 4.8828125e-4f, v);   // hi + lo * 2^-11
          if (!MERGED || t4 < 2) sums[(8 * j + 2 * t4 + (x & 1)) * COLS + g + (x < 2 ? 0 : 8)] = v;
        }
    }
  } else {   // a warp without columns: zeros
    for (int i = lane; i < have * TOK * (COLS / 2); i += 32) {
      const int r = i / (TOK * (COLS / 2));
      *reinterpret_cast<float2*>(smem + r * UNIT_PIECES + warp * NW_PIECE + (i - r * (TOK * (COLS / 2))) * 8) = make_float2(0.f, 0.f);
    }
  }
  __syncthreads();

  // ---- sums over K: the CTA's warps in ascending order, then the cluster's CTAs in theirs
  auto local = [&](int e) {
    const uint32_t at = smem_u32(smem) + e / PAIRS * UNIT_PIECES + (token(e) * COLS + e % 8 * 2) * 4;
    uint2 o[NW_WARPS];   // all loads in flight, none behind a branch: a conditional load a warp took 1500 cycles
#pragma unroll
    for (int w = 0; w < NW_WARPS; ++w) o[w] = lds_v2(at + w * NW_PIECE);
    float2 v = make_float2(__uint_as_float(o[0].x), __uint_as_float(o[0].y));
#pragma unroll
    for (int w = 1; w < NW_WARPS; ++w) v = add2(v, make_float2(__uint_as_float(o[w].x), __uint_as_float(o[w].y)));
    return v;
  };
  if (!NORM && ranks > 1) {
    cg::this_cluster().barrier_wait();
    if (rank != 0) {
      const uint32_t to = smem_of_rank(pushed + (rank - 1) * all * 8, 0), bar = smem_of_rank(smem_u32(&s_bar), 0);
      for (int e = tid; e < all; e += NW_THREADS) push8(to + e * 8, local(e), bar);
      return;
    }
  }
  for (int e = tid; e < all; e += NW_THREADS) {
    float2 v = local(e);
    if (!NORM && ranks > 1) {
      if (e == tid && !mbar_wait_cluster(&s_bar, 0)) {
        // a peer is late: once all have ended or are here, what is still on its way arrives at once
        atomicCAS(p.status, 0, 4010);
        cluster_meet();
        mbar_wait_cluster(&s_bar, 0);
        return;
      }
      for (int r = 1; r < ranks; ++r) {
        const uint2 o = lds_v2(pushed + ((r - 1) * all + e) * 8);
        v = add2(v, make_float2(__uint_as_float(o.x), __uint_as_float(o.y)));
      }
    }
    const int n = column(e), t = token(e);
    if (n >= p.n || t >= rows || s_prior != 0) continue;
    const int64_t row = m0 + t;
    if (OUT == NARROW_SWIGLU) {
      act_store(p.planes, row * (p.n / 2) + n / 2, __fmul_rn(silu_f(v.x), v.y));   // columns (2j, 2j + 1) are (gate_j, up_j)
    } else {
      float2* c = reinterpret_cast<float2*>(p.c + row * p.n + n);
      if (!NORM) v = add2(e == tid ? h0 : __ldcg(c), v);
      *c = v;
    }
  }
}

// How a product is cut: as many units a CTA as spread the matrix over all SMs once.
struct NarrowPlan {
  int tok, ranks, rt, groups;
  size_t smem;
};

NarrowPlan narrow_plan(int64_t m, int64_t n, int64_t k, int sms) {
  NarrowPlan pl;
  pl.tok = m <= 4 ? 4 : m <= 8 ? 8 : 16;
  const int64_t slices = k / 64, units = (n + NW_UNIT - 1) / NW_UNIT, chunks = (m + pl.tok - 1) / pl.tok;
  pl.ranks = (int)((slices + NW_WARPS - 1) / NW_WARPS);
  const int64_t most = std::max<int64_t>(1, sms / (pl.ranks * chunks));   // groups that run at once
  pl.rt = (int)((units + most - 1) / most);
  pl.groups = (int)((units + pl.rt - 1) / pl.rt);
  pl.smem = (size_t)NW_WARPS * pl.rt * NW_PIECE + (size_t)(pl.ranks - 1) * pl.rt * NW_UNIT * pl.tok * 4;
  return pl;
}

template <int TOK, int OUT>
logos_status_t launch_t(const NarrowArgs& a, const NarrowPlan& pl, cudaStream_t st) {
  NarrowParams p{};
  p.q = a.q; p.s = a.s;
  p.n = (int)a.n; p.k = (int)a.k; p.m = (int)a.m;
  p.units = (int)((a.n + NW_UNIT - 1) / NW_UNIT); p.rt = pl.rt; p.ranks = pl.ranks;
  p.h_in = a.h_in; p.gain = a.gain; p.eps = a.eps; p.inv_k = 1.0f / (float)a.k;
  p.a_hi = a.a.hi; p.a_lo = a.a.mode == LOGOS_F32 ? a.a.lo : nullptr;
  p.act_mode = a.act_mode;
  p.c = a.c; p.planes = a.planes;
  p.status = kernel_status_ptr(a.device);
  if (!p.status) return fail(LOGOS_ERROR, "q8_narrow: no kernel status word");
  auto kernel = q8_narrow_kernel<TOK, OUT>;
  LOGOS_TRY(allow_smem(reinterpret_cast<const void*>(kernel), a.device, (int)pl.smem));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(pl.groups * pl.ranks), (unsigned)((a.m + TOK - 1) / TOK), 1u);
  cfg.blockDim = dim3(NW_THREADS);
  cfg.dynamicSmemBytes = pl.smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  int attrs = 0;
  if (pl.ranks > 1) {
    attr[attrs].id = cudaLaunchAttributeClusterDimension;
    attr[attrs].val.clusterDim.x = (unsigned)pl.ranks;
    attr[attrs].val.clusterDim.y = 1;
    attr[attrs++].val.clusterDim.z = 1;
  }
  if (pdl_active()) {
    attr[attrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[attrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = attrs;
  LOGOS_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, p));
  count_launch(LK_GEMM_TC);
  return check_launch("q8_narrow_kernel");
}

template <int TOK>
logos_status_t launch_tok(const NarrowArgs& a, const NarrowPlan& pl, cudaStream_t st) {
  switch (a.out) {
    case NARROW_F32: return launch_t<TOK, NARROW_F32>(a, pl, st);
    case NARROW_SWIGLU: return launch_t<TOK, NARROW_SWIGLU>(a, pl, st);
    default: return launch_t<TOK, NARROW_RESIDUAL>(a, pl, st);
  }
}

}  // namespace

bool narrow_applicable(int64_t m, int64_t n, int64_t k, bool norm, int device) {
  if (m < 1 || n < 2 || n % 2 || k < 128 || k % 128 || n > (1 << 24)) return false;
  if (k > NW_WARPS * 64 * (norm ? 1 : NW_MAX_RANKS)) return false;   // a norm needs whole rows in a CTA
  return narrow_plan(m, n, k, sm_count(device)).smem <= (size_t)NW_MAX_SMEM;
}

logos_status_t launch_q8_narrow(const NarrowArgs& a, cudaStream_t st) {
  const bool norm = a.out != NARROW_RESIDUAL;
  if (!narrow_applicable(a.m, a.n, a.k, norm, a.device)) return fail(LOGOS_ERROR, "q8_narrow: extents out of its range");
  const NarrowPlan pl = narrow_plan(a.m, a.n, a.k, sm_count(a.device));
  switch (pl.tok) {
    case 4: return launch_tok<4>(a, pl, st);
    case 8: return launch_tok<8>(a, pl, st);
    default: return launch_tok<16>(a, pl, st);
  }
}

}  // namespace logos
