// GQA decode attention over an fp16 KV cache, with the rotary embedding and
// the KV-cache append fused in.
//
// HBM-bound where the cache is large: every step streams the whole K and V history once (512 bytes per
// position per KV head at D=128).  Latency-bound where it is small.  So:
//   * a (sequence, KV head) pair is a cluster of one to eight CTAs (up to sixteen where sequences can be long), each of which takes an
//     equal part of the pair's 64-position K/V tiles: as many as make the fewest and shortest rounds (attn_cut).  Clusters
//     start as room comes free, so ragged lengths and several rounds of them even out by themselves;
//   * a producer thread moves the tiles into a shared-memory ring with TMA tile loads (128-byte swizzle, no multicast)
//     signalled on mbarriers; four consumer warps each own 16 positions of every tile;
//   * all query heads that share the KV head (up to 16) form the M side of
//     m16n8k16 tensor-core MMAs, so a K/V tile is read from shared memory once
//     for the whole group; scores, softmax and the running output stay in f32
//     registers; the probabilities enter the second MMA as an fp16 high part
//     plus an fp16 residual so the product keeps f32-class accuracy;
//   * the CTA whose part holds the position being appended rotates the new key
//     (f32 multiply and add rounded separately, fp16 store), writes the new
//     K/V row to the cache and patches it into its own shared-memory tile;
//   * the parts meet in shared memory: row i of the query group is finished by CTA i % parts, into whose memory the others
//     push their sums for it (st.async, counted on an mbarrier), and added there in the order of their positions: nothing
//     goes through global memory;
//   * in a decode step what is older than it (lengths, cached rows) is read before the wait for
//     the predecessor (AttnArgs::early_reads); every row of the query and the new K/V is one round of loads.
// With cold caches and the events' 8 us (us): 64 sequences of 1024, 64/8 heads of 128 68; 32 of 4096, 28/4 66; 4 of 32768, 28/4 70;
// 7 of up to 2000, 14/2 of 64 15; one of 4096, 64/8 19.  Three ring stages at head dimension 128 against two: 64 of 1300, 64/8 86 -> 85,
// 25 of 2000, 28/4 41 -> 40.
#include "ops.cuh"
#include "q8_gemm_tc.cuh"
#include "ptx.cuh"

#include <cooperative_groups.h>
#include <math.h>

#include <limits.h>

#include <algorithm>
#include <mutex>
#include <unordered_map>

namespace logos {

namespace {

using namespace ptx;
namespace cg = cooperative_groups;

constexpr int ATT_TILE = 64;
constexpr int ATT_CWARPS = 4;
constexpr int ATT_CTHREADS = ATT_CWARPS * 32;
constexpr int ATT_THREADS = (ATT_CWARPS + 1) * 32;
constexpr int ATT_BOX_BYTES = 64 * 128;  // 64 rows x 128 bytes
constexpr int ATT_MAX_BATCH = 2048;      // sequences a call
constexpr int ATT_PUSHED_ROWS = 21;      // parts x ceil(group / parts), exact for up to 8 parts; of more, only counts that keep to it
constexpr int ATT_WIDE = 16;             // CTAs of the largest cluster; the next has 8, as many as are portable

struct AttnParams {
  const __half* q_f16;
  const float*  q_f32;
  int64_t       q_ld;
  int           rotate_q;
  const __half* k_new_f16;
  const __half* v_new_f16;
  const float*  k_new_f32;
  const float*  v_new_f32;
  int64_t       kv_ld;
  int           f32_parts;        // split-K partial copies of the f32 inputs, summed while staging
  int64_t       f32_part_stride;
  const float*  q_bias;           // f32 inputs only: added after the partial copies (null = none)
  const float*  k_bias;
  const float*  v_bias;
  int           fused;
  __half*       k_cache;
  __half*       v_cache;
  const float*  rope;
  int32_t* seq_len;
  unsigned*     arrive;   // with bump: CTAs that have their length; zero before and after every launch (it wraps by itself)
  int           bump;     // the last CTA to have its length advances the lengths
  int           early_reads;   // see AttnArgs
  void*         o;        // [B][Hq][D]
  int           o_dtype;
  ActOut        o_act;
  int           b, h_q, h_kv, l_max;
  int           ranks;    // CTAs of a pair's cluster; all of them have tiles from `all_from` tiles on, at most `few` below that
  int           few, all_from;
  float         scale_log2;
  int*          status;
};

__device__ __forceinline__ uint32_t pack_half2(float a, float b) {
  __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}

__device__ __forceinline__ int attn_len_eff(const AttnParams& p, int len0) {
  int len_eff = p.fused ? len0 + 1 : len0;
  if (len_eff > p.l_max) len_eff = p.l_max;
  return len_eff < 0 ? 0 : len_eff;
}

// Counts up to `last`, then wraps to zero; releases what came before and acquires what the others released.
__device__ __forceinline__ unsigned arrive_inc(unsigned* counter, unsigned last) {
  unsigned old;
  asm volatile("atom.acq_rel.gpu.global.inc.u32 %0, [%1], %2;" : "=r"(old) : "l"(counter), "r"(last) : "memory");
  return old;
}

__device__ __forceinline__ void store_out(const AttnParams& p, int64_t oi, float v) {
  if (p.o_dtype == LOGOS_ACT_PLANES) act_store(p.o_act, oi, v);
  else if (p.o_dtype == LOGOS_F16) reinterpret_cast<__half*>(p.o)[oi] = __float2half_rn(v);
  else if (p.o_dtype == LOGOS_BF16) reinterpret_cast<__nv_bfloat16*>(p.o)[oi] = __float2bfloat16_rn(v);
  else reinterpret_cast<float*>(p.o)[oi] = v;
}

// Four neighbouring outputs (their index a multiple of four) over their row's normaliser.
__device__ __forceinline__ void store_out4(const AttnParams& p, int64_t oi, float4 v, float l) {
  v = make_float4(__fdiv_rn(v.x, l), __fdiv_rn(v.y, l), __fdiv_rn(v.z, l), __fdiv_rn(v.w, l));
  if (p.o_dtype == LOGOS_ACT_PLANES) {
    act_store4(p.o_act, oi, v);
  } else {
    store_out(p, oi, v.x);
    store_out(p, oi + 1, v.y);
    store_out(p, oi + 2, v.z);
    store_out(p, oi + 3, v.w);
  }
}

// The query heads of a pair (rotated when asked) and zeros in the padding rows of qs; with owns_new the appended row too: rotated,
// rounded to fp16, written to the cache and kept in new_k, new_v.  A thread takes four columns of a row and their
// partners half a head away, so that all rows are one round of loads (every part of a split sum in flight at once).
template <int D>
__device__ __forceinline__ void stage_query(const AttnParams& p, int b, int kvh, int len0, bool owns_new, int64_t row_base, int ctid,
                                            __half* qs, __half* new_k, __half* new_v) {
  constexpr int QS_STRIDE = D + 8;
  const int G = p.h_q / p.h_kv, pos_new = len0;
  constexpr int half_d = D / 2, QUADS = half_d / 4;
  int pos_q = len0 < p.l_max ? len0 : p.l_max - 1;
  if (pos_q < 0) pos_q = 0;
  const int fresh = owns_new ? 2 : 0;   // rows G and G + 1 of the list: the new k and v
  for (int i = ctid; i < (16 + fresh) * QUADS; i += ATT_CTHREADS) {
    const int row = i / QUADS, e = 4 * (i - row * QUADS);
    const int kind = row < G ? 0 : row < G + fresh ? row - G + 1 : 3;   // query, k, v, padding
    if (kind == 3) {
      *reinterpret_cast<uint2*>(qs + (row - fresh) * QS_STRIDE + e) = make_uint2(0u, 0u);
      *reinterpret_cast<uint2*>(qs + (row - fresh) * QS_STRIDE + e + half_d) = make_uint2(0u, 0u);
      continue;
    }
    const int head = kind == 0 ? kvh * G + row : kvh;
    float x1[4], x2[4];
    if (p.q_f16) {
      const __half* src = kind == 0 ? p.q_f16 + ((int64_t)b * p.h_q + head) * D
                                    : (kind == 1 ? p.k_new_f16 : p.v_new_f16) + ((int64_t)b * p.h_kv + head) * D;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        x1[j] = __half2float(__ldcg(src + e + j));
        x2[j] = __half2float(__ldcg(src + e + half_d + j));
      }
    } else {
      const float* src = (kind == 0 ? p.q_f32 + (int64_t)b * p.q_ld : (kind == 1 ? p.k_new_f32 : p.v_new_f32) + (int64_t)b * p.kv_ld) +
                         (int64_t)head * D + e;
      const float* bias = kind == 0 ? p.q_bias : kind == 1 ? p.k_bias : p.v_bias;
      float4 u1 = __ldcg(reinterpret_cast<const float4*>(src)), u2 = __ldcg(reinterpret_cast<const float4*>(src + half_d));
      x1[0] = u1.x; x1[1] = u1.y; x1[2] = u1.z; x1[3] = u1.w;
      x2[0] = u2.x; x2[1] = u2.y; x2[2] = u2.z; x2[3] = u2.w;
#pragma unroll 4
      for (int sp = 1; sp < p.f32_parts; ++sp) {
        const float* part = src + sp * p.f32_part_stride;
        u1 = __ldcg(reinterpret_cast<const float4*>(part));
        u2 = __ldcg(reinterpret_cast<const float4*>(part + half_d));
        x1[0] = __fadd_rn(x1[0], u1.x); x1[1] = __fadd_rn(x1[1], u1.y); x1[2] = __fadd_rn(x1[2], u1.z); x1[3] = __fadd_rn(x1[3], u1.w);
        x2[0] = __fadd_rn(x2[0], u2.x); x2[1] = __fadd_rn(x2[1], u2.y); x2[2] = __fadd_rn(x2[2], u2.z); x2[3] = __fadd_rn(x2[3], u2.w);
      }
      if (bias)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          x1[j] = __fadd_rn(x1[j], __ldg(bias + head * D + e + j));
          x2[j] = __fadd_rn(x2[j], __ldg(bias + head * D + e + half_d + j));
        }
    }
    if (kind == 1 || (kind == 0 && p.rotate_q)) {
      const float* tab = p.rope + ((int64_t)(kind == 0 ? pos_q : pos_new) * half_d + e) * 2;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float c = tab[2 * j], s = tab[2 * j + 1];
        const float r1 = __fsub_rn(__fmul_rn(x1[j], c), __fmul_rn(x2[j], s));
        const float r2 = __fadd_rn(__fmul_rn(x2[j], c), __fmul_rn(x1[j], s));
        x1[j] = r1;
        x2[j] = r2;
      }
    }
    const uint2 h1 = make_uint2(pack_half2(x1[0], x1[1]), pack_half2(x1[2], x1[3]));
    const uint2 h2 = make_uint2(pack_half2(x2[0], x2[1]), pack_half2(x2[2], x2[3]));
    __half* dst = kind == 0 ? qs + row * QS_STRIDE : kind == 1 ? new_k : new_v;
    *reinterpret_cast<uint2*>(dst + e) = h1;
    *reinterpret_cast<uint2*>(dst + e + half_d) = h2;
    if (kind != 0) {
      __half* cache = (kind == 1 ? p.k_cache : p.v_cache) + (row_base + pos_new) * D;
      *reinterpret_cast<uint2*>(cache + e) = h1;
      *reinterpret_cast<uint2*>(cache + e + half_d) = h2;
    }
  }
}

// What a warp has of a pair: the query's fragments, its 16 positions' share of the softmax and the output.
template <int D>
struct AttnState {
  uint32_t qa[D / 16][4];
  float m_run[2], l_run[2];
  float o[D / 8][4];
  __device__ __forceinline__ void start(const __half* qs, int lane) {
    constexpr int QS_STRIDE = D + 8;
    const int row = (lane & 7) + 8 * ((lane >> 3) & 1), colh = 8 * (lane >> 4);
#pragma unroll
    for (int ks = 0; ks < D / 16; ++ks)
      ldmatrix_x4(qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3], smem_u32(qs + row * QS_STRIDE + ks * 16 + colh));
    m_run[0] = m_run[1] = -INFINITY;
    l_run[0] = l_run[1] = 0.f;
#pragma unroll
    for (int i = 0; i < D / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
  }
  __device__ __forceinline__ void reduce_sums() {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      l_run[r] += __shfl_xor_sync(0xffffffffu, l_run[r], 1);
      l_run[r] += __shfl_xor_sync(0xffffffffu, l_run[r], 2);
    }
  }
  // mo [warp][16][D], mml [warp][16][2]
  __device__ __forceinline__ void put(float* mo, float* mml, int warp, int lane) const {
    const int g4 = lane >> 2, t4 = lane & 3;
#pragma unroll
    for (int i = 0; i < D / 8; ++i) {
      float* r0 = mo + (warp * 16 + g4) * D + i * 8 + 2 * t4;
      float* r1 = r0 + 8 * D;
      r0[0] = o[i][0]; r0[1] = o[i][1];
      r1[0] = o[i][2]; r1[1] = o[i][3];
    }
    if (t4 == 0) {
      mml[(warp * 16 + g4) * 2 + 0] = m_run[0];
      mml[(warp * 16 + g4) * 2 + 1] = l_run[0];
      mml[(warp * 16 + g4 + 8) * 2 + 0] = m_run[1];
      mml[(warp * 16 + g4 + 8) * 2 + 1] = l_run[1];
    }
  }
};
// Columns d .. d + 3 of query row r over the four warps: unnormalised sums, the row's maximum and its sum.
template <int D>
__device__ __forceinline__ float4 combine_warps(const float* mo, const float* mml, int r, int d, float* mstar_out, float* l_out) {
  float mstar = -INFINITY;
#pragma unroll
  for (int w = 0; w < ATT_CWARPS; ++w) mstar = fmaxf(mstar, mml[(w * 16 + r) * 2]);
  const float muse = (mstar == -INFINITY) ? 0.f : mstar;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  float L = 0.f;
#pragma unroll
  for (int w = 0; w < ATT_CWARPS; ++w) {
    const float wgt = exp2f(mml[(w * 16 + r) * 2] - muse);
    const float4 v = *reinterpret_cast<const float4*>(mo + (w * 16 + r) * D + d);
    acc.x = fmaf(v.x, wgt, acc.x); acc.y = fmaf(v.y, wgt, acc.y);
    acc.z = fmaf(v.z, wgt, acc.z); acc.w = fmaf(v.w, wgt, acc.w);
    L = fmaf(mml[(w * 16 + r) * 2 + 1], wgt, L);
  }
  *mstar_out = mstar;
  *l_out = L;
  return acc;
}
// The warp's 16 positions of a tile (K at kb, V at vb, in shared memory), positions my_pos0 on.
template <int D>
__device__ __forceinline__ void attn_tile(const AttnParams& p, AttnState<D>& st, uint8_t* kb, uint8_t* vb, int warp, int lane, int my_pos0,
                                          int len_eff, bool owns_new, int pos_new, const __half* new_k, const __half* new_v) {
  constexpr int KSTEPS = D / 16;
  const int t4 = lane & 3;
  uint32_t (&qa)[D / 16][4] = st.qa;
  float (&m_run)[2] = st.m_run;
  float (&l_run)[2] = st.l_run;
  float (&o)[D / 8][4] = st.o;
  // patch the appended row / clear rows past the end (only this warp reads its 16 rows)
  if (my_pos0 + 16 > len_eff || (owns_new && pos_new >= my_pos0 && pos_new < my_pos0 + 16)) {
    for (int i = lane; i < 16 * (D / 8); i += 32) {
      const int r = i / (D / 8), c = i - r * (D / 8);
      if (my_pos0 + r >= len_eff) *reinterpret_cast<uint4*>(vb + (c >> 3) * ATT_BOX_BYTES + swz128(16 * warp + r, c & 7)) = make_uint4(0, 0, 0, 0);
    }
    if (owns_new && pos_new >= my_pos0 && pos_new < my_pos0 + 16 && lane < 2 * (D / 8)) {
      const bool is_v = lane >= D / 8;
      const int c = is_v ? lane - D / 8 : lane;
      const uint4 val = *reinterpret_cast<const uint4*>((is_v ? new_v : new_k) + c * 8);
      *reinterpret_cast<uint4*>((is_v ? vb : kb) + (c >> 3) * ATT_BOX_BYTES + swz128(16 * warp + pos_new - my_pos0, c & 7)) = val;
    }
    fence_proxy_async_smem();   // the next tile's loads write here
    __syncwarp();
  }

  // ---- S = Q K^T for 16 positions.  A warp's instructions issue in order and an MMA waits for the one whose sums it
  // adds to: four chains side by side, and below the high parts before the low.  (A step of the 0.5B shape at batch 1 518 -> 499 us,
  // at batch 64 and 1500 positions 1285 -> 1228; with at most 128 registers, so that three CTAs of head dimension 64 fit an SM,
  // batch 16 at 1500 positions gains 3 % and batch 64 loses 4.)
  float s[2][4];
  {
    float part[2][2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j) part[i][j][0] = part[i][j][1] = part[i][j][2] = part[i][j][3] = 0.f;
    const uint32_t row = 16 * warp + (lane & 7) + 8 * (lane >> 4);
    const int ch = (lane >> 3) & 1;
    const uint32_t k0 = smem_u32(kb);
#pragma unroll
    for (int ks0 = 0; ks0 < KSTEPS; ks0 += 2) {
      uint32_t r[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int chunk = (ks0 + i) * 2 + ch;
        ldmatrix_x4(r[i][0], r[i][1], r[i][2], r[i][3], k0 + (chunk >> 3) * ATT_BOX_BYTES + swz128(row, chunk & 7));
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        mma_f16_16816(part[i][0], qa[ks0 + i], r[i][0], r[i][1]);
        mma_f16_16816(part[i][1], qa[ks0 + i], r[i][2], r[i][3]);
      }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int x = 0; x < 4; ++x) s[i][x] = part[0][i][x] + part[1][i][x];
  }
  // ---- mask, scale, online softmax
  float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
  for (int nt = 0; nt < 2; ++nt)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      int pos = my_pos0 + nt * 8 + 2 * t4 + (j & 1);
      float v = (pos < len_eff) ? s[nt][j] * p.scale_log2 : -INFINITY;
      s[nt][j] = v;
      mx[j >> 1] = fmaxf(mx[j >> 1], v);
    }
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
    mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
  }
  float corr[2], m_use[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    float m_new = fmaxf(m_run[r], mx[r]);
    m_use[r] = (m_new == -INFINITY) ? 0.f : m_new;
    corr[r] = exp2f(m_run[r] - m_use[r]);
    m_run[r] = m_new;
  }
  float pr[2][4];
  float psum[2] = {0.f, 0.f};
#pragma unroll
  for (int nt = 0; nt < 2; ++nt)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float e = exp2f(s[nt][j] - m_use[j >> 1]);
      pr[nt][j] = e;
      psum[j >> 1] += e;
    }
#pragma unroll
  for (int r = 0; r < 2; ++r) l_run[r] = l_run[r] * corr[r] + psum[r];
#pragma unroll
  for (int i = 0; i < D / 8; ++i) {
    o[i][0] *= corr[0]; o[i][1] *= corr[0];
    o[i][2] *= corr[1]; o[i][3] *= corr[1];
  }
  // ---- P as fp16 high part + fp16 residual
  uint32_t a_hi[4], a_lo[4];
  {
    const float (*q)[4] = pr;
    float h[8] = {q[0][0], q[0][1], q[0][2], q[0][3], q[1][0], q[1][1], q[1][2], q[1][3]};
    float lo[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float hi = __half2float(__float2half_rn(h[i]));
      lo[i] = h[i] - hi;
    }
    a_hi[0] = pack_half2(h[0], h[1]); a_hi[1] = pack_half2(h[2], h[3]);
    a_hi[2] = pack_half2(h[4], h[5]); a_hi[3] = pack_half2(h[6], h[7]);
    a_lo[0] = pack_half2(lo[0], lo[1]); a_lo[1] = pack_half2(lo[2], lo[3]);
    a_lo[2] = pack_half2(lo[4], lo[5]); a_lo[3] = pack_half2(lo[6], lo[7]);
  }
  // ---- O += P V
  {
    const uint32_t row = 16 * warp + (lane & 7) + 8 * ((lane >> 3) & 1);
    const int ch = lane >> 4;
    const uint32_t v0 = smem_u32(vb);
#pragma unroll
    for (int dn = 0; dn < D / 16; dn += 2) {
      uint32_t r[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int chunk = (dn + i) * 2 + ch;
        ldmatrix_x4_trans(r[i][0], r[i][1], r[i][2], r[i][3], v0 + (chunk >> 3) * ATT_BOX_BYTES + swz128(row, chunk & 7));
      }
#pragma unroll
      for (int l = 0; l < 2; ++l)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          mma_f16_16816(o[2 * (dn + i)], l ? a_lo : a_hi, r[i][0], r[i][1]);
          mma_f16_16816(o[2 * (dn + i) + 1], l ? a_lo : a_hi, r[i][2], r[i][3]);
        }
    }
  }
}

// Dynamic shared memory of a CTA: the ring, the staged query, the appended rows and the warps' (max, sum), what other CTAs
// push, the barriers.
template <int D>
struct AttnSmem {
  static constexpr int QS_STRIDE = D + 8;  // halfs; +16 bytes keeps ldmatrix rows on distinct banks
  static constexpr int STAGE_BYTES = 2 * (D / 64) * ATT_BOX_BYTES;
  static constexpr int STAGES = D == 64 ? 4 : 3;
  static constexpr int PUSHED_ROWS = ATT_PUSHED_ROWS;
  static constexpr int ROW_BYTES = (D + 4) * 4;                  // sums, maximum, sum of weights, padding
  static constexpr int WORK = (16 * QS_STRIDE * 2 + 2 * D * 2 + ATT_CWARPS * 16 * 2 * 4 + 15) / 16 * 16;
  static constexpr int BYTES = STAGES * STAGE_BYTES + WORK + PUSHED_ROWS * ROW_BYTES + (2 * STAGES + 2) * 8;
};
static_assert(2 * (AttnSmem<128>::BYTES + 1024) <= 228 * 1024, "two CTAs fit an SM");

// Grid: (sequence, KV head) pairs x CTAs of a cluster, up to MAX_PARTS.
template <int D, int MAX_PARTS>
__global__ void __launch_bounds__(ATT_THREADS, 2)
gqa_decode_attn_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const AttnParams p) {
  using Smem = AttnSmem<D>;
  static_assert(Smem::STAGE_BYTES >= ATT_CWARPS * 16 * D * 4, "a ring stage doubles as the scratch that combines the warps");
  constexpr int STAGES = Smem::STAGES, NBOX = D / 64, STAGE_BYTES = Smem::STAGE_BYTES, ROW_BYTES = Smem::ROW_BYTES;
  extern __shared__ __align__(1024) uint8_t attn_smem[];   // TMA's swizzle counts from multiples of 1024
  uint8_t* stages = attn_smem;
  __half* qs = reinterpret_cast<__half*>(stages + STAGES * STAGE_BYTES);
  __half* new_k = qs + 16 * AttnSmem<D>::QS_STRIDE;
  __half* new_v = new_k + D;
  float* mml = reinterpret_cast<float*>(new_v + D);
  uint8_t* pushed = reinterpret_cast<uint8_t*>(qs) + Smem::WORK;      // [part][row slot] of the rows finished here
  uint64_t* bar_full = reinterpret_cast<uint64_t*>(pushed + Smem::PUSHED_ROWS * ROW_BYTES);
  uint64_t* bar_empty = bar_full + STAGES;
  uint64_t* bar_parts = bar_empty + STAGES;
  int& s_bump = *reinterpret_cast<int*>(bar_parts + 1);

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int G = p.h_q / p.h_kv;
  const int ranks = p.ranks, rank = (int)(blockIdx.x % (unsigned)ranks), pair = (int)(blockIdx.x / (unsigned)ranks);
  const int b = pair / p.h_kv, kvh = pair - b * p.h_kv;

  // In a decode step the lengths and the cached rows are older than the step, so reading them and loading the first tiles
  // overlap the predecessor's end, and only what reads the query and the new K/V rows waits.  Elsewhere the predecessor may
  // write any of them: everything waits.
  if (!p.early_reads) pdl_wait();
  // a kernel that gave up earlier left a code behind: do not start new work on top of it
  // (the CTA takes one decision: a code that any of its threads has read)
  const int status = *reinterpret_cast<volatile int*>(p.status);
  const int len = __ldcg(p.seq_len + b);
  const int len0 = len < p.l_max ? len : p.l_max, len_eff = attn_len_eff(p, len0);
  const int tiles = (len_eff + ATT_TILE - 1) / ATT_TILE;
  const int parts = tiles >= p.all_from ? ranks : min(p.few, tiles);   // CTAs with tiles
  const int t0 = rank < parts ? rank * tiles / parts : 0, t1 = rank < parts ? (rank + 1) * tiles / parts : 0;
  const int per = parts > 0 ? (G + parts - 1) / parts : G;   // row slots a part
  const int mine = rank < parts ? (G - rank + parts - 1) / parts : 0;   // rows finished here: rank, rank + parts, ...
  if (tid == 0) {
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(&bar_full[i], 1);
      mbar_init(&bar_empty[i], ATT_CWARPS);
    }
    mbar_init(bar_parts, 1);
    fence_barrier_init();
    mbar_arrive_expect_tx(bar_parts, (parts > 1 ? parts - 1 : 0) * mine * (D * 4 + 8));
  }
  const bool prior = __syncthreads_or(status != 0);
  cg::cluster_group cluster = cg::this_cluster();
  cluster.barrier_arrive();   // "this CTA runs, its barrier stands": before anyone pushes into it
  const int64_t row_base = ((int64_t)b * p.h_kv + kvh) * p.l_max;

  // the last CTA of the grid to have its length advances the lengths (before the producer starts: it may wait for the consumers),
  // unless there is a code: nothing is appended then
  if (p.bump && !prior) {
    pdl_wait();
    if (tid == 0) s_bump = arrive_inc(p.arrive, gridDim.x - 1) == gridDim.x - 1;
    __syncthreads();
    if (s_bump)
      for (int i = tid; i < p.b; i += ATT_THREADS) {
        const int l = __ldcg(p.seq_len + i);
        if (l < p.l_max) p.seq_len[i] = l + 1;
      }
  }
  // The last loads of tiles [t0, t): this CTA's shared memory is its own until they have landed.
  auto drain = [&](int t) {
    for (int i = max(0, t - t0 - STAGES); i < t - t0; ++i) mbar_wait(&bar_full[i % STAGES], (i / STAGES) & 1);
  };
  if (warp == ATT_CWARPS) {
    // ---------------------------------------------------------------- producer
    if (lane == 0 && !prior) {
      for (int t = t0; t < t1; ++t) {
        const int i = t - t0, st = i % STAGES;
        if (!mbar_wait(&bar_empty[st], ((i / STAGES) & 1) ^ 1)) {
          atomicExch(p.status, 101);
          drain(t);
          break;
        }
        uint8_t* sb = stages + st * STAGE_BYTES;
        mbar_arrive_expect_tx(&bar_full[st], STAGE_BYTES);
        const int y = (int)(row_base + (int64_t)t * ATT_TILE);
#pragma unroll
        for (int j = 0; j < NBOX; ++j) {
          tma_load_2d(sb + j * ATT_BOX_BYTES, &map_k, &bar_full[st], j * 64, y);
          tma_load_2d(sb + (NBOX + j) * ATT_BOX_BYTES, &map_v, &bar_full[st], j * 64, y);
        }
      }
    }
  }
  pdl_wait();
  pdl_trigger();
  if (warp == ATT_CWARPS) return;
  if (tiles == 0) {   // nothing to attend to: zeros
    if (rank == 0 && !prior)
      for (int e = tid; e < G * D; e += ATT_CTHREADS) store_out(p, ((int64_t)b * p.h_q + kvh * G) * D + e, 0.f);
    return;
  }
  if (rank >= parts) return;

  // ---------------------------------------------------------------- consumers
  // Whatever happens, a CTA pushes what its peers count on and takes what they push: nothing arrives in the memory of one
  // that has left.  Without sums (a code was there, or a wait gave up) it pushes a mark in place of a row's sum of
  // weights, which is never negative, and a row with a mark is not written.
  constexpr float NO_SUMS = -1.f;
  // Everything that peers push here has arrived.  Otherwise a peer is late (each of its waits is bounded): once the others have ended
  // or are here too, what is still on its way arrives at once.
  auto all_pushed = [&]() {
    if (mbar_wait_cluster(bar_parts, 0)) return true;
    atomicCAS(p.status, 0, 103);
    cluster_meet();
    mbar_wait_cluster(bar_parts, 0);
    return false;
  };
  if (!prior) {
    const int pos_new = len0;
    const bool owns_new = p.fused && len0 < p.l_max && pos_new >= t0 * ATT_TILE && pos_new < t1 * ATT_TILE;
    stage_query<D>(p, b, kvh, len0, owns_new, row_base, tid, qs, new_k, new_v);
    asm volatile("bar.sync 1, %0;" ::"n"(ATT_CTHREADS) : "memory");
    AttnState<D> w;
    w.start(qs, lane);
    bool ok = true;
    int st = 0;
    for (int t = t0; t < t1; ++t) {
      const int i = t - t0;
      st = i % STAGES;
      if (!mbar_wait(&bar_full[st], (i / STAGES) & 1)) {
        ok = false;
        break;
      }
      uint8_t* kb = stages + st * STAGE_BYTES;
      attn_tile<D>(p, w, kb, kb + NBOX * ATT_BOX_BYTES, warp, lane, t * ATT_TILE + 16 * warp, len_eff, owns_new, pos_new, new_k, new_v);
      __syncwarp();
      if (t + 1 < t1 && lane == 0) mbar_arrive(&bar_empty[st]);
    }
    w.reduce_sums();
    int all_ok;
    asm volatile(
        "{\n\t.reg .pred q, r;\n\tsetp.ne.u32 q, %1, 0;\n\tbar.red.and.pred r, 1, %2, q;\n\tselp.u32 %0, 1, 0, r;\n\t}"
        : "=r"(all_ok)
        : "r"((uint32_t)ok), "n"(ATT_CTHREADS)
        : "memory");
    if (all_ok) {
      float* mo = reinterpret_cast<float*>(stages + st * STAGE_BYTES);   // [warp][16][D]: every warp has read its rows of the last tile
      w.put(mo, mml, warp, lane);
      asm volatile("bar.sync 1, %0;" ::"n"(ATT_CTHREADS) : "memory");
      if (parts > 1) cluster.barrier_wait();
      const int64_t o0 = ((int64_t)b * p.h_q + kvh * G) * D;
      for (int e = 4 * tid; e < G * D; e += 4 * ATT_CTHREADS) {
        const int r = e / D, d = e - r * D;
        float m, L;
        const float4 acc = combine_warps<D>(mo, mml, r, d, &m, &L);
        if (parts == 1) {
          store_out4(p, o0 + e, acc, L);
          continue;
        }
        const int to = r % parts;
        const uint32_t at = smem_u32(pushed) + (rank * per + r / parts) * ROW_BYTES;
        if (to == rank) {
          *reinterpret_cast<float4*>(pushed + (rank * per + r / parts) * ROW_BYTES + d * 4) = acc;
          if (d == 0) *reinterpret_cast<float2*>(pushed + (rank * per + r / parts) * ROW_BYTES + D * 4) = make_float2(m, L);
        } else {
          const uint32_t there = smem_of_rank(at, to), bar = smem_of_rank(smem_u32(bar_parts), to);
          push16(there + d * 4, acc, bar);
          if (d == 0) push8(there + D * 4, make_float2(m, L), bar);
        }
      }
      if (parts == 1) return;
      asm volatile("bar.sync 1, %0;" ::"n"(ATT_CTHREADS) : "memory");
      if (!all_pushed()) return;
      // the rows finished here, the parts in the order of their positions
      for (int e = 4 * tid; e < mine * D; e += 4 * ATT_CTHREADS) {
        const int slot = e / D, d = e - slot * D;
        const uint8_t* row = pushed + slot * ROW_BYTES;
        constexpr int SOME = 8;   // parts whose maxima and sums are in registers
        const auto of_part = [&](int i) { return *reinterpret_cast<const float2*>(row + i * per * ROW_BYTES + D * 4); };
        float2 ml[SOME];
        float m = -INFINITY;
        bool whole = true;
#pragma unroll
        for (int i = 0; i < SOME; ++i) {
          ml[i] = i < parts ? of_part(i) : make_float2(-INFINITY, 0.f);
          m = fmaxf(m, ml[i].x);
          whole = whole && ml[i].y != NO_SUMS;
        }
        if constexpr (MAX_PARTS > SOME)
#pragma unroll 1
          for (int i = SOME; i < parts; ++i) {
            m = fmaxf(m, of_part(i).x);
            whole = whole && of_part(i).y != NO_SUMS;
          }
        if (!whole) continue;
        const float muse = (m == -INFINITY) ? 0.f : m;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        float L = 0.f;
        const auto add = [&](int i, float2 of) {
          const float wgt = exp2f(of.x - muse);
          const float4 v = *reinterpret_cast<const float4*>(row + i * per * ROW_BYTES + d * 4);
          acc.x = fmaf(v.x, wgt, acc.x); acc.y = fmaf(v.y, wgt, acc.y);
          acc.z = fmaf(v.z, wgt, acc.z); acc.w = fmaf(v.w, wgt, acc.w);
          L = fmaf(of.y, wgt, L);
        };
#pragma unroll
        for (int i = 0; i < SOME; ++i)
          if (i < parts) add(i, ml[i]);
        if constexpr (MAX_PARTS > SOME)
#pragma unroll 1
          for (int i = SOME; i < parts; ++i) add(i, of_part(i));
        store_out4(p, o0 + (int64_t)(rank + slot * parts) * D + d, acc, L);
      }
      return;
    }
    if (!ok && lane == 0) atomicExch(p.status, 102);
    if (tid == 0) drain(t1);   // the producer may be done and gone (one that is not drains what it has issued)
  }
  if (parts == 1) return;
  cluster.barrier_wait();
  for (int e = 4 * tid; e < G * D; e += 4 * ATT_CTHREADS) {
    const int r = e / D, d = e - r * D, to = r % parts;
    if (to == rank) continue;
    const uint32_t there = smem_of_rank(smem_u32(pushed) + (rank * per + r / parts) * ROW_BYTES, to), bar = smem_of_rank(smem_u32(bar_parts), to);
    push16(there + d * 4, make_float4(0.f, 0.f, 0.f, 0.f), bar);
    if (d == 0) push8(there + D * 4, make_float2(0.f, NO_SUMS), bar);
  }
  all_pushed();
}

__global__ void bump_seq_len_kernel(int32_t* seq_len, int b, int l_max) {
  pdl_wait();
  pdl_trigger();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < b && seq_len[i] < l_max) seq_len[i] += 1;
}

// Stand-alone append (no attention): one CTA per (sequence, KV head).
__global__ void kv_append_rope_kernel(__half* k_cache, __half* v_cache, const __half* k_new, const __half* v_new,
                                      const float* rope, const int32_t* seq_len, int h_kv, int d, int l_max) {
  const int kvh = blockIdx.x, b = blockIdx.y;
  const int pos = seq_len[b];
  if (pos < 0 || pos >= l_max) return;
  const int half_d = d / 2;
  const float* tab = rope + (int64_t)pos * half_d * 2;
  const __half* kp = k_new + ((int64_t)b * h_kv + kvh) * d;
  const __half* vp = v_new + ((int64_t)b * h_kv + kvh) * d;
  __half* kd = k_cache + (((int64_t)b * h_kv + kvh) * l_max + pos) * d;
  __half* vd = v_cache + (((int64_t)b * h_kv + kvh) * l_max + pos) * d;
  for (int e = threadIdx.x; e < half_d; e += blockDim.x) {
    float k1 = __half2float(kp[e]), k2 = __half2float(kp[e + half_d]);
    float c = tab[2 * e], s = tab[2 * e + 1];
    kd[e] = __float2half_rn(__fsub_rn(__fmul_rn(k1, c), __fmul_rn(k2, s)));
    kd[e + half_d] = __float2half_rn(__fadd_rn(__fmul_rn(k2, c), __fmul_rn(k1, s)));
    vd[e] = vp[e];
    vd[e + half_d] = vp[e + half_d];
  }
}

// Clusters of 1 to 16 CTAs that run at once, with two CTAs an SM and with one.  A cluster lies within a GPC, so that is fewer than
// the SMs would hold: of 8 CTAs 33 and 15 on a B200, of 7 37 and 15, of 16 14 and 7.
struct ClusterRoom {
  int two[ATT_WIDE + 1] = {}, one[ATT_WIDE + 1] = {};
};
constexpr int ATT_ONE_AN_SM = 115 * 1024;   // bytes of shared memory of which an SM has no two

template <int D>
logos_status_t cluster_room(int device, const ClusterRoom** out) {
  static std::mutex mu;
  static std::unordered_map<int, ClusterRoom> rooms;
  std::lock_guard<std::mutex> lk(mu);
  auto it = rooms.find(device);
  if (it == rooms.end()) {
    // a size that the device or the driver does not take has no room; one CTA always has
    ClusterRoom room;
    const int most = cudaFuncSetAttribute(gqa_decode_attn_kernel<D, ATT_WIDE>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess ? ATT_WIDE : 8;
    for (int r = 1; r <= most; ++r) {
      auto kernel = r <= 8 ? gqa_decode_attn_kernel<D, 8> : gqa_decode_attn_kernel<D, ATT_WIDE>;
      LOGOS_TRY(allow_smem(reinterpret_cast<const void*>(kernel), device, std::max(AttnSmem<D>::BYTES, ATT_ONE_AN_SM)));
      for (int* fit : {&room.two[r], &room.one[r]}) {
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = (unsigned)r;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)r);
        cfg.blockDim = dim3(ATT_THREADS);
        cfg.dynamicSmemBytes = (size_t)(fit == &room.two[r] ? AttnSmem<D>::BYTES : ATT_ONE_AN_SM);
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(fit, kernel, &cfg) != cudaSuccess) *fit = 0;
      }
    }
    cudaGetLastError();
    room.two[1] = std::max(room.two[1], 1);
    room.one[1] = std::max(room.one[1], 1);
    it = rooms.emplace(device, room).first;
  }
  *out = &it->second;
  return LOGOS_OK;
}

// How the pairs' tiles are cut.
struct AttnCut {
  int ranks = 1, few = 1, all_from = INT_MAX;   // see AttnParams
  bool one_an_sm = false;
};

// What bounds a cut is its rounds: a cluster that does not run at once waits for one that does, and a last round of few clusters
// takes nearly as long as a full one (0.9 of it, from 34 to 128 pairs of 32768).  So: rounds x (tiles of a part + 16, for what a round
// has besides: start, ramp, exchange).  In a decode step the neighbouring kernels have CTAs on the SMs too, and a round that
// needs nearly all of them waits: 32 pairs in clusters of 8, of which 33 fit, 1187 us a step of the 32B shape, of 7 1149.
// The rule before took 2 x SMs / pairs CTAs without a look at what fits, and so two rounds for 16 pairs (8 x 16 with
// one CTA an SM: 15 clusters fit) or 38 (7 x 38: 37 fit).  That one -> this one, us:
//   28/4 heads of 128, 4 x 32768 101 -> 67; 64/8, 38 x 4096 148 -> 134; 14/2 of 64, 7 ragged ones up to 131072 121 -> 85;
//   a step of the 0.5B shape at batch 8 and 450 positions 638 -> 564, 9 and 1500 771 -> 689, 24 and 128 921 -> 829; of the 32B shape
//   (8 layers) at batch 2 and 2000 1294 -> 1255.
AttnCut attn_cut(int64_t pairs, int64_t tiles_max, int group, int d, bool in_step, const ClusterRoom& room) {
  AttnCut c;
  // In a step, short sequences at head dimension 64 get parts of two tiles at least: a tile takes 0.4 us there, no more than what a
  // part costs the chain.  A step of the 0.5B shape at batch 16 and 128 positions 678 -> 663 us, 600 708 -> 696, batch 12 and 350 672 -> 663,
  // 24 and 128 827 -> 816.  With fewer pairs the SMs are idle anyway (batch 1 at 260 469 -> 481), with more they are full
  // of one tile's parts too (batch 48 at 350 1001 -> 1015).
  const bool pays = !in_step || d != 64 || pairs < 8 || pairs > 56 || tiles_max >= 12;
  // More than eight CTAs, which are not portable, only where sequences can be long: such clusters start later (8/1 heads, 8 x 3000
  // in a cache of 131073 17.8 -> 21 us; 8 x 131072 162 -> 99).  They are used from four tiles a CTA on.  In a step only the largest:
  // 12 layers of the 0.5B shape in a cache of 33000, batch 4 at 3000 / 30000 positions 284 / 540 -> 293 / 453 us, but by clusters of 13
  // batch 7 298 / 560 -> 312 / 523.
  const int64_t most = pays ? std::min<int64_t>(tiles_max, tiles_max >= 512 ? ATT_WIDE : 8) : std::max<int64_t>(1, tiles_max / 2);
  // More pairs than run at once: parts shorten the last round, but want 16 tiles each, in the sequence at hand too.
  const bool many = pairs > room.two[1];
  double best = 0.;
  for (int r = 1; r <= most; ++r) {
    if (room.two[r] < 1 || (in_step && r > 8 && r < ATT_WIDE) || r * ((group + r - 1) / r) > ATT_PUSHED_ROWS || (many && r > 1 && tiles_max < 16 * r)) continue;
    const int64_t full = pairs / room.two[r], rest = pairs % room.two[r];
    double rounds = (double)full + (rest ? std::max(0.9, (double)rest / room.two[r]) : 0.);
    if (in_step && rounds > 0.93 && rounds <= 1.) rounds = 1.1;
    const double cost = rounds * (double)((tiles_max + r - 1) / r + 16);
    if (best > 0. && cost > best) continue;
    best = cost;
    c.ranks = r;
  }
  c.few = many ? 1 : std::min(c.ranks, 8);
  if (c.ranks > c.few) c.all_from = (many ? 16 : 4) * c.ranks;
  // Where all clusters run at once with a CTA an SM, a CTA asks for more than half of an SM's shared memory: a cluster's CTAs are packed
  // onto an SM otherwise.  A step of the 0.5B shape, batch 16 at 128 positions (96 CTAs) 748 -> 685 us; with more CTAs than
  // that it only keeps them and the neighbouring kernels' CTAs apart: batch 16 at 1500 positions (256 CTAs) 769 -> 963.
  c.one_an_sm = pairs <= room.one[c.ranks];
  return c;
}

template <int D>
logos_status_t launch_attn_t(const AttnArgs& a, cudaStream_t st) {
  if (a.b > ATT_MAX_BATCH)
    return fail(LOGOS_OUT_OF_BOUNDS, "attention: batch %lld exceeds %d sequences per call", (long long)a.b, ATT_MAX_BATCH);
  const int64_t rows_total = a.b * a.h_kv * a.l_max;
  CUtensorMap mk, mv;
  LOGOS_TRY(cached_map(&mk, a.k_cache, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, D, rows_total, D * 2, 64, ATT_TILE));
  LOGOS_TRY(cached_map(&mv, a.v_cache, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, D, rows_total, D * 2, 64, ATT_TILE));
  AttnParams p{};
  p.q_f16 = a.q_f16; p.q_f32 = a.q_f32; p.q_ld = a.q_ld; p.rotate_q = a.rotate_q;
  p.k_new_f16 = a.k_new_f16; p.v_new_f16 = a.v_new_f16; p.k_new_f32 = a.k_new_f32; p.v_new_f32 = a.v_new_f32;
  p.kv_ld = a.kv_ld;
  p.f32_parts = a.f32_parts > 1 ? a.f32_parts : 1;
  p.f32_part_stride = a.f32_part_stride;
  p.q_bias = a.q_bias; p.k_bias = a.k_bias; p.v_bias = a.v_bias;
  p.fused = (a.k_new_f16 || a.k_new_f32) ? 1 : 0;
  p.k_cache = a.k_cache; p.v_cache = a.v_cache; p.rope = a.rope; p.seq_len = a.seq_len;
  p.bump = a.bump_seq_len;
  if (p.bump) {
    void* arrive = nullptr;
    LOGOS_TRY(counters_get(a.device, ATT_COUNTER_BYTES, &arrive));
    p.arrive = reinterpret_cast<unsigned*>(arrive);
  }
  p.early_reads = a.early_reads;
  p.o = a.o; p.o_dtype = a.o_dtype; p.o_act = a.o_act;
  p.b = (int)a.b; p.h_q = (int)a.h_q; p.h_kv = (int)a.h_kv; p.l_max = (int)a.l_max;
  p.scale_log2 = a.scale * 1.4426950408889634f;
  p.status = a.ext_status ? a.ext_status : kernel_status_ptr(a.device);
  if (!p.status) return fail(LOGOS_ERROR, "attention: no kernel status word");

  const ClusterRoom* room = nullptr;
  LOGOS_TRY(cluster_room<D>(a.device, &room));
  const int64_t pairs = a.b * a.h_kv;
  const AttnCut cut = attn_cut(pairs, (a.l_max + ATT_TILE - 1) / ATT_TILE, (int)(a.h_q / a.h_kv), D, a.early_reads, *room);
  auto kernel = cut.ranks <= 8 ? gqa_decode_attn_kernel<D, 8> : gqa_decode_attn_kernel<D, ATT_WIDE>;
  p.ranks = cut.ranks; p.few = cut.few; p.all_from = cut.all_from;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(pairs * cut.ranks));
  cfg.blockDim = dim3(ATT_THREADS);
  cfg.dynamicSmemBytes = (size_t)(cut.one_an_sm ? std::max(AttnSmem<D>::BYTES, ATT_ONE_AN_SM) : AttnSmem<D>::BYTES);
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)p.ranks;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_active() ? 2 : 1;
  LOGOS_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, mk, mv, p));
  count_launch(LK_ATTN);
  return check_launch("gqa_decode_attn_kernel");
}

}  // namespace

void rope_table_host(float* out, int64_t l_max, int64_t d, double theta) {
  int64_t half = d / 2;
  for (int64_t pos = 0; pos < l_max; ++pos)
    for (int64_t i = 0; i < half; ++i) {
      double inv = pow(theta, -2.0 * (double)i / (double)d);
      double ang = (double)pos * inv;
      out[(pos * half + i) * 2 + 0] = (float)cos(ang);
      out[(pos * half + i) * 2 + 1] = (float)sin(ang);
    }
}

logos_status_t launch_gqa_decode_attn(const AttnArgs& a, cudaStream_t st) {
  if (a.b == 0 || a.h_q == 0) return LOGOS_OK;
  if (a.h_kv <= 0 || a.h_q % a.h_kv) return fail(LOGOS_ERROR, "attention: h_q must be a multiple of h_kv");
  if (a.h_q / a.h_kv > 16) return fail(LOGOS_ERROR, "attention: at most 16 query heads per KV head");
  if (a.l_max <= 0) return fail(LOGOS_OUT_OF_BOUNDS, "attention: l_max must be positive");
  if (a.d == 128) return launch_attn_t<128>(a, st);
  if (a.d == 64) return launch_attn_t<64>(a, st);
  return fail(LOGOS_ERROR, "attention: head_dim %lld is not supported (64 or 128)", (long long)a.d);
}

logos_status_t launch_kv_append_rope(__half* k_cache, __half* v_cache, const __half* k_new, const __half* v_new,
                                     const float* rope, int32_t* seq_len, int64_t b, int64_t h_kv, int64_t d,
                                     int64_t l_max, int device, cudaStream_t st) {
  (void)device;
  if (b == 0 || h_kv == 0) return LOGOS_OK;
  dim3 grid((unsigned)h_kv, (unsigned)b);
  kv_append_rope_kernel<<<grid, 64, 0, st>>>(k_cache, v_cache, k_new, v_new, rope, seq_len, (int)h_kv, (int)d, (int)l_max);
  LOGOS_TRY(check_launch("kv_append_rope_kernel"));
  bump_seq_len_kernel<<<(unsigned)((b + 127) / 128), 128, 0, st>>>(seq_len, (int)b, (int)l_max);
  return check_launch("bump_seq_len_kernel");
}

// ---------------------------------------------------------------- the entry point that allocates nothing
// Its status word lives in the library image instead of coming from cudaMalloc; the kernel keeps nothing else in global memory.
static __device__ __align__(256) int g_static_attn_status[8];

namespace {
constexpr int kMaxStaticDevices = 64;
int* g_static_addr[kMaxStaticDevices];
std::mutex g_static_mu;

// In host code the array name above is a host-side stand-in, not a device address: the
// address a kernel may use comes from cudaGetSymbolAddress, asked once per device with
// that device current.
logos_status_t static_status_for(int device, int** out) {
  if (device < 0 || device >= kMaxStaticDevices)
    return fail(LOGOS_OUT_OF_BOUNDS, "fixed-scratch attention: device %d is beyond the %d this build tracks", device,
                kMaxStaticDevices);
  std::lock_guard<std::mutex> lk(g_static_mu);
  if (!g_static_addr[device]) {
    void* q = nullptr;
    LOGOS_CUDA_TRY(cudaGetSymbolAddress(&q, g_static_attn_status));
    g_static_addr[device] = static_cast<int*>(q);
  }
  *out = g_static_addr[device];
  return LOGOS_OK;
}
}  // namespace

// The fixed-scratch entry point's own status word, for logos_kernel_status: copies the eight
// words out (and zeroes them when asked) if that entry point has run on `device`; *used tells
// whether it has.  A device-to-host copy of eight words: no allocation here either.
logos_status_t static_attn_status_read(int device, int words_out[8], bool clear, bool* used) {
  *used = false;
  if (device < 0 || device >= kMaxStaticDevices) return LOGOS_OK;
  int* status;
  {
    std::lock_guard<std::mutex> lk(g_static_mu);
    status = g_static_addr[device];
  }
  if (!status) return LOGOS_OK;
  LOGOS_CUDA_TRY(cudaSetDevice(device));
  LOGOS_CUDA_TRY(cudaMemcpy(words_out, status, sizeof(int) * 8, cudaMemcpyDeviceToHost));
  if (clear && words_out[0] != 0) LOGOS_CUDA_TRY(cudaMemset(status, 0, sizeof(int) * 8));
  *used = true;
  return LOGOS_OK;
}

}  // namespace logos

using namespace logos;

extern "C" {

logos_status_t logos_gqa_decode_attn_fixed_scratch(logos_handle_t q, logos_handle_t k_cache, logos_handle_t v_cache,
                                                   logos_handle_t seq_len, logos_handle_t o, int64_t b, int64_t h_q,
                                                   int64_t h_kv, int64_t d, int64_t l_max, float softmax_scale,
                                                   void* stream_or_null) {
  return guarded([&]() -> logos_status_t {
    if (b < 0 || h_q < 0 || h_kv <= 0 || d <= 0 || l_max <= 0)
      return fail(LOGOS_OUT_OF_BOUNDS, "logos_gqa_decode_attn_fixed_scratch: bad extents");
    AttnArgs a;
    __half *qp, *kc, *vc, *op;
    int32_t* sl;
    int32_t dev = 0;
    LOGOS_TRY(buf_ptr<__half>(q, b * h_q * d, "q", &qp, &dev));
    LOGOS_TRY(buf_ptr<__half>(k_cache, b * h_kv * l_max * d, "k_cache", &kc));
    LOGOS_TRY(buf_ptr<__half>(v_cache, b * h_kv * l_max * d, "v_cache", &vc));
    LOGOS_TRY(buf_ptr<int32_t>(seq_len, b, "seq_len", &sl));
    LOGOS_TRY(buf_ptr<__half>(o, b * h_q * d, "o", &op));
    LOGOS_CUDA_TRY(cudaSetDevice(dev));
    // The status word starts at zero with the library image and is sticky like the per-device one: a kernel that gave up
    // leaves its code there, later calls on this entry point do no work on top of it, and logos_kernel_status
    // reports and clears it.
    LOGOS_TRY(static_status_for(dev, &a.ext_status));
    cudaStream_t st = as_stream(stream_or_null);
    a.q_f16 = qp; a.k_cache = kc; a.v_cache = vc; a.seq_len = sl; a.o = op; a.o_dtype = LOGOS_F16;
    a.b = b; a.h_q = h_q; a.h_kv = h_kv; a.d = d; a.l_max = l_max; a.scale = softmax_scale; a.device = dev;
    OrderedScope ordered(st);
    return launch_gqa_decode_attn(a, st);
  });
}

logos_status_t logos_rope_table(float* out_host, int64_t l_max, int64_t d, double theta) {
  return guarded([&]() -> logos_status_t {
    if (!out_host) return fail(LOGOS_NULL_POINTER, "logos_rope_table: out_host is null");
    if (l_max < 0 || d <= 0 || (d & 1)) return fail(LOGOS_OUT_OF_BOUNDS, "logos_rope_table: bad extents");
    rope_table_host(out_host, l_max, d, theta);
    return LOGOS_OK;
  });
}

logos_status_t logos_kv_append_rope(logos_handle_t k_cache, logos_handle_t v_cache, logos_handle_t k_new,
                                    logos_handle_t v_new, logos_handle_t rope_table, logos_handle_t seq_len,
                                    int64_t b, int64_t h_kv, int64_t d, int64_t l_max, void* stream_or_null) {
  return guarded([&]() -> logos_status_t {
    if (b < 0 || h_kv < 0 || d <= 0 || l_max <= 0 || (d & 1))
      return fail(LOGOS_OUT_OF_BOUNDS, "logos_kv_append_rope: bad extents");
    __half *kc, *vc, *kn, *vn;
    float* rt;
    int32_t* sl;
    int32_t dev = 0;
    LOGOS_TRY(buf_ptr<__half>(k_cache, b * h_kv * l_max * d, "k_cache", &kc, &dev));
    LOGOS_TRY(buf_ptr<__half>(v_cache, b * h_kv * l_max * d, "v_cache", &vc));
    LOGOS_TRY(buf_ptr<__half>(k_new, b * h_kv * d, "k_new", &kn));
    LOGOS_TRY(buf_ptr<__half>(v_new, b * h_kv * d, "v_new", &vn));
    LOGOS_TRY(buf_ptr<float>(rope_table, l_max * d, "rope_table", &rt));
    LOGOS_TRY(buf_ptr<int32_t>(seq_len, b, "seq_len", &sl));
    LOGOS_CUDA_TRY(cudaSetDevice(dev));
    return launch_kv_append_rope(kc, vc, kn, vn, rt, sl, b, h_kv, d, l_max, dev, as_stream(stream_or_null));
  });
}

static logos_status_t attn_abi(bool fused, logos_handle_t q, logos_handle_t k_new, logos_handle_t v_new,
                               logos_handle_t k_cache, logos_handle_t v_cache, logos_handle_t rope_table,
                               logos_handle_t seq_len, logos_handle_t o, int64_t b, int64_t h_q, int64_t h_kv,
                               int64_t d, int64_t l_max, float scale, void* stream) {
  if (b < 0 || h_q < 0 || h_kv <= 0 || d <= 0 || l_max <= 0)
    return fail(LOGOS_OUT_OF_BOUNDS, "gqa_decode_attn: bad extents");
  AttnArgs a;
  __half *qp, *kc, *vc, *op;
  int32_t* sl;
  int32_t dev = 0;
  LOGOS_TRY(buf_ptr<__half>(q, b * h_q * d, "q", &qp, &dev));
  LOGOS_TRY(buf_ptr<__half>(k_cache, b * h_kv * l_max * d, "k_cache", &kc));
  LOGOS_TRY(buf_ptr<__half>(v_cache, b * h_kv * l_max * d, "v_cache", &vc));
  LOGOS_TRY(buf_ptr<int32_t>(seq_len, b, "seq_len", &sl));
  LOGOS_TRY(buf_ptr<__half>(o, b * h_q * d, "o", &op));
  a.q_f16 = qp; a.k_cache = kc; a.v_cache = vc; a.seq_len = sl; a.o = op; a.o_dtype = LOGOS_F16;
  if (fused) {
    __half *kn, *vn;
    float* rt;
    LOGOS_TRY(buf_ptr<__half>(k_new, b * h_kv * d, "k_new", &kn));
    LOGOS_TRY(buf_ptr<__half>(v_new, b * h_kv * d, "v_new", &vn));
    LOGOS_TRY(buf_ptr<float>(rope_table, l_max * d, "rope_table", &rt));
    a.k_new_f16 = kn; a.v_new_f16 = vn; a.rope = rt; a.rotate_q = 1; a.bump_seq_len = 1;
  }
  a.b = b; a.h_q = h_q; a.h_kv = h_kv; a.d = d; a.l_max = l_max; a.scale = scale; a.device = dev;
  LOGOS_CUDA_TRY(cudaSetDevice(dev));
  const cudaStream_t st = as_stream(stream);
  OrderedScope ordered(st);
  return launch_gqa_decode_attn(a, st);
}

logos_status_t logos_gqa_decode_attn(logos_handle_t q, logos_handle_t k_cache, logos_handle_t v_cache,
                                     logos_handle_t seq_len, logos_handle_t o, int64_t b, int64_t h_q, int64_t h_kv,
                                     int64_t d, int64_t l_max, float softmax_scale, void* stream_or_null) {
  return guarded([&]() -> logos_status_t {
    return attn_abi(false, q, nullptr, nullptr, k_cache, v_cache, nullptr, seq_len, o, b, h_q, h_kv, d, l_max,
                    softmax_scale, stream_or_null);
  });
}

logos_status_t logos_gqa_decode_attn_fused(logos_handle_t q_raw, logos_handle_t k_new, logos_handle_t v_new,
                                           logos_handle_t k_cache, logos_handle_t v_cache, logos_handle_t rope_table,
                                           logos_handle_t seq_len, logos_handle_t o, int64_t b, int64_t h_q,
                                           int64_t h_kv, int64_t d, int64_t l_max, float softmax_scale,
                                           void* stream_or_null) {
  return guarded([&]() -> logos_status_t {
    return attn_abi(true, q_raw, k_new, v_new, k_cache, v_cache, rope_table, seq_len, o, b, h_q, h_kv, d, l_max,
                    softmax_scale, stream_or_null);
  });
}

}  // extern "C"
