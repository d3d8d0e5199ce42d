// GQA decode attention over an fp16 KV cache, with the rotary embedding and
// the KV-cache append fused in.
//
// HBM-bound: every step streams the whole K and V history once (512 bytes per
// position per KV head at D=128), so the kernel is built around that stream:
//   * the work is the sequence of 64-position K/V tiles of all (sequence, KV head)
//     pairs, in order; the grid is persistent (two CTAs per SM) and CTA c takes the
//     c-th equal share of that sequence, whatever pairs it crosses: every CTA streams
//     the same number of tiles, and a pair is cut only where a share ends;
//   * a producer thread moves the tiles into a 3-stage shared-memory ring with TMA
//     tile loads (128-byte swizzle, no multicast) signalled on mbarriers; the ring
//     keeps running across pairs, so the loads of the next pair are in flight while
//     the consumers finish and write out the previous one; four consumer warps each
//     own 16 positions of every tile;
//   * all query heads that share the KV head (up to 16) form the M side of
//     m16n8k16 tensor-core MMAs, so a K/V tile is read from shared memory once
//     for the whole group; scores, softmax and the running output stay in f32
//     registers; the probabilities enter the second MMA as an fp16 high part
//     plus an fp16 residual so the product keeps f32-class accuracy;
//   * the CTA whose share holds the position being appended rotates the new key
//     (f32 multiply and add rounded separately, fp16 store), writes the new
//     K/V row to the cache and patches it into its own shared-memory tile;
//   * a pair that lies inside one share is normalised and written by that CTA; the parts of a pair
//     that was cut are merged, in the fixed order of their shares, by the CTA that finishes the
//     last of them (a kernel of its own for this cost a launch and a start-up);
//   * a small batch is bound by the chain from the predecessor's end to the output: in a decode step
//     what is older than it (lengths, cached rows) is read, and the work cut, before the wait for
//     the predecessor (AttnArgs::early_reads); every row of the query and the new K/V is one round of loads; the fold is three.
// Measured, before -> after these two: 32 sequences of 4096, 28/4 heads of 128: 69.3 -> 62.7 us
// (4.3 TB/s, launch and ramp included); seven ragged sequences 18.4 -> 14.3 us; a decode step of the 0.5B shape at batch 16
// 954 -> 887 us (24 layers).
#include "ops.cuh"
#include "q8_gemm_tc.cuh"
#include "ptx.cuh"

#include <math.h>

#include <algorithm>
#include <mutex>

namespace logos {

namespace {

using namespace ptx;

constexpr int ATT_TILE = 64;
constexpr int ATT_STAGES = 3;
constexpr int ATT_CWARPS = 4;
constexpr int ATT_CTHREADS = ATT_CWARPS * 32;
constexpr int ATT_THREADS = (ATT_CWARPS + 1) * 32;
constexpr int ATT_BOX_BYTES = 64 * 128;  // 64 rows x 128 bytes
constexpr int ATT_MAX_BATCH = 2048;      // sequences whose lengths a CTA keeps in shared memory

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
  // Parts of cut pairs.  Only the first and the last pair of a share can be cut, so a share writes
  // at most two: slot 0 for a part that begins at the share's first tile, slot 1 otherwise.
  float*        part_o;   // [shares][2][16][D]   unnormalised outputs
  float*        part_ml;  // [shares][2][16][2]   their (max, sum)
  // Arrivals: [shares] parts written of the pair that the end of a share cuts (one pair at most, whatever their
  // number), then CTAs that are done.  Zero before and after every launch (the counters wrap by themselves).
  unsigned*     arrive;
  int           bump;     // the last CTA to finish advances the lengths
  int           early_reads;   // see AttnArgs
  void*         o;        // [B][Hq][D]
  int           o_dtype;
  ActOut        o_act;
  int           b, h_q, h_kv, l_max;
  int           shares;   // the persistent grid's size: the tile sequence is cut into this many shares
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

// Share c of `shares` takes tiles [c * total / shares, (c + 1) * total / shares); the share that
// holds tile g is the largest c whose first tile is <= g.
__device__ __forceinline__ int64_t tile_div(int64_t n, int64_t d) {   // a 64-bit division costs ~100 cycles; n rarely needs it
  return (uint64_t)n >> 32 ? n / d : (int64_t)((uint32_t)n / (uint32_t)d);
}
__device__ __forceinline__ int64_t share_begin(int64_t c, int64_t total, int shares) { return tile_div(c * total, shares); }
__device__ __forceinline__ int share_of_tile(int64_t g, int64_t total, int shares) {
  return (int)tile_div((g + 1) * shares - 1, total);
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

// Folds the parts of a cut pair in ascending order of their shares, for every query row of the group; run by the
// consumer warps of the CTA that wrote the last part.  The first part sits in slot `slot0` of its share
// (0 if it begins at the share's first tile, else 1), every later one in slot 0 of its share.
// The parts are listed once (a lane per share: which shares hold tiles), every row's maximum, weights and
// normaliser are computed once by a warp, and the threads then sum the parts' output rows with all their loads
// independent of one another: a fold is three rounds of global loads whatever the number of parts.  A
// pair cut into more than ATT_MERGE_PARTS shares goes through a plain loop.
// The lists lie where the query was staged, which nothing reads any more.
constexpr int ATT_MERGE_PARTS = 64;
struct MergeScratch {
  int   row0[ATT_MERGE_PARTS];    // first of the 16 rows of each part that holds tiles
  float w[ATT_MERGE_PARTS][16];   // weight of a part for a query row
  float sum[ATT_CWARPS][ATT_MERGE_PARTS];   // the parts' sums for the row that a warp is at
  float l[16];                    // the row's normaliser
  int   np;
};
template <int D>
__device__ __forceinline__ void merge_parts(const AttnParams& p, MergeScratch& ms, int b, int kvh, int first, int last, int slot0,
                                         int64_t total) {
  const int G = p.h_q / p.h_kv;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // with more shares than tiles some shares in between hold no tile
  auto empty = [&](int c) { return share_begin(c, total, p.shares) == share_begin(c + 1, total, p.shares); };
  auto row0_of = [&](int c) -> int { return (c * 2 + (c == first ? slot0 : 0)) * 16; };
  if (last - first + 1 > ATT_MERGE_PARTS) {
    for (int e = tid; e < G * D; e += ATT_CTHREADS) {
      const int r = e / D, d = e - r * D;
      float mstar = -INFINITY;
      for (int c = first; c <= last; ++c)
        if (!empty(c)) mstar = fmaxf(mstar, __ldcg(p.part_ml + (int64_t)(row0_of(c) + r) * 2));
      float muse = (mstar == -INFINITY) ? 0.f : mstar;
      float acc = 0.f, L = 0.f;
      for (int c = first; c <= last; ++c) {
        if (empty(c)) continue;
        const int64_t row = row0_of(c) + r;
        float wgt = exp2f(__ldcg(p.part_ml + row * 2) - muse);
        acc = fmaf(__ldcg(p.part_o + row * D + d), wgt, acc);
        L = fmaf(__ldcg(p.part_ml + row * 2 + 1), wgt, L);
      }
      store_out(p, ((int64_t)b * p.h_q + kvh * G + r) * D + d, __fdiv_rn(acc, L));
    }
    return;
  }
  if (warp == 0) {  // list the parts in ascending order of their shares
    int np = 0;
    for (int c0 = first; c0 <= last; c0 += 32) {
      const int c = c0 + lane;
      const bool has = c <= last && !empty(c);
      const uint32_t m = __ballot_sync(0xffffffffu, has);
      if (has) ms.row0[np + __popc(m & ((1u << lane) - 1u))] = row0_of(c);
      np += __popc(m);
    }
    if (lane == 0) ms.np = np;
  }
  asm volatile("bar.sync 1, %0;" ::"n"(ATT_CTHREADS) : "memory");
  const int np = ms.np;
  // per query row (a warp each): maximum, weights in part order, normaliser summed in part order
  for (int r = warp; r < G; r += ATT_CWARPS) {
    float2 ml[ATT_MERGE_PARTS / 32];   // (max, sum) of parts lane, lane + 32: one round of loads
#pragma unroll
    for (int j = 0; j < ATT_MERGE_PARTS / 32; ++j) {
      const int pi = lane + 32 * j;
      ml[j] = pi < np ? __ldcg(reinterpret_cast<const float2*>(p.part_ml) + ms.row0[pi] + r) : make_float2(-INFINITY, 0.f);
    }
    float mloc = -INFINITY;
#pragma unroll
    for (int j = 0; j < ATT_MERGE_PARTS / 32; ++j) mloc = fmaxf(mloc, ml[j].x);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mloc = fmaxf(mloc, __shfl_xor_sync(0xffffffffu, mloc, o));
    const float muse = (mloc == -INFINITY) ? 0.f : mloc;
#pragma unroll
    for (int j = 0; j < ATT_MERGE_PARTS / 32; ++j) {
      const int pi = lane + 32 * j;
      if (pi < np) {
        ms.w[pi][r] = exp2f(ml[j].x - muse);
        ms.sum[warp][pi] = ml[j].y;
      }
    }
    __syncwarp();
    if (lane == 0) {
      float L = 0.f;
#pragma unroll 4
      for (int pi = 0; pi < np; ++pi) L = fmaf(ms.sum[warp][pi], ms.w[pi][r], L);
      ms.l[r] = L;
    }
    __syncwarp();   // the next row's sums go where these are
  }
  asm volatile("bar.sync 1, %0;" ::"n"(ATT_CTHREADS) : "memory");
  // four neighbouring elements a thread, four parts' loads in flight: a part at a time took a round of latency
  // each (8 us for the twenty parts of a long sequence in a small batch)
  for (int e = 4 * tid; e < G * D; e += 4 * ATT_CTHREADS) {   // row e / D, column e % D: a part's rows are contiguous
    const int r = e / D;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int p0 = 0; p0 < np; p0 += 4) {
      float4 v[4];
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (p0 + k < np) v[k] = __ldcg(reinterpret_cast<const float4*>(p.part_o + (int64_t)ms.row0[p0 + k] * D + e));
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (p0 + k < np) {
          const float w = ms.w[p0 + k][r];
          acc.x = fmaf(v[k].x, w, acc.x); acc.y = fmaf(v[k].y, w, acc.y);
          acc.z = fmaf(v[k].z, w, acc.z); acc.w = fmaf(v[k].w, w, acc.w);
        }
    }
    store_out4(p, ((int64_t)b * p.h_q + kvh * G) * D + e, acc, ms.l[r]);
  }
}

// Dynamic shared memory of a CTA: the ring, the staged query, the appended rows and the warps' (max, sum), whose place
// the fold's lists take over, the barriers, then by sequence the tiles before it and its last tile.
template <int D>
struct AttnSmem {
  static constexpr int QS_STRIDE = D + 8;  // halfs; +16 bytes keeps ldmatrix rows on distinct banks
  static constexpr int STAGE_BYTES = 2 * (D / 64) * ATT_BOX_BYTES;
  static constexpr int STAGED = 16 * QS_STRIDE * 2 + 2 * D * 2 + ATT_CWARPS * 16 * 2 * 4;
  static constexpr int WORK = ((STAGED > (int)sizeof(MergeScratch) ? STAGED : (int)sizeof(MergeScratch)) + 15) / 16 * 16;
  static constexpr int BARS = 2 * ATT_STAGES * 8;
  static constexpr int FLAGS = 16;
  static constexpr int bytes(int batch) {
    return 1024 + ATT_STAGES * STAGE_BYTES + WORK + BARS + FLAGS + (batch + 1) * 4 + batch;
  }
};
// An SM has 228 KB and keeps 1 KB of it for each CTA.  With one CTA an SM the grid takes two rounds: 512 sequences of
// 1024 positions, 28/4 heads of 128, 240 us against 181.
static_assert(2 * (AttnSmem<128>::bytes(ATT_MAX_BATCH) + 1024) <= 228 * 1024, "two CTAs fit an SM whatever the batch");
static_assert(2 * (AttnSmem<64>::bytes(ATT_MAX_BATCH) + 1024) <= 228 * 1024, "two CTAs fit an SM whatever the batch");

template <int D>
__global__ void __launch_bounds__(ATT_THREADS, 2)
gqa_decode_attn_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                       const AttnParams p) {
  constexpr int NBOX = D / 64;
  using Smem = AttnSmem<D>;
  constexpr int STAGE_BYTES = Smem::STAGE_BYTES;
  constexpr int QS_STRIDE = Smem::QS_STRIDE;
  constexpr int KSTEPS = D / 16;
  static_assert(STAGE_BYTES >= ATT_CWARPS * 16 * D * 4, "a ring stage doubles as the scratch that combines the warps");

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* stages = smem;                                            // ATT_STAGES * STAGE_BYTES
  __half* qs = reinterpret_cast<__half*>(stages + ATT_STAGES * STAGE_BYTES);  // [16][QS_STRIDE]
  __half* new_k = qs + 16 * QS_STRIDE;                               // [D]
  __half* new_v = new_k + D;                                         // [D]
  float* mml = reinterpret_cast<float*>(new_v + D);                  // [warp][16][2]
  MergeScratch& s_merge = *reinterpret_cast<MergeScratch*>(qs);      // in place of all of these, once a pair is done
  uint64_t* bar_full = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(qs) + Smem::WORK);
  uint64_t* bar_empty = bar_full + ATT_STAGES;
  int& prior_status = *reinterpret_cast<int*>(bar_empty + ATT_STAGES);
  int& s_bump = *(&prior_status + 1);   // this CTA is the last to have its lengths
  int& s_last = *(&prior_status + 2);   // this CTA wrote a pair's last part (the consumers' own: the producer may still look at s_bump)
  int32_t* s_pref = &prior_status + 4;                               // [B + 1] tiles before it
  uint8_t* s_tail = reinterpret_cast<uint8_t*>(s_pref + p.b + 1);    // [B] positions that its last tile lacks; FULL: the length is l_max or more
  constexpr int FULL = 128;
  static_assert(ATT_TILE <= FULL, "a tile's positions beside the flag");

  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const int G = p.h_q / p.h_kv;
  auto tiles_of = [&](int b) { return s_pref[b + 1] - s_pref[b]; };

  // In a decode step the lengths and the cached rows are older than the step, so reading them, cutting the work and
  // loading the first tiles overlap the predecessor's end, and only what reads the query and the new K/V rows waits.
  // Elsewhere the predecessor may write any of them: everything waits.
  if (!p.early_reads) pdl_wait();
  // a kernel that gave up earlier left a code behind: do not start new work on top of it
  // (one thread reads, everyone takes the same decision)
  if (tid == 0) {
    prior_status = *reinterpret_cast<volatile int*>(p.status);
    for (int i = 0; i < ATT_STAGES; ++i) {
      mbar_init(&bar_full[i], 1);
      mbar_init(&bar_empty[i], ATT_CWARPS);
    }
    fence_barrier_init();
    prefetch_tensormap(&map_k);
    prefetch_tensormap(&map_v);
  }
  for (int b = tid; b < p.b; b += ATT_THREADS) {
    const int len0 = __ldcg(p.seq_len + b), len_eff = attn_len_eff(p, len0);
    const int tiles = (len_eff + ATT_TILE - 1) / ATT_TILE;
    s_pref[b] = tiles;
    s_tail[b] = (uint8_t)((tiles * ATT_TILE - len_eff) | (len0 >= p.l_max ? FULL : 0));
  }
  __syncthreads();
  if (prior_status != 0) {
    pdl_wait();
    return;
  }
  if (warp == 0) {  // exclusive prefix over the sequences: lane l sums a contiguous run, then a warp scan
    const int per = (p.b + 31) / 32;
    int run = 0;
    for (int i = 0; i < per; ++i) {
      const int b = lane * per + i;
      if (b < p.b) run += s_pref[b];
    }
    int incl = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    int acc = incl - run;
    for (int i = 0; i < per; ++i) {
      const int b = lane * per + i;
      if (b < p.b) {
        const int tiles = s_pref[b];
        s_pref[b] = acc;
        acc += tiles;
      }
    }
    if (lane == 31) s_pref[p.b] = incl;
  }
  __syncthreads();
  const int64_t total = (int64_t)p.h_kv * s_pref[p.b];
  const int64_t g_lo = total ? share_begin(blockIdx.x, total, p.shares) : 0, g_hi = total ? share_begin(blockIdx.x + 1, total, p.shares) : 0;
  if (warp < ATT_CWARPS || g_lo >= g_hi) {
    pdl_wait();   // (a CTA that leaves must not let the grid end before its predecessor)
    pdl_trigger();
  }
  // a sequence without any position to attend to has no tile, hence no CTA: its output rows are zero
  if (warp < ATT_CWARPS)
    for (int b = blockIdx.x; b < p.b; b += gridDim.x)
      if (tiles_of(b) == 0)
        for (int e = tid; e < p.h_q * D; e += ATT_CTHREADS) store_out(p, (int64_t)b * p.h_q * D + e, 0.f);
  // everyone has its lengths by now: the last CTA to come by advances them
  if (p.bump) {
    if (tid == 0) s_bump = arrive_inc(p.arrive + p.shares, gridDim.x - 1) == gridDim.x - 1;
    __syncthreads();
    if (s_bump)
      for (int b = tid; b < p.b; b += ATT_THREADS) {
        const int len = __ldcg(p.seq_len + b);
        if (len < p.l_max) p.seq_len[b] = len + 1;
      }
  }
  if (g_lo >= g_hi) return;

  // Both roles walk the share the same way: tile g belongs to sequence b (the one with
  // h_kv * pref[b] <= g < h_kv * pref[b + 1]), KV head (g - h_kv * pref[b]) / tiles[b], tile
  // (g - h_kv * pref[b]) % tiles[b] of that pair.
  int b_cur = 0;
  {
    int lo = 0, hi = p.b;  // last b with h_kv * pref[b] <= g_lo
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if ((int64_t)p.h_kv * s_pref[mid] <= g_lo) lo = mid; else hi = mid;
    }
    b_cur = lo;
  }

  bool ok = true;

  if (warp == ATT_CWARPS) {
    // ---------------------------------------------------------------- producer
    if (lane == 0) {
      int t_ring = 0;
      int b = b_cur;
      for (int64_t g = g_lo; g < g_hi && ok;) {
        while ((int64_t)p.h_kv * s_pref[b + 1] <= g) ++b;
        const int tiles_b = tiles_of(b);
        const int64_t within = g - (int64_t)p.h_kv * s_pref[b];
        const int kvh = (int)(within / tiles_b), t0 = (int)(within - (int64_t)kvh * tiles_b);
        const int t1 = (int)min((int64_t)tiles_b, t0 + (g_hi - g));
        const int64_t row_base = ((int64_t)b * p.h_kv + kvh) * p.l_max;
        for (int t = t0; t < t1 && ok; ++t, ++t_ring) {
          const int st = t_ring % ATT_STAGES;
          const uint32_t ph = (uint32_t)(t_ring / ATT_STAGES) & 1u;
          ok = mbar_wait(&bar_empty[st], ph ^ 1u);
          if (!ok) break;
          uint8_t* sb = stages + st * STAGE_BYTES;
          mbar_arrive_expect_tx(&bar_full[st], STAGE_BYTES);
          const int y = (int)(row_base + (int64_t)t * ATT_TILE);
#pragma unroll
          for (int j = 0; j < NBOX; ++j) {
            tma_load_2d(sb + j * ATT_BOX_BYTES, &map_k, &bar_full[st], j * 64, y);
            tma_load_2d(sb + (NBOX + j) * ATT_BOX_BYTES, &map_v, &bar_full[st], j * 64, y);
          }
        }
        g += t1 - t0;
      }
      if (!ok) atomicExch(p.status, 101);
    }
  } else {
    // ---------------------------------------------------------------- consumers
    const int g4 = lane >> 2, t4 = lane & 3;
    const int ctid = tid;  // 0 .. ATT_CTHREADS - 1
    int t_ring = 0;
    int b = b_cur;
    for (int64_t g = g_lo; g < g_hi && ok;) {
      while ((int64_t)p.h_kv * s_pref[b + 1] <= g) ++b;
      const int tiles_b = tiles_of(b);
      const int64_t pair0 = (int64_t)p.h_kv * s_pref[b];
      const int64_t within = g - pair0;
      const int kvh = (int)(within / tiles_b), t0 = (int)(within - (int64_t)kvh * tiles_b);
      const int t1 = (int)min((int64_t)tiles_b, t0 + (g_hi - g));
      const int64_t pair_g0 = pair0 + (int64_t)kvh * tiles_b;  // first tile of the pair in the whole sequence
      const int share_first = share_of_tile(pair_g0, total, p.shares);
      const int share_last = share_of_tile(pair_g0 + tiles_b - 1, total, p.shares);
      const bool whole = share_first == share_last;   // the pair lies inside this share: write the result itself
      const int slot = g == g_lo ? 0 : 1;
      const int len_eff = tiles_b * ATT_TILE - (s_tail[b] & (FULL - 1));
      const int len0 = (s_tail[b] & FULL) ? p.l_max : p.fused ? len_eff - 1 : len_eff;   // up to l_max
      const int64_t row_base = ((int64_t)b * p.h_kv + kvh) * p.l_max;
      const int pos_new = len0;  // where the appended row goes
      const bool append = p.fused && len0 < p.l_max;
      const bool owns_new = append && pos_new >= t0 * ATT_TILE && pos_new < t1 * ATT_TILE;

      // ---- stage the query heads (rotated when asked), zero the padding rows; the appended row is rotated, rounded
      // to fp16, written to the cache and kept.  A thread takes four columns of a row and their partners half a
      // head away, so that all rows are one round of loads (every part of a split sum in flight at once).
      {
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
      asm volatile("bar.sync 1, %0;" ::"n"(ATT_CTHREADS));

      uint32_t qa[KSTEPS][4];
      {
        int row = (lane & 7) + 8 * ((lane >> 3) & 1);
        int colh = 8 * (lane >> 4);
#pragma unroll
        for (int ks = 0; ks < KSTEPS; ++ks) {
          uint32_t addr = smem_u32(qs + row * QS_STRIDE + ks * 16 + colh);
          ldmatrix_x4(qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3], addr);
        }
      }
      float m_run[2] = {-INFINITY, -INFINITY};
      float l_run[2] = {0.f, 0.f};
      float o[D / 8][4];
#pragma unroll
      for (int i = 0; i < D / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;

      int st = 0;
      for (int t = t0; t < t1; ++t, ++t_ring) {
        st = t_ring % ATT_STAGES;
        uint32_t ph = (uint32_t)(t_ring / ATT_STAGES) & 1u;
        if (!mbar_wait(&bar_full[st], ph)) {
          ok = false;
          break;
        }
        uint8_t* kb = stages + st * STAGE_BYTES;
        uint8_t* vb = kb + NBOX * ATT_BOX_BYTES;
        const int tile_pos0 = t * ATT_TILE;
        const int my_pos0 = tile_pos0 + 16 * warp;

        // patch the appended row / clear rows past the end (only this warp reads its 16 rows)
        if (my_pos0 + 16 > len_eff || (owns_new && pos_new >= my_pos0 && pos_new < my_pos0 + 16)) {
          for (int r = 0; r < 16; ++r) {
            int pos = my_pos0 + r;
            uint32_t row = 16 * warp + r;
            if (owns_new && pos == pos_new) {
              for (int c = lane; c < 2 * (D / 8); c += 32) {
                bool is_v = c >= D / 8;
                int cc = is_v ? c - D / 8 : c;
                const uint4 val = *reinterpret_cast<const uint4*>((is_v ? new_v : new_k) + cc * 8);
                uint8_t* base = (is_v ? vb : kb) + (cc >> 3) * ATT_BOX_BYTES;
                *reinterpret_cast<uint4*>(base + swz128(row, cc & 7)) = val;
              }
            } else if (pos >= len_eff) {
              for (int c = lane; c < D / 8; c += 32) {
                uint8_t* base = vb + (c >> 3) * ATT_BOX_BYTES;
                *reinterpret_cast<uint4*>(base + swz128(row, c & 7)) = make_uint4(0, 0, 0, 0);
              }
            }
          }
          fence_proxy_async_smem();   // the next tile's loads write here
          __syncwarp();
        }

        // ---- S = Q K^T for 16 positions
        float s[2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i) s[i][0] = s[i][1] = s[i][2] = s[i][3] = 0.f;
        {
          uint32_t row = 16 * warp + (lane & 7) + 8 * (lane >> 4);
          int ch = (lane >> 3) & 1;
#pragma unroll
          for (int ks = 0; ks < KSTEPS; ++ks) {
            int chunk = ks * 2 + ch;
            uint32_t addr = smem_u32(kb + (chunk >> 3) * ATT_BOX_BYTES + swz128(row, chunk & 7));
            uint32_t r0, r1, r2, r3;
            ldmatrix_x4(r0, r1, r2, r3, addr);
            mma_f16_16816(s[0], qa[ks], r0, r1);
            mma_f16_16816(s[1], qa[ks], r2, r3);
          }
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
          uint32_t row = 16 * warp + (lane & 7) + 8 * ((lane >> 3) & 1);
          int ch = lane >> 4;
#pragma unroll
          for (int dn = 0; dn < D / 16; ++dn) {
            int chunk = dn * 2 + ch;
            uint32_t addr = smem_u32(vb + (chunk >> 3) * ATT_BOX_BYTES + swz128(row, chunk & 7));
            uint32_t r0, r1, r2, r3;
            ldmatrix_x4_trans(r0, r1, r2, r3, addr);
            mma_f16_16816(o[2 * dn], a_hi, r0, r1);
            mma_f16_16816(o[2 * dn], a_lo, r0, r1);
            mma_f16_16816(o[2 * dn + 1], a_hi, r2, r3);
            mma_f16_16816(o[2 * dn + 1], a_lo, r2, r3);
          }
        }
        __syncwarp();
        // the last tile of this part keeps its ring stage: it is the scratch the warps are combined in
        if (t + 1 < t1 && lane == 0) mbar_arrive(&bar_empty[st]);
      }
      // ---- combine the four warps in the ring stage of the part's last tile (every warp has
      // read its rows of it once all four have passed the barrier), then hand the stage back.
      // The barrier also carries the outcome: a warp whose wait gave up takes the others with it.
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        l_run[r] += __shfl_xor_sync(0xffffffffu, l_run[r], 1);
        l_run[r] += __shfl_xor_sync(0xffffffffu, l_run[r], 2);
      }
      {
        int all_ok;
        asm volatile(
            "{\n\t.reg .pred q, r;\n\tsetp.ne.u32 q, %1, 0;\n\tbar.red.and.pred r, 1, %2, q;\n\tselp.u32 %0, 1, 0, r;\n\t}"
            : "=r"(all_ok)
            : "r"((uint32_t)ok), "n"(ATT_CTHREADS)
            : "memory");
        if (!all_ok) {
          if (!ok && lane == 0) atomicExch(p.status, 102);
          ok = false;
          break;
        }
      }
      float* mo = reinterpret_cast<float*>(stages + st * STAGE_BYTES);   // [warp][16][D]
#pragma unroll
      for (int i = 0; i < D / 8; ++i) {
        int col = i * 8 + 2 * t4;
        float* r0p = mo + ((warp * 16 + g4) * D) + col;
        float* r1p = mo + ((warp * 16 + g4 + 8) * D) + col;
        r0p[0] = o[i][0]; r0p[1] = o[i][1];
        r1p[0] = o[i][2]; r1p[1] = o[i][3];
      }
      if (t4 == 0) {
        mml[(warp * 16 + g4) * 2 + 0] = m_run[0];
        mml[(warp * 16 + g4) * 2 + 1] = l_run[0];
        mml[(warp * 16 + g4 + 8) * 2 + 0] = m_run[1];
        mml[(warp * 16 + g4 + 8) * 2 + 1] = l_run[1];
      }
      asm volatile("bar.sync 1, %0;" ::"n"(ATT_CTHREADS));
      const int64_t pi = ((int64_t)blockIdx.x * 2 + slot) * 16;   // row 0 of this part's slot
      for (int e = 4 * ctid; e < G * D; e += 4 * ATT_CTHREADS) {   // four columns a thread: one pass over the weights
        const int r = e / D, d = e - r * D;
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
        if (whole) {
          store_out4(p, ((int64_t)b * p.h_q + kvh * G) * D + e, acc, L);
        } else {
          *reinterpret_cast<float4*>(p.part_o + pi * D + e) = acc;
          if (d == 0) *reinterpret_cast<float2*>(p.part_ml + (pi + r) * 2) = make_float2(mstar, L);
        }
      }
      fence_proxy_async_smem();   // the scratch is a ring stage: the next tile's loads write there
      asm volatile("bar.sync 1, %0;" ::"n"(ATT_CTHREADS) : "memory");   // everyone has read the scratch and qs
      if (lane == 0) mbar_arrive(&bar_empty[st]);
      if (!whole) {
        // with no more shares than tiles every share in between holds some; with more, each holds one at most
        const unsigned parts = p.shares <= total ? (unsigned)(share_last - share_first + 1) : (unsigned)tiles_b;
        // (the barrier above put all of this CTA's part before the releasing increment)
        if (ctid == 0) s_last = arrive_inc(p.arrive + share_first, parts - 1) == parts - 1;
        asm volatile("bar.sync 1, %0;" ::"n"(ATT_CTHREADS) : "memory");
        if (s_last) {
          merge_parts<D>(p, s_merge, b, kvh, share_first, share_last, share_begin(share_first, total, p.shares) == pair_g0 ? 0 : 1, total);
          asm volatile("bar.sync 1, %0;" ::"n"(ATT_CTHREADS) : "memory");   // s_merge and s_last may be written again
        }
      }
      g += t1 - t0;
    }
  }
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

// The persistent grid: the tile sequence is cut into this many shares, one per CTA.
int attn_shares(const AttnArgs& a) {
  const int sms = sm_count(a.device);
  const int64_t tiles_max = (a.l_max + ATT_TILE - 1) / ATT_TILE;
  int64_t g = std::min<int64_t>(2 * sms, ATT_COUNTER_BYTES / sizeof(unsigned) - 1);   // two CTAs of up to 113 KB of shared memory fit an SM (AttnSmem)
  // With no more (sequence, KV head) pairs than CTAs, a whole number of shares per pair: where the
  // sequences are equally long every share boundary then falls on a pair boundary or cuts a pair
  // into equal pieces, and a CTA stages one pair's query instead of two (measured 4-8 % on the
  // operator at the shapes a rank of four or eight holds; neutral for ragged lengths).
  const int64_t pairs = a.b * a.h_kv;
  if (pairs > 0 && pairs <= g) g = g / pairs * pairs;
  const int64_t most = a.b * a.h_kv * tiles_max;
  if (g > most) g = most > 0 ? most : 1;
  return (int)g;
}

template <int D>
logos_status_t launch_attn_t(const AttnArgs& a, cudaStream_t st) {
  if (a.b > ATT_MAX_BATCH)
    return fail(LOGOS_OUT_OF_BOUNDS, "attention: batch %lld exceeds %d sequences per call", (long long)a.b, ATT_MAX_BATCH);
  const int64_t rows_total = a.b * a.h_kv * a.l_max;
  CUtensorMap mk, mv;
  LOGOS_TRY(cached_map(&mk, a.k_cache, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, D, rows_total, D * 2, 64, ATT_TILE));
  LOGOS_TRY(cached_map(&mv, a.v_cache, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, D, rows_total, D * 2, 64, ATT_TILE));
  const int shares = attn_shares(a);

  // parts of cut pairs, then the arrival counters, which have to be zero when the first launch comes
  const int64_t part_bytes = (int64_t)shares * 2 * 16 * (D + 2) * (int64_t)sizeof(float);
  void* scratch = a.ext_scratch;
  void* arrive = a.ext_arrive;
  if (a.ext_scratch) {
    if (part_bytes > a.ext_scratch_bytes)
      return fail(LOGOS_OUT_OF_BOUNDS, "attention: this shape needs %lld bytes of split-KV scratch, the fixed scratch holds %lld",
                  (long long)part_bytes, (long long)a.ext_scratch_bytes);
  } else {
    LOGOS_TRY(scratch_get(a.device, 1, part_bytes, &scratch));
    LOGOS_TRY(counters_get(a.device, ATT_COUNTER_BYTES, &arrive));
  }

  AttnParams p{};
  p.q_f16 = a.q_f16; p.q_f32 = a.q_f32; p.q_ld = a.q_ld; p.rotate_q = a.rotate_q;
  p.k_new_f16 = a.k_new_f16; p.v_new_f16 = a.v_new_f16; p.k_new_f32 = a.k_new_f32; p.v_new_f32 = a.v_new_f32;
  p.kv_ld = a.kv_ld;
  p.f32_parts = a.f32_parts > 1 ? a.f32_parts : 1;
  p.f32_part_stride = a.f32_part_stride;
  p.q_bias = a.q_bias; p.k_bias = a.k_bias; p.v_bias = a.v_bias;
  p.fused = (a.k_new_f16 || a.k_new_f32) ? 1 : 0;
  p.k_cache = a.k_cache; p.v_cache = a.v_cache; p.rope = a.rope; p.seq_len = a.seq_len;
  p.part_o = reinterpret_cast<float*>(scratch);
  p.part_ml = p.part_o + (int64_t)shares * 2 * 16 * D;
  p.arrive = reinterpret_cast<unsigned*>(arrive);
  p.bump = a.bump_seq_len;
  p.early_reads = a.early_reads;
  p.o = a.o; p.o_dtype = a.o_dtype; p.o_act = a.o_act;
  p.b = (int)a.b; p.h_q = (int)a.h_q; p.h_kv = (int)a.h_kv; p.l_max = (int)a.l_max;
  p.shares = shares;
  p.scale_log2 = a.scale * 1.4426950408889634f;
  p.status = a.ext_status ? a.ext_status : kernel_status_ptr(a.device);
  if (!p.status) return fail(LOGOS_ERROR, "attention: no kernel status word");

  const int smem = AttnSmem<D>::bytes((int)a.b);
  LOGOS_TRY(allow_smem(reinterpret_cast<const void*>(gqa_decode_attn_kernel<D>), a.device, smem));
  LOGOS_CUDA_TRY(launch_kernel(gqa_decode_attn_kernel<D>, dim3((unsigned)shares), dim3(ATT_THREADS), (size_t)smem, st, mk, mv, p));
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

int64_t attn_scratch_bytes(const AttnArgs& a) {
  return (int64_t)attn_shares(a) * 2 * 16 * (a.d + 2) * (int64_t)sizeof(float);
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

// ---------------------------------------------------------------- fixed-scratch variant
// Scratch that lives in the library image instead of coming from cudaMalloc: every GPU
// that loads the library holds these 6 MiB (+ one status word) until the process exits.
// The kernel needs two part slots of 16 x (D + 2) floats per CTA of its persistent grid (two
// CTAs per SM): 4.7 MiB on a 148-SM B200 at D = 128; what is left before the counters provides for 188 SMs.
constexpr int64_t kStaticScratchBytes = 6ll << 20;
static __device__ __align__(256) unsigned char g_static_attn_scratch[kStaticScratchBytes];
static __device__ __align__(256) int g_static_attn_status[8];

namespace {
constexpr int kMaxStaticDevices = 64;
struct StaticAddr {
  void* scratch = nullptr;
  int*  status = nullptr;
  bool  ready = false;
};
StaticAddr g_static_addr[kMaxStaticDevices];
std::mutex g_static_mu;

// In host code the array names above are host-side stand-ins, not device addresses: the
// address a kernel may use comes from cudaGetSymbolAddress, asked once per device with
// that device current.
logos_status_t static_scratch_for(int device, StaticAddr* out) {
  if (device < 0 || device >= kMaxStaticDevices)
    return fail(LOGOS_OUT_OF_BOUNDS, "fixed-scratch attention: device %d is beyond the %d this build tracks", device,
                kMaxStaticDevices);
  std::lock_guard<std::mutex> lk(g_static_mu);
  StaticAddr& sa = g_static_addr[device];
  if (!sa.ready) {
    void* p = nullptr;
    void* q = nullptr;
    LOGOS_CUDA_TRY(cudaGetSymbolAddress(&p, g_static_attn_scratch));
    LOGOS_CUDA_TRY(cudaGetSymbolAddress(&q, g_static_attn_status));
    sa.scratch = p;
    sa.status = static_cast<int*>(q);
    sa.ready = true;
  }
  *out = sa;
  return LOGOS_OK;
}
}  // namespace

// The fixed-scratch entry point's own status word, for logos_kernel_status: copies the eight
// words out (and zeroes them when asked) if that entry point has run on `device`; *used tells
// whether it has.  A device-to-host copy of eight words: no allocation here either.
logos_status_t static_attn_status_read(int device, int words_out[8], bool clear, bool* used) {
  *used = false;
  if (device < 0 || device >= kMaxStaticDevices) return LOGOS_OK;
  StaticAddr sa;
  {
    std::lock_guard<std::mutex> lk(g_static_mu);
    sa = g_static_addr[device];
  }
  if (!sa.ready) return LOGOS_OK;
  LOGOS_CUDA_TRY(cudaSetDevice(device));
  LOGOS_CUDA_TRY(cudaMemcpy(words_out, sa.status, sizeof(int) * 8, cudaMemcpyDeviceToHost));
  if (clear && words_out[0] != 0) {
    // a kernel that gave up leaves arrivals uncounted
    LOGOS_CUDA_TRY(cudaMemset(static_cast<char*>(sa.scratch) + kStaticScratchBytes - ATT_COUNTER_BYTES, 0, ATT_COUNTER_BYTES));
    LOGOS_CUDA_TRY(cudaMemset(sa.status, 0, sizeof(int) * 8));
  }
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
    StaticAddr sa;
    LOGOS_TRY(static_scratch_for(dev, &sa));
    cudaStream_t st = as_stream(stream_or_null);
    // Nothing in the array has to be cleared.  The partials: every entry the merge reads is
    // written by this call first.  The counters wrap to zero by themselves.  The status word starts at zero with the library image and is
    // sticky like the per-device one: a kernel that gave up leaves its code there, later calls
    // on this entry point do no work on top of it, and logos_kernel_status reports and clears it.
    a.q_f16 = qp; a.k_cache = kc; a.v_cache = vc; a.seq_len = sl; a.o = op; a.o_dtype = LOGOS_F16;
    a.b = b; a.h_q = h_q; a.h_kv = h_kv; a.d = d; a.l_max = l_max; a.scale = softmax_scale; a.device = dev;
    a.ext_scratch = sa.scratch;
    a.ext_scratch_bytes = kStaticScratchBytes - ATT_COUNTER_BYTES;
    a.ext_arrive = static_cast<char*>(sa.scratch) + a.ext_scratch_bytes;
    a.ext_status = sa.status;
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
  return launch_gqa_decode_attn(a, as_stream(stream));
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
