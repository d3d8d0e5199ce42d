// Q8 GEMM on the 5th-generation tensor cores (tcgen05).
//
//   acc[n, m] = sum_kb s[n,kb] * ( sum_{k in kb} q[n,k] * a[m,k] )
//
// "Weights on the M side": a tile is 128 weight rows (MMA M = 128, one TMEM lane per row) and T
// tokens (MMA N), so the f32 scale of a (row, K block) pair is one scalar per thread when the
// block's partial sum is drained from tensor memory.  A work unit is a pair of neighbouring row
// tiles (or a single one, for what full rounds of pairs leave over) x a K split x a token tile: the
// activation loads of a K stage serve both tiles, which matters because at 64 tokens in two
// planes they are 32 KB per stage against the 18 KB of weights and scales of a tile, and an SM's
// L2 port takes about 64 bytes a cycle.
//
// Data flow per 128-column K stage (4 Q8 blocks) and tile, in two groups of half a stage:
//   TMA  int8 weights [128 rows][128 B], 128-byte swizzle, and the stage's scales [128 rows][4]
//        -> shared-memory rings                                                    (warp 0)
//   TMA  fp16 activation planes of the stage [planes][2 halves][T][64] -> ring, one 4-D copy (warp 1)
//   4 converter warps (one per TMEM lane quarter): int8 -> fp16 (exact: 0x6400|b trick),
//        tcgen05.st into the operand ring; the weights never go back to shared memory
//   MMA warps 2 and 3, one per half: per Q8 block two tcgen05.mma kind::f16 (K = 16 each) per plane, A
//        from TMEM, B = activations from smem, into a fresh accumulator entry: first q*lo', then
//        q*hi + D*2^-11 through the MMA's own accumulator scaling, so hi + lo*2^-11 is
//        recombined on the tensor core
//   16 drain warps (8 up to 32 tokens): tcgen05.ld a group's partial sums, acc += s * partial in f32
//        registers.  Of a pair, half of the warps take one tile each (lane quarter x a share of the tokens);
//        a single tile is shared by all.  Then the epilogue, straight from registers: a warp's lanes
//        hold consecutive output columns of a token.
// A CTA is persistent and the rings keep running across units.  All hand-offs are mbarriers; every
// wait is bounded and reports through the device status word instead of spinning for ever.
//
// What bounds it, in SM cycles (stage traces and micro-measurements on a B200).  A wait for a barrier
// that is ready costs 65 to 80, a hand-off between two warps 93, an MMA of N = 64 38 with its completion
// seen ~160 later, tcgen05.ld ~100; FFMA2 issues every 2.3 cycles per scheduler, PRMT and HSUB2 every 2.
// So a tile's stage at 64 tokens has 430 of FMA pipe, 610 of tensor pipe in two planes and about 730 of
// HBM time, and everything else is latency: with one accumulator entry per half stage the kernel ran at
// that entry's round trip (1500 per tile stage, with one plane or two and whatever the ring depths), with
// eight drain warps at the drain's serial chain (1225).  Hence several entries, two groups of drain
// warps, few and coarse hand-offs, ring positions kept as 32-bit shared addresses, and registers moved
// from the other warps to the drain warps.
//
// Registers are what 96 tokens run out of: the kernel spills 112 to 172 bytes a thread there (`-Xptxas -v`), up to 40
// elsewhere.  With many tokens and enough row tiles another form of it runs, see WideCfg.
//
// HBM roofline: 1.125 bytes per weight (int8 + f32/32); activations and outputs are small next to
// that at decode batch sizes.  With many tokens the FMA and tensor pipes are the bound.
#include "q8_gemm_tc.cuh"

#include "ptx.cuh"

#include <algorithm>
#include <mutex>
#include <type_traits>
#include <unordered_map>

namespace logos {

namespace {

using namespace ptx;

constexpr int TC_ROWS = 128;     // weight rows per tile (MMA M)
constexpr int TC_KSTAGE = 128;   // K per stage: one raw slot; a group, an operand or activation slot is half of it
constexpr int RAW_BYTES = TC_ROWS * TC_KSTAGE;  // 16 KB
constexpr int SC_BYTES = TC_ROWS * 16;          // four f32 per row and stage
constexpr int TA_SLOTS = 4;                     // operand ring, in groups
constexpr int TA_SLOT_COLS = 32;                // TMEM columns of 64 fp16 per row
constexpr uint32_t TMEM_COLS = 512;
// Barrier sets of the accumulators: group n hands off through set n % GROUPS, over entry n % ENTRIES.  The MMA warp
// of one half may wait for releases of the other half's groups (odd ENTRIES).  Those run at most one pair stage
// (four groups) ahead of it, because the drain takes the halves in turn; with eight sets a set cannot go
// through a second phase unseen, which the parity test could not tell from none (with four it could).
constexpr int GROUPS = 8;
constexpr int CONV_WARP0 = 4, DRAIN_WARP0 = 8;  // 4 single-role warps, 4 converter warps, then the drain warps

// Shapes of the rings by token count.  Tensor memory: operand slots x 32 + entries x 2 T columns of the
// 512; shared memory: raw, activation and scale rings within 227 KB.
template <int T, int LIMBS>
struct TcCfg {
  // Accumulator entries, a group (two blocks) each, and blocks per hand-off: one where only two entries fit, so
  // that each block's columns go back to the MMAs as soon as they are read.
  static constexpr int ENTRIES = T == 96 ? 2 : T == 64 ? 3 : T == 32 ? 4 : 8;
  static_assert(ENTRIES <= GROUPS, "a barrier set belongs to one group in flight");
  static constexpr int IB = T == 96 ? 1 : 2;
  static constexpr int PER = 2 / IB;                               // hand-offs per group
  static constexpr int ACT_BYTES = 2 * T * 128 * LIMBS;            // a stage of activations
  static constexpr int ACT_SLOTS = T * LIMBS >= 192 ? 2 : T * LIMBS == 128 ? 3 : T * LIMBS >= 64 ? 4 : 6;
  // The scale ring needs no barriers of its own.  A stage's scales count into its raw_full barrier, so whoever
  // sees the stage's sums sees them.  The scales of tile stage n are written once the converters have released
  // stage n - RAW_SLOTS; by then its operand slots were free, so the MMAs of stage n - RAW_SLOTS - TA_SLOTS / 2
  // were complete; those could start once the drain had released what was in their entries, the groups ENTRIES
  // before, so (ENTRIES + 1) / 2 stages further back everything has been read.
  static constexpr int SC_MORE = TA_SLOTS / 2 + (ENTRIES + 1) / 2 + 1;   // (and one to spare)
  static constexpr int RAW_SLOTS_FIT = (225 * 1024 - 2048 - ACT_SLOTS * ACT_BYTES - SC_MORE * SC_BYTES) / (RAW_BYTES + SC_BYTES);
  static constexpr int RAW_SLOTS = RAW_SLOTS_FIT < 9 ? RAW_SLOTS_FIT : 9;
  static constexpr int SC_SLOTS = RAW_SLOTS + SC_MORE;
  // Drain warpgroups: up to 32 tokens there is little to drain, and two groups (all tokens of a tile per warp) take
  // a whole stage in one round of latency; from 64 on the drain needs sixteen warps and the registers.  One
  // converter group: every further warp costs its own waits and ring steps, and issue slots are what the
  // kernel runs short of (0.64 of them were taken with sixteen converter warps at 16 tokens).
  static constexpr int DRAIN_WGS = T <= 32 ? 2 : 4;
  static constexpr int WGS = 2 + DRAIN_WGS;
  static constexpr int THREADS = WGS * 128;
  // registers per thread after the split (warpgroups: single roles, converters, drain); the sum stays within
  // what the block is launched with: an SM's 65536 registers over its threads, in steps of 8
  static constexpr int REGS_LAUNCH = 65536 / THREADS / 8 * 8;
  static constexpr int REGS_DRAIN = T <= 32 ? 168 : T == 96 ? 96 : 88;
  static constexpr int REGS_MISC = T == 96 ? 40 : 56;
  static constexpr int REGS_CONV = T <= 32 ? 96 : T == 96 ? 56 : 72;
  static_assert(REGS_MISC + REGS_CONV + DRAIN_WGS * REGS_DRAIN <= WGS * REGS_LAUNCH, "register split");
  static constexpr int ACC_COL0 = TA_SLOTS * TA_SLOT_COLS;
  static constexpr size_t SMEM = 1024 + (size_t)RAW_SLOTS * RAW_BYTES + (size_t)ACT_SLOTS * ACT_BYTES +
                                 (size_t)SC_SLOTS * SC_BYTES + 1024;
  static_assert(SMEM <= 227 * 1024 && SMEM > 114 * 1024, "shared memory: one CTA per SM, since it takes all of tensor memory");
  static constexpr int ENTRY_COLS = 2 * T;
  static_assert(ACC_COL0 + ENTRIES * ENTRY_COLS <= (int)TMEM_COLS, "TMEM budget");
};

// The wide form, for many tokens: a unit is one row tile x 2 T tokens (x a K split), so that converted weights serve twice as
// many tokens.  Half a stage is one slot of the operand ring and of the activation ring.
template <int T, int LIMBS>
struct WideCfg {
  // One MMA of N = 2 T for both halves of the tokens, a block for each MMA warp, with one plane; an MMA warp for each
  // half of the tokens with two, where a joint block would be complete only after twice the time.
  static constexpr bool JOINT = LIMBS == 1;
  static constexpr int ENTRIES = 2;                                // accumulator entries: blocks of 2 T columns
  static constexpr int FULLS = JOINT ? ENTRIES : 2 * ENTRIES;      // hand-offs of a block: together, or each half of the tokens
  static constexpr int ACT_BYTES = 2 * T * 128 * LIMBS;
  static constexpr int ACT_SLOTS = T == 96 ? (LIMBS == 2 ? 3 : 5) : (LIMBS == 2 ? 4 : 6);
  // Scales need no barriers of their own (see TcCfg): those of stage n are written once the converters have released stage
  // n - RAW_SLOTS; its operand slots were free by then, so all MMAs of stage n - RAW_SLOTS - 2 were complete, and the last
  // two of its blocks needed the entries of the first two, whose readers had that stage's scales.
  static constexpr int SC_MORE = 3;                                // (one to spare)
  static constexpr int RAW_SLOTS_FIT = (225 * 1024 - 2048 - ACT_SLOTS * ACT_BYTES - SC_MORE * SC_BYTES) / (RAW_BYTES + SC_BYTES);
  static constexpr int RAW_SLOTS = RAW_SLOTS_FIT < 5 ? RAW_SLOTS_FIT : 5;
  static constexpr int SC_SLOTS = RAW_SLOTS + SC_MORE;
  static constexpr int CONV_WARP0 = 4, DRAIN_WARP0 = 8, DRAIN_WARPS = 8;   // four single-role warps, then these
  static constexpr int THREADS = (DRAIN_WARP0 + DRAIN_WARPS) * 32;
  // T sums a thread, and 48 (32) columns on their way to them.  Not one register of that may be spilled: with 9 % of the
  // instructions spills the kernel took half as long again.
  static constexpr int REGS_MISC = 64, REGS_CONV = 80, REGS_DRAIN = 184;
  static_assert(4 * REGS_MISC + 4 * REGS_CONV + DRAIN_WARPS * REGS_DRAIN <= (DRAIN_WARP0 + DRAIN_WARPS) * (65536 / THREADS / 8 * 8), "register split");
  static constexpr int ACC_COL0 = 4 * TA_SLOT_COLS;
  static_assert(ACC_COL0 + ENTRIES * 2 * T <= (int)TMEM_COLS, "TMEM budget");
  static constexpr size_t SMEM = 1024 + (size_t)RAW_SLOTS * RAW_BYTES + (size_t)ACT_SLOTS * ACT_BYTES + (size_t)SC_SLOTS * SC_BYTES + 1024;
  static_assert(RAW_SLOTS >= 3 && SMEM <= 227 * 1024 && SMEM > 114 * 1024, "shared memory: one CTA per SM, since it takes all of tensor memory");
};

struct TcParams {
  const float* s;
  int64_t n, m;
  void* c;
  int c_dtype;
  ActOut c_act;
  int64_t ldc;
  const void* aux;
  int epilogue;
  float* partials;
  int splits;
  int stages_total;
  // Units: `pairs` x splits pair items, then `solos` x splits single tiles, each for mtiles token tiles.
  int pairs, solos, mtiles, group;
  int s_tiled;        // scales are [row tile][stage][128 rows][4] (always with tile-major weights)
  int wait_scales;    // the scales are the previous kernel's output too
  int stream_once;    // one token tile: the weights are not read again
  int* status;
};

struct TcUnit {
  int tile, ntile, split, st_begin, nst, mtile;
};
// CTAs that run side by side hold consecutive units: `group` token tiles of a row-tile pair, then the next
// pair, so that a wave of CTAs covers a near-square part of the output and both operands are
// shared through L2.
__device__ __forceinline__ TcUnit tc_unit(const TcParams& p, int u) {
  TcUnit r;
  const int pair_units = p.pairs * p.splits * p.mtiles;
  const bool solo = u >= pair_units;
  if (solo) u -= pair_units;
  int item = u;
  r.mtile = 0;
  if (p.mtiles > 1) {
    const int items = (solo ? p.solos : p.pairs) * p.splits;
    const int g = u / (items * p.group);                       // token-tile group
    u -= g * items * p.group;
    const int in_group = min(p.group, p.mtiles - g * p.group);  // the last group may be smaller
    item = u / in_group;
    r.mtile = g * p.group + (u - item * in_group);
  }
  int t = item;
  r.split = 0;
  r.st_begin = 0;
  r.nst = p.stages_total;
  if (p.splits > 1) {   // (a division takes a hundred cycles, and every role of a CTA starts with this)
    t = item / p.splits;
    r.split = item - t * p.splits;
    r.st_begin = r.split * p.stages_total / p.splits;
    r.nst = (r.split + 1) * p.stages_total / p.splits - r.st_begin;
  }
  r.tile = solo ? 2 * p.pairs + t : 2 * t;
  r.ntile = solo ? 1 : 2;
  return r;
}

// First failure wins: code in word 0, where it happened in words 1..5.
__device__ __forceinline__ void tc_report(int* status, int code, int stage, int nst) {
  if (atomicCAS(status, 0, code) == 0) {
    status[1] = blockIdx.x; status[2] = blockIdx.y; status[3] = stage; status[4] = nst; status[5] = threadIdx.x >> 5;
  }
}

// Position in a ring: slot, and the parity of the pass over it.
template <int N, int STEP = 1>
struct Ring {
  int slot;
  uint32_t ph;
  __device__ __forceinline__ explicit Ring(int first = 0, uint32_t phase = 0) : slot(first), ph(phase) {}
  __device__ __forceinline__ void next() {
    slot += STEP;
    const bool wrap = slot >= N;
    slot = wrap ? slot - N : slot;
    ph ^= wrap ? 1u : 0u;
  }
};

// 1-D bulk copy global -> shared, completion counted in bytes on an mbarrier; both addresses and the
// size are multiples of 16
__device__ __forceinline__ void bulk_load(uint32_t smem_dst, const void* gmem_src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_dst), "l"(gmem_src), "r"(bytes), "r"(bar)
               : "memory");
}

// N columns of a row into r[0 .. N)
template <int N>
__device__ __forceinline__ void tc_ld_cols(uint32_t taddr, uint32_t* r) {
  if constexpr (N > 32) {
    tc_ld_cols<32>(taddr, r);
    tc_ld_cols<N - 32>(taddr + 32, r + 32);
  } else if constexpr (N == 32) tc_ld_32x32b_x32(taddr, *reinterpret_cast<uint32_t(*)[32]>(r));
  else if constexpr (N == 24) {
    tc_ld_32x32b_x16(taddr, *reinterpret_cast<uint32_t(*)[16]>(r));
    tc_ld_32x32b_x8(taddr + 16, *reinterpret_cast<uint32_t(*)[8]>(r + 16));
  } else if constexpr (N == 16) tc_ld_32x32b_x16(taddr, *reinterpret_cast<uint32_t(*)[16]>(r));
  else if constexpr (N == 8) tc_ld_32x32b_x8(taddr, *reinterpret_cast<uint32_t(*)[8]>(r));
  else tc_ld_32x32b_x4(taddr, *reinterpret_cast<uint32_t(*)[4]>(r));
}
// tcgen05.wait::ld, and the loaded registers tied to this point: no use of them moves above it
template <int N>
__device__ __forceinline__ void tc_loaded(uint32_t (&r)[N]) {
  tc_wait_ld();
#pragma unroll
  for (int i = 0; i < N; ++i) asm volatile("" : "+r"(r[i]));
}
template <int N>
__device__ __forceinline__ void regs_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N>
__device__ __forceinline__ void regs_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

// sum += s * (columns of a block), two-wide f32 FMAs
template <int N>
__device__ __forceinline__ void add_cols(float2* sum, float s, const uint32_t* b) {
  const float2 s2 = make_float2(s, s);
#pragma unroll
  for (int x = 0; x < N / 2; ++x)
    sum[x] = __ffma2_rn(s2, make_float2(__uint_as_float(b[2 * x]), __uint_as_float(b[2 * x + 1])), sum[x]);
}

// HC columns each of the BLKS blocks at `ta` (blocks are T columns apart); `release` runs once all are read.
template <int HC, int BLKS, int T, class Release>
__device__ __forceinline__ void drain_blocks(float2* sum, uint32_t ta, const float* s, Release release) {
  if constexpr (HC * BLKS <= (T <= 32 ? 64 : 32)) {   // few columns: all of them in one round of latency
    uint32_t b[HC * BLKS];
#pragma unroll
    for (int k = 0; k < BLKS; ++k) tc_ld_cols<HC>(ta + k * T, b + k * HC);
    tc_loaded(b);
    release();
#pragma unroll
    for (int k = 0; k < BLKS; ++k) add_cols<HC>(sum, s[k], b + k * HC);
  } else {
    constexpr int CH = HC <= 32 ? HC : HC / 2;
#pragma unroll
    for (int k = 0; k < BLKS; ++k) {
#pragma unroll
      for (int c = 0; c < HC / CH; ++c) {
        uint32_t b[CH];
        tc_ld_cols<CH>(ta + k * T + c * CH, b);
        tc_loaded(b);
        if (k == BLKS - 1 && c == HC / CH - 1) release();
        add_cols<CH>(sum + c * (CH / 2), s[k], b);
      }
    }
  }
}

// 64 bytes of a row of weights in shared memory (four chunks) -> fp16 in an operand slot.  Exact: see cvt_pair.
template <bool TILED>
__device__ __forceinline__ void convert_half(const uint4 (&wv)[4], uint32_t t_dst) {
  uint32_t o[32];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const uint32_t ws[4] = {wv[c].x, wv[c].y, wv[c].z, wv[c].w};
#pragma unroll
    for (int wi = 0; wi < 4; ++wi) {
      const uint32_t w = TILED ? ws[wi] : ws[wi] ^ 0x80808080u;   // tile-major bytes hold q + 128 already
      o[c * 8 + 2 * wi] = cvt_pair(w, 0x4140);
      o[c * 8 + 2 * wi + 1] = cvt_pair(w, 0x4342);
    }
  }
  tc_st_32x32b_x32(t_dst, o);
}

// A thread's HC sums of output column n, tokens m0 ..: a warp stores 32 consecutive columns of a token at a time.
// What is chosen at run time (output form, whether all tokens exist) is chosen once, and a row's address is the
// last one's plus the stride: with both inside the loop the epilogue of one tile took 5800 cycles.
template <int ROWS, class Put>
__device__ __forceinline__ void each_row(int rows, Put put) {
  if (rows >= ROWS) {
#pragma unroll
    for (int x = 0; x < ROWS; ++x) put(x);
  } else {
#pragma unroll
    for (int x = 0; x < ROWS; ++x)
      if (x < rows) put(x);
  }
}
template <int ROWS, class Value>
__device__ __forceinline__ void put_rows(const TcParams& p, int64_t at, int rows, Value value) {
  const int64_t ld = p.ldc;
  if (p.c_dtype == LOGOS_F32) {
    float* d = reinterpret_cast<float*>(p.c) + at;
    each_row<ROWS>(rows, [&](int x) { *d = value(x); d += ld; });
  } else if (p.c_dtype == LOGOS_BF16) {
    __nv_bfloat16* d = reinterpret_cast<__nv_bfloat16*>(p.c) + at;
    each_row<ROWS>(rows, [&](int x) { *d = __float2bfloat16_rn(value(x)); d += ld; });
  } else if (p.c_dtype == LOGOS_F16) {
    __half* d = reinterpret_cast<__half*>(p.c) + at;
    each_row<ROWS>(rows, [&](int x) { *d = __float2half_rn(value(x)); d += ld; });
  } else if ((p.m + ROWS) * ld < (1ll << 30)) {
    // planes two tokens a conversion, addresses by 32-bit offsets (1088 x 9728 x 896 with SwiGLU: 62.8 -> 59.9 us, by ncu)
    __half* const hi = p.c_act.hi;
    __half* const lo = p.c_act.lo;
    const bool two = p.c_act.mode == LOGOS_F32, rounded = p.c_act.mode == LOGOS_BF16;
    uint32_t off = (uint32_t)at;
    const uint32_t step = (uint32_t)ld;
    auto put = [&](int x) {
      uint32_t h, l;
      float2 v = make_float2(value(x), value(x + 1));
      if (rounded) v = __bfloat1622float2(__floats2bfloat162_rn(v.x, v.y));
      act_words(v, &h, &l);
      hi[off] = __ushort_as_half((unsigned short)h);
      if (two) lo[off] = __ushort_as_half((unsigned short)l);
      off += step;
      if (x + 1 < rows) {
        hi[off] = __ushort_as_half((unsigned short)(h >> 16));
        if (two) lo[off] = __ushort_as_half((unsigned short)(l >> 16));
      }
      off += step;
    };
    if (rows >= ROWS) {
#pragma unroll
      for (int x = 0; x < ROWS; x += 2) put(x);
    } else {
#pragma unroll
      for (int x = 0; x < ROWS; x += 2)
        if (x < rows) put(x);
    }
  } else {
    ActOut o = p.c_act;
    o.hi += at;
    if (o.mode == LOGOS_F32) o.lo += at;
    each_row<ROWS>(rows, [&](int x) { act_store(o, 0, value(x)); o.hi += ld; o.lo += ld; });
  }
}
template <int HC>
__device__ __forceinline__ void store_tile(const TcParams& p, const float2* acc, int split, int64_t n, int64_t m0, int lane) {
  const int rows = (int)(p.m - m0 < HC ? p.m - m0 : HC);
  auto sum = [&](int e) { return (e & 1) ? acc[e >> 1].y : acc[e >> 1].x; };
  if (p.splits > 1) {
    float* d = p.partials + ((int64_t)split * p.m + m0) * p.n + n;
    if (n < p.n) each_row<HC>(rows, [&](int x) { *d = sum(x); d += p.n; });
  } else if (p.epilogue == EPI_SWIGLU) {
    // rows (2j, 2j+1) are (gate_j, up_j): neighbouring lanes.  The even lane takes the first half of the
    // tokens, the odd lane the second half.
    const int par = lane & 1, first = par * (HC / 2);
    float g[HC / 2], up[HC / 2];
    bool plain = true;
#pragma unroll
    for (int x = 0; x < HC / 2; ++x) {
      const float a = sum(x), b = sum(x + HC / 2);
      const float recv = __shfl_xor_sync(0xffffffffu, par ? a : b, 1);
      g[x] = par ? recv : a;
      up[x] = par ? b : recv;
      plain &= silu_plain(g[x]);
    }
    // One decision for all: a division with its special operands behind a branch costs a hundred cycles a value
    // (2048 x 37888 x 3584: 849 -> 814 us).
    if (__all_sync(0xffffffffu, plain)) {
#pragma unroll
      for (int x = 0; x < HC / 2; ++x) g[x] = __fmul_rn(silu_markstein(g[x]), up[x]);
    } else {
#pragma unroll
      for (int x = 0; x < HC / 2; ++x) g[x] = __fmul_rn(silu_f(g[x]), up[x]);
    }
    if ((n | 1) < p.n) put_rows<HC / 2>(p, (m0 + first) * p.ldc + (n >> 1), rows - first, [&](int x) { return g[x]; });
  } else if (n < p.n) {
    const int64_t at = m0 * p.ldc + n;
    if (p.epilogue == EPI_RESIDUAL) {
      const __nv_bfloat16* r = reinterpret_cast<const __nv_bfloat16*>(p.aux) + at;   // only bf16 results have a residual
      __nv_bfloat16* d = reinterpret_cast<__nv_bfloat16*>(p.c) + at;
      each_row<HC>(rows, [&](int x) {
        *d = __float2bfloat16_rn(__fadd_rn(sum(x), __bfloat162float(*r)));
        r += p.ldc;
        d += p.ldc;
      });
    } else {
      put_rows<HC>(p, at, rows, [&](int x) { return sum(x); });
    }
  }
}

template <int T, int LIMBS, bool TILED>
__global__ void __launch_bounds__(TcCfg<T, LIMBS>::THREADS, 1)
q8_gemm_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_a,
                  const __grid_constant__ CUtensorMap map_s, const TcParams p) {
  using Cfg = TcCfg<T, LIMBS>;
  constexpr int ENTRIES = Cfg::ENTRIES, IB = Cfg::IB, PER = Cfg::PER, ACT_SLOTS = Cfg::ACT_SLOTS, RAW_SLOTS = Cfg::RAW_SLOTS,
                SC_SLOTS = Cfg::SC_SLOTS;

  // Shared memory by 32-bit window addresses: rings of slots, then the barriers.
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = (smem_u32(smem_raw) + 1023u) & ~1023u;       // [RAW_SLOTS] x 16 KB
  const uint32_t act = raw + RAW_SLOTS * RAW_BYTES;                 // [ACT_SLOTS] x ACT_BYTES
  const uint32_t scl = act + ACT_SLOTS * Cfg::ACT_BYTES;            // [SC_SLOTS] x 2 KB
  const uint32_t raw_full = scl + SC_SLOTS * SC_BYTES;              // barriers, 8 bytes each: [RAW_SLOTS]
  const uint32_t raw_empty = raw_full + 8 * RAW_SLOTS;
  const uint32_t act_full = raw_empty + 8 * RAW_SLOTS;              // [ACT_SLOTS]
  const uint32_t act_empty = act_full + 8 * ACT_SLOTS;
  const uint32_t ta_full = act_empty + 8 * ACT_SLOTS;               // [TA_SLOTS]
  const uint32_t ta_empty = ta_full + 8 * TA_SLOTS;
  const uint32_t acc_full = ta_empty + 8 * TA_SLOTS;                // [GROUPS][PER]
  const uint32_t acc_empty = acc_full + 8 * GROUPS * PER;
  __shared__ uint32_t tmem_slot;

  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;

  // a kernel that gave up earlier left a code behind: do not start new work on top of it
  // (one thread reads, everyone takes the same decision)
  __shared__ int prior_status;
  constexpr int NBARS = 2 * (RAW_SLOTS + ACT_SLOTS + TA_SLOTS + GROUPS * PER);
  static_assert(NBARS <= 128, "one barrier a thread");
  if (warp >= CONV_WARP0 && tid - CONV_WARP0 * 32 < NBARS) {
    const int i = tid - CONV_WARP0 * 32;
    const uint32_t bar = raw_full + 8 * i;
    uint32_t count = 1;                                             // TMA and tcgen05.commit arrive once
    if (bar >= raw_empty && bar < act_full) count = 4;              // the converter warps
    else if (bar >= ta_full && bar < ta_empty) count = 4;
    else if (bar >= act_empty && bar < ta_full) count = 2;          // a commit of each MMA warp
    else if (bar >= acc_empty) count = 4 * Cfg::DRAIN_WGS;          // the drain warps
    mbar_init(bar, count);
    fence_barrier_init();
  }
  if (tid == 0) prior_status = *reinterpret_cast<volatile int*>(p.status);
  if (warp == 1 && lane == 0) {
    prefetch_tensormap(&map_q);
    prefetch_tensormap(&map_a);
    if (!p.s_tiled) prefetch_tensormap(&map_s);
  }
  if (warp == 3) {
    tmem_alloc(&tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  // Dependent launch: this CTA holds its SM's shared and tensor memory by now, so a successor's
  // CTAs may be scheduled wherever room is left.  Weights and scales are read without waiting
  // for the previous kernel (nothing in a decode step writes them); the activation producer
  // and the drain warps (the only ones that touch what other kernels write) wait first.
  pdl_trigger();
  // nothing to do on top of an earlier failure
  const int pair_units = prior_status != 0 ? 0 : p.pairs * p.splits * p.mtiles;
  const int units = prior_status != 0 ? 0 : (p.pairs + p.solos) * p.splits * p.mtiles;

  bool ok = true;
  uint32_t since = wait_start();   // see mbar_wait; a new limit every unit

  // Every role walks the same sequence of groups: units, stages, the unit's tiles, halves.
  if (warp < 4) {
    regs_dec<Cfg::REGS_MISC>();
    if (warp == 0) {
      // ------------------------------------------------------------ weight and scale producer
      // The single-role warps run their loops with all lanes and issue from one elected lane: addresses and
      // descriptors stay in uniform registers.  Under a plain `lane == 0` branch a TMA instruction took its
      // thread about 230 cycles (a stage's four activation loads 1100, more than the stage itself) and a group
      // of MMAs three times as long.
      if (p.wait_scales) pdl_wait();
      const uint64_t pol = p.stream_once ? policy_evict_first() : policy_evict_normal();
      Ring<RAW_SLOTS> r;
      Ring<SC_SLOTS> c;
      for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
        const TcUnit it = tc_unit(p, u);
        since = wait_start();
        for (int i = it.st_begin; i < it.st_begin + it.nst && ok; ++i) {
          for (int j = it.tile; j < it.tile + it.ntile; ++j) {
            const int block = j * p.stages_total + i;   // of a tile-major array
            const uint32_t bar = raw_full + 8 * r.slot;
            mbar_wait(raw_empty + 8 * r.slot, r.ph ^ 1u, &since);
            if (elect_one()) {
              mbar_arrive_expect_tx(bar, RAW_BYTES + SC_BYTES);
              // row-major weights: tile (row, stage) of a [N][K] map; tile-major: 128 rows of 128 bytes at
              // row block * 128 of a [tiles * stages * 128][128 B] map
              if (TILED) tma_load_2d_hint(raw + r.slot * RAW_BYTES, &map_q, bar, 0, block * TC_ROWS, pol);
              else tma_load_2d_hint(raw + r.slot * RAW_BYTES, &map_q, bar, i * TC_KSTAGE, j * TC_ROWS, pol);
              // the stage's scales, four per row: tile-major they are 2 contiguous KB, row-major a
              // [128 rows][4] box of the [N][K/32] matrix (rows past N read as zero)
              if (TILED || p.s_tiled) bulk_load(scl + c.slot * SC_BYTES, p.s + (int64_t)block * (TC_ROWS * 4), SC_BYTES, bar);
              else tma_load_2d(scl + c.slot * SC_BYTES, &map_s, bar, i * 4, j * TC_ROWS);
            }
            __syncwarp();
            r.next();
            c.next();
          }
          if (since == WAIT_OVER) {
            if (lane == 0) tc_report(p.status, 2010, i, it.nst);
            ok = false;
          }
        }
      }
    } else if (warp == 1) {
      // ------------------------------------------------------------ activation producer
      pdl_wait();  // the activations are the previous kernel's output
      const uint64_t pol = policy_evict_last();
      Ring<ACT_SLOTS> r;
      for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
        const TcUnit it = tc_unit(p, u);
        since = wait_start();
        const int m0 = it.mtile * T;
        for (int i = it.st_begin; i < it.st_begin + it.nst && ok; ++i) {
          const uint32_t bar = act_full + 8 * r.slot;
          mbar_wait(act_empty + 8 * r.slot, r.ph ^ 1u, &since);
          if (elect_one()) {
            mbar_arrive_expect_tx(bar, Cfg::ACT_BYTES);
            tma_load_4d_hint(act + r.slot * Cfg::ACT_BYTES, &map_a, bar, 0, m0, 2 * i, 0, pol);
          }
          __syncwarp();
          r.next();
          if (since == WAIT_OVER) {
            if (lane == 0) tc_report(p.status, 2020, i, it.nst);
            ok = false;
          }
        }
      }
    } else {
      // ------------------------------------------------------------ MMA issuers, one warp per half of a stage
      // The barriers a group needs are polled together: one round of latency, not three.
      constexpr uint32_t idesc = make_idesc_f16(0, 0, TC_ROWS, T);
      const int half = warp - 2;
      const uint64_t bdesc_first = make_desc_sw128(act + half * T * 128);
      Ring<ACT_SLOTS> ra;
      Ring<TA_SLOTS, 2> rt(half);
      Ring<GROUPS, 2> rf(half);                                    // the group's own barriers
      Ring<GROUPS, 2> re((half + GROUPS - ENTRIES) % GROUPS, 1u);  // those of the entry's previous group
      Ring<ENTRIES, 2> rd(half % ENTRIES);                         // the entry
      for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
        const TcUnit it = tc_unit(p, u);
        since = wait_start();
        for (int i = 0; i < it.nst; ++i) {
          const uint64_t bdesc0 = bdesc_first + (uint32_t)(ra.slot * (Cfg::ACT_BYTES >> 4));   // start address field: no carry out of it
          for (int j = 0; j < it.ntile; ++j) {
            const uint32_t a0 = tmem_base + rt.slot * TA_SLOT_COLS;
            const uint32_t free_bar = acc_empty + 8 * PER * re.slot, full_bar = acc_full + 8 * PER * rf.slot;
#pragma unroll
            for (int k = 0; k < PER; ++k) {
              if (k > 0) mbar_wait(free_bar + 8 * k, re.ph, &since);
              else if (j == 0) mbar_wait3(act_full + 8 * ra.slot, ra.ph, ta_full + 8 * rt.slot, rt.ph, free_bar, re.ph, &since);
              else mbar_wait2(ta_full + 8 * rt.slot, rt.ph, free_bar, re.ph, &since);
              tc_fence_after();
              const uint32_t d0 = tmem_base + Cfg::ACC_COL0 + rd.slot * Cfg::ENTRY_COLS + k * IB * T;
              if (elect_one()) {
                // Per block: d = q * lo' first, then d = q * hi + d * 2^-11 (the residual plane is folded in by the
                // accumulator scaling of the MMA itself, from one copy of the weights).
#pragma unroll
                for (int v = 0; v < 2 * LIMBS; ++v) {
#pragma unroll
                  for (int b = 0; b < IB; ++b) {
                    const int l = (LIMBS == 2) ? 1 - (v >> 1) : 0;
                    const int kk = (k * IB + b) * 2 + (v & 1);     // K = 16 step inside the half stage
                    const uint64_t bdesc = bdesc0 + (uint32_t)((l * 2 * T * 128 + kk * 32) >> 4);
                    if (LIMBS == 2 && v == 2) tc_mma_f16_ts_scaled_d<11>(d0 + b * T, a0 + kk * 8, bdesc, idesc);
                    else if (v == 0) tc_mma_f16_ts<false>(d0 + b * T, a0 + kk * 8, bdesc, idesc);
                    else tc_mma_f16_ts<true>(d0 + b * T, a0 + kk * 8, bdesc, idesc);
                  }
                }
                tc_commit(full_bar + 8 * k);
                if (k == PER - 1) {
                  tc_commit(ta_empty + 8 * rt.slot);
                  if (j + 1 == it.ntile) tc_commit(act_empty + 8 * ra.slot);   // free once these MMAs have completed
                }
              }
              __syncwarp();
            }
            rt.next();
            rf.next();
            re.next();
            rd.next();
          }
          ra.next();
          if (since == WAIT_OVER) {
            if (lane == 0) tc_report(p.status, 2030, i, it.nst);
            ok = false;
            break;
          }
        }
      }
    }
  } else if (warp < DRAIN_WARP0) {
    // ------------------------------------------------------------ converters: int8 smem -> fp16 TMEM
    regs_dec<Cfg::REGS_CONV>();
    const int qd = warp & 3;
    const uint32_t row = qd * 32 + lane;
    const uint32_t t_lane = tmem_base + ((uint32_t)(qd * 32) << 16);
    // the row's eight 16-byte chunks: chunk c sits at c ^ (row & 7) (128-byte swizzle)
    uint32_t off[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) off[c] = raw + swz128(row, c);   // chunk c + 4: bit 6 of the address flipped
    Ring<RAW_SLOTS> r;
    Ring<TA_SLOTS, 2> a(0, 1u);   // a stage takes slots a and a + 1
    for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
      const TcUnit it = tc_unit(p, u);
      since = wait_start();
      const int count = it.nst * it.ntile;
      for (int i = 0; i < count && ok; ++i) {
        // everything the stage needs in one wait, all its loads together, one wait for its stores: a round of
        // latency costs as much as fifty instructions
        mbar_wait3(raw_full + 8 * r.slot, r.ph, ta_empty + 8 * a.slot, a.ph, ta_empty + 8 * (a.slot + 1), a.ph, &since);
        tc_fence_after();
        uint4 wv[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) wv[c] = lds_v4((off[c & 3] ^ (c & 4 ? 64u : 0u)) + r.slot * RAW_BYTES);
        const uint32_t t_dst = t_lane + a.slot * TA_SLOT_COLS;
#pragma unroll
        for (int c2 = 0; c2 < 2; ++c2) {
          uint32_t o[32];
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const uint4 w4 = wv[c2 * 4 + c];
            const uint32_t ws[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
            for (int wi = 0; wi < 4; ++wi) {
              const uint32_t w = TILED ? ws[wi] : ws[wi] ^ 0x80808080u;   // tile-major bytes hold q + 128 already
              o[c * 8 + 2 * wi] = cvt_pair(w, 0x4140);
              o[c * 8 + 2 * wi + 1] = cvt_pair(w, 0x4342);
            }
          }
          tc_st_32x32b_x32(t_dst + c2 * 32, o);
        }
        mbar_arrive_if(raw_empty + 8 * r.slot, lane == 0);
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        mbar_arrive_if(ta_full + 8 * a.slot, lane == 0);
        mbar_arrive_if(ta_full + 8 * (a.slot + 1), lane == 0);
        a.next();
        r.next();
        if (since == WAIT_OVER) {
          if (lane == 0) tc_report(p.status, 2040, i, count);
          ok = false;
        }
      }
    }
  } else {
    // ------------------------------------------------------------ drain + epilogue
    regs_inc<Cfg::REGS_DRAIN>();
    const int qd = warp & 3;
    constexpr int DW = 4 * Cfg::DRAIN_WGS;
    constexpr int SHARE = Cfg::DRAIN_WGS / 2;       // warps that share a lane quarter of a tile of a pair
    const int g = (warp - DRAIN_WARP0) / (DW / 2);  // the tile of a pair
    const int th = ((warp - DRAIN_WARP0) >> 2) % SHARE;
    const int nl = qd * 32 + lane;                  // row of the tile this thread drains
    const uint32_t t_lane = tmem_base + ((uint32_t)(qd * 32) << 16) + Cfg::ACC_COL0;
    const uint32_t s_lane = scl + nl * 16;
    pdl_wait();  // before any write to global memory (nothing to drain before the activations are in anyway)
    int ent = (2 * g) % ENTRIES;     // entry of the next group
    int rc = g;                      // scale slot of the next stage
    int grp = 2 * g;                 // barrier set of the next stage's first group, and the parity of its phase
    uint32_t ph = 0;
    auto step = [](int& v, int by, int n) {
      v += by;
      if (v >= n) v -= n;
    };
    // one stage of a tile, from this warp's first column `col` on
    auto drain_stage = [&](auto hc, float2* sum, uint32_t col, auto arrivals) {
      float s[4];
      auto scales = [&] {
        const uint4 sc = lds_v4(s_lane + rc * SC_BYTES);
        s[0] = __uint_as_float(sc.x); s[1] = __uint_as_float(sc.y); s[2] = __uint_as_float(sc.z); s[3] = __uint_as_float(sc.w);
      };
      if constexpr (T <= 32 && 4 * hc <= 64) {   // few columns: the whole stage in one round of latency
        const uint32_t at0 = t_lane + col + ent * Cfg::ENTRY_COLS;
        step(ent, 1, ENTRIES);
        const uint32_t at1 = t_lane + col + ent * Cfg::ENTRY_COLS;
        step(ent, 1, ENTRIES);
        mbar_wait2(acc_full + 8 * grp, ph, acc_full + 8 * (grp + 1), ph, &since);
        tc_fence_after();
        uint32_t b[4 * hc];
        tc_ld_cols<hc>(at0, b);
        tc_ld_cols<hc>(at0 + T, b + hc);
        tc_ld_cols<hc>(at1, b + 2 * hc);
        tc_ld_cols<hc>(at1 + T, b + 3 * hc);
        scales();
        tc_loaded(b);
        tc_fence_before();
        __syncwarp();
        mbar_arrive_n_if<arrivals>(acc_empty + 8 * grp, lane == 0);
        mbar_arrive_n_if<arrivals>(acc_empty + 8 * (grp + 1), lane == 0);
#pragma unroll
        for (int k = 0; k < 4; ++k) add_cols<hc>(sum, s[k], b + k * hc);
      } else {
        if (PER == 1) mbar_wait2(acc_full + 8 * grp, ph, acc_full + 8 * (grp + 1), ph, &since);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint32_t at = t_lane + col + ent * Cfg::ENTRY_COLS;
          step(ent, 1, ENTRIES);
#pragma unroll
          for (int k = 0; k < PER; ++k) {
            const uint32_t bar = 8 * (PER * (grp + h) + k);
            if (PER > 1) mbar_wait(acc_full + bar, ph, &since);
            if (PER > 1 || h == 0) tc_fence_after();
            if (h == 0 && k == 0) scales();
            drain_blocks<hc, IB, T>(sum, at + k * IB * T, s + h * 2 + k * IB, [&] {
              tc_fence_before();
              __syncwarp();
              mbar_arrive_n_if<arrivals>(acc_empty + bar, lane == 0);
            });
          }
        }
      }
    };
    constexpr std::integral_constant<int, T / SHARE> pair_cols{};
    constexpr std::integral_constant<int, T / Cfg::DRAIN_WGS> solo_cols{};
    constexpr std::integral_constant<int, 1> one{};
    constexpr std::integral_constant<int, 2> two{};   // half of the drain warps stand for all of them

    int u = blockIdx.x;
    for (; u < pair_units && ok; u += gridDim.x) {
      const TcUnit it = tc_unit(p, u);
      since = wait_start();
      float2 acc[pair_cols / 2];
#pragma unroll
      for (int x = 0; x < pair_cols / 2; ++x) acc[x] = make_float2(0.f, 0.f);
      for (int i = 0; i < it.nst && since != WAIT_OVER; ++i) {
        drain_stage(pair_cols, acc, th * pair_cols, two);
        step(ent, 2 % ENTRIES, ENTRIES);            // past the other tile's two groups
        step(rc, 2, SC_SLOTS);
        grp ^= 4;
        ph ^= (uint32_t)(grp < 4);
      }
      if (since == WAIT_OVER) {
        if (lane == 0) tc_report(p.status, 2050, 0, it.nst);
        ok = false;
        break;
      }
      store_tile<pair_cols>(p, acc, it.split, (int64_t)(it.tile + g) * TC_ROWS + nl, (int64_t)it.mtile * T + th * pair_cols, lane);
    }
    // From here on a warp waits for barriers that only the other tile's warps have followed so far: once all have
    // come this far, their phases of the pair units are over.  (Every drain warp passes here exactly once.)
    asm volatile("bar.sync 1, %0;" ::"n"(DW * 32) : "memory");
    ent = (ent + 2 * ENTRIES - 2 * g) % ENTRIES;
    rc = (rc + SC_SLOTS - g) % SC_SLOTS;
    grp -= 2 * g;
    for (; u < units && ok; u += gridDim.x) {
      const TcUnit it = tc_unit(p, u);
      since = wait_start();
      float2 acc[solo_cols / 2];
#pragma unroll
      for (int x = 0; x < solo_cols / 2; ++x) acc[x] = make_float2(0.f, 0.f);
      const uint32_t col = (SHARE * g + th) * solo_cols;
      for (int i = 0; i < it.nst && since != WAIT_OVER; ++i) {
        drain_stage(solo_cols, acc, col, one);
        step(rc, 1, SC_SLOTS);
        step(grp, 2, GROUPS);
        ph ^= (uint32_t)(grp == 0);
      }
      if (since == WAIT_OVER) {
        if (lane == 0) tc_report(p.status, 2051, 0, it.nst);
        ok = false;
        break;
      }
      store_tile<solo_cols>(p, acc, it.split, (int64_t)it.tile * TC_ROWS + nl, (int64_t)it.mtile * T + col, lane);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 3) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// The wide form (WideCfg).  The same arithmetic in the same order as the kernel above, so the same bits.
//
// What bounds it with many tokens: a block's sums go through registers once, 96 columns x 128 rows for each half of the
// tokens, and two entries of tensor memory are all there is room for.  A block takes 500 cycles: 96 to 192 of MMA, about 160
// until its completion is seen, two loads of 48 columns with the FMAs of the first half between them, and the MMA warp's
// wake-up.  So eight drain warps with a whole channel's columns each instead of sixteen with half of them (hand-offs are what
// costs: a poll of a ready barrier is 80 cycles, an arrival seven for each warp), the second load released before its FMAs.
// Against pairs of row tiles (calls in a row, 1000 W, bf16 2048 x 37888 x 3584 / f32 4096 x 10240 x 5120, us): 965 -> 777 / 983 -> 852.
// A joint MMA for both planes 872, two MMA warps for one plane 795; loads of 16 columns, each ahead of the FMAs of the one
// before, 815 / 887.
template <int T, int LIMBS, bool TILED>
__global__ void __launch_bounds__(WideCfg<T, LIMBS>::THREADS, 1)
q8_gemm_wide_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_a,
                    const __grid_constant__ CUtensorMap map_s, const TcParams p) {
  using Cfg = WideCfg<T, LIMBS>;
  constexpr bool JOINT = Cfg::JOINT;
  constexpr int FULLS = Cfg::FULLS, ACT_SLOTS = Cfg::ACT_SLOTS, RAW_SLOTS = Cfg::RAW_SLOTS, SC_SLOTS = Cfg::SC_SLOTS;

  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = (smem_u32(smem_raw) + 1023u) & ~1023u;       // [RAW_SLOTS] x 16 KB
  const uint32_t act = raw + RAW_SLOTS * RAW_BYTES;                 // [ACT_SLOTS] x ACT_BYTES: [planes][2 T][64]
  const uint32_t scl = act + ACT_SLOTS * Cfg::ACT_BYTES;            // [SC_SLOTS] x 2 KB
  const uint32_t raw_full = scl + SC_SLOTS * SC_BYTES;              // barriers, 8 bytes each: [RAW_SLOTS]
  const uint32_t raw_empty = raw_full + 8 * RAW_SLOTS;
  const uint32_t act_full = raw_empty + 8 * RAW_SLOTS;              // [ACT_SLOTS]
  const uint32_t act_empty = act_full + 8 * ACT_SLOTS;
  const uint32_t ta_full = act_empty + 8 * ACT_SLOTS;               // [TA_SLOTS]
  const uint32_t ta_empty = ta_full + 8 * TA_SLOTS;
  const uint32_t acc_full = ta_empty + 8 * TA_SLOTS;                // [FULLS]
  const uint32_t acc_empty = acc_full + 8 * FULLS;
  __shared__ uint32_t tmem_slot;
  __shared__ int prior_status;

  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  constexpr int NBARS = 2 * (RAW_SLOTS + ACT_SLOTS + TA_SLOTS + FULLS);
  static_assert(NBARS <= 128, "one barrier a thread");
  if (warp >= Cfg::CONV_WARP0 && tid - Cfg::CONV_WARP0 * 32 < NBARS) {
    const int i = tid - Cfg::CONV_WARP0 * 32;
    const uint32_t bar = raw_full + 8 * i;
    uint32_t count = 1;                                                  // TMA and tcgen05.commit arrive once
    if (bar >= raw_empty && bar < act_full) count = 4;                   // the converter warps
    else if (bar >= act_empty && bar < ta_full) count = 2;               // a commit of each MMA warp
    else if (bar >= ta_full && bar < ta_empty) count = 4;
    else if (bar >= ta_empty && bar < acc_full) count = 2;
    else if (bar >= acc_empty) count = JOINT ? Cfg::DRAIN_WARPS : Cfg::DRAIN_WARPS / 2;
    mbar_init(bar, count);
    fence_barrier_init();
  }
  if (tid == 0) prior_status = *reinterpret_cast<volatile int*>(p.status);   // as above
  if (warp == 1 && lane == 0) {
    prefetch_tensormap(&map_q);
    prefetch_tensormap(&map_a);
    if (!p.s_tiled) prefetch_tensormap(&map_s);
  }
  if (warp == 3) {
    tmem_alloc(&tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  pdl_trigger();   // as above
  const int units = prior_status != 0 ? 0 : p.solos * p.splits * p.mtiles;

  bool ok = true;
  uint32_t since = wait_start();

  if (warp < Cfg::CONV_WARP0) {
    regs_dec<Cfg::REGS_MISC>();
    if (warp == 0) {
      // ------------------------------------------------------------ weight and scale producer
      if (p.wait_scales) pdl_wait();
      const uint64_t pol = p.stream_once ? policy_evict_first() : policy_evict_normal();
      Ring<RAW_SLOTS> r;
      Ring<SC_SLOTS> c;
      for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
        const TcUnit it = tc_unit(p, u);
        since = wait_start();
        for (int i = it.st_begin; i < it.st_begin + it.nst && ok; ++i) {
          const int block = it.tile * p.stages_total + i;   // of a tile-major array
          const uint32_t bar = raw_full + 8 * r.slot;
          mbar_wait(raw_empty + 8 * r.slot, r.ph ^ 1u, &since);
          if (elect_one()) {
            mbar_arrive_expect_tx(bar, RAW_BYTES + SC_BYTES);
            if (TILED) tma_load_2d_hint(raw + r.slot * RAW_BYTES, &map_q, bar, 0, block * TC_ROWS, pol);
            else tma_load_2d_hint(raw + r.slot * RAW_BYTES, &map_q, bar, i * TC_KSTAGE, it.tile * TC_ROWS, pol);
            if (TILED || p.s_tiled) bulk_load(scl + c.slot * SC_BYTES, p.s + (int64_t)block * (TC_ROWS * 4), SC_BYTES, bar);
            else tma_load_2d(scl + c.slot * SC_BYTES, &map_s, bar, i * 4, it.tile * TC_ROWS);
          }
          __syncwarp();
          r.next();
          c.next();
          if (since == WAIT_OVER) {
            if (lane == 0) tc_report(p.status, 2110, i, it.nst);
            ok = false;
          }
        }
      }
    } else if (warp == 1) {
      // ------------------------------------------------------------ activation producer, half a stage at a time
      pdl_wait();  // the activations are the previous kernel's output
      const uint64_t pol = policy_evict_last();
      Ring<ACT_SLOTS> r;
      for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
        const TcUnit it = tc_unit(p, u);
        since = wait_start();
        for (int i = 2 * it.st_begin; i < 2 * (it.st_begin + it.nst) && ok; ++i) {
          const uint32_t bar = act_full + 8 * r.slot;
          mbar_wait(act_empty + 8 * r.slot, r.ph ^ 1u, &since);
          if (elect_one()) {
            mbar_arrive_expect_tx(bar, Cfg::ACT_BYTES);
            tma_load_4d_hint(act + r.slot * Cfg::ACT_BYTES, &map_a, bar, 0, it.mtile * 2 * T, i, 0, pol);
          }
          __syncwarp();
          r.next();
          if (since == WAIT_OVER) {
            if (lane == 0) tc_report(p.status, 2120, i, it.nst);
            ok = false;
          }
        }
      }
      // the last commits land before the CTA ends
      for (int i = 0; i < ACT_SLOTS && ok; ++i) {
        mbar_wait(act_empty + 8 * r.slot, r.ph ^ 1u, &since);
        r.next();
      }
    } else {
      // ------------------------------------------------------------ MMA issuers
      constexpr uint32_t idesc = make_idesc_f16(0, 0, TC_ROWS, JOINT ? 2 * T : T);
      const int w = warp - 2;
      const uint64_t bdesc_first = make_desc_sw128(act + (JOINT ? 0 : w * T * 128));
      const uint32_t d_first = tmem_base + Cfg::ACC_COL0 + (JOINT ? 0 : w * T);
      const uint32_t bars = JOINT ? 0u : 8u * Cfg::ENTRIES * w;
      Ring<ACT_SLOTS> ra;
      Ring<TA_SLOTS> rt;
      uint32_t e_ph = 1;   // of both entries
      // block k of a half stage, into entry k; whether it begins and ends this warp's part of it
      auto block = [&](int k, bool first, bool last) {
        const uint64_t bdesc0 = bdesc_first + (uint32_t)(ra.slot * (Cfg::ACT_BYTES >> 4) + k * 4);   // start address field: no carry out of it
        const uint32_t a0 = tmem_base + rt.slot * TA_SLOT_COLS + k * 16, d0 = d_first + k * 2 * T;
        if (first) mbar_wait3_ready(act_full + 8 * ra.slot, ra.ph, ta_full + 8 * rt.slot, rt.ph, acc_empty + bars + 8 * k, e_ph, &since);
        else mbar_wait_ready(acc_empty + bars + 8 * k, e_ph, &since);
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int v = 0; v < 2 * LIMBS; ++v) {   // d = q * lo' first, then d = q * hi + d * 2^-11
            const int l = (LIMBS == 2) ? 1 - (v >> 1) : 0;
            const uint64_t bdesc = bdesc0 + (uint32_t)((l * 2 * T * 128 + (v & 1) * 32) >> 4);
            if (LIMBS == 2 && v == 2) tc_mma_f16_ts_scaled_d<11>(d0, a0 + (v & 1) * 8, bdesc, idesc);
            else if (v == 0) tc_mma_f16_ts<false>(d0, a0 + (v & 1) * 8, bdesc, idesc);
            else tc_mma_f16_ts<true>(d0, a0 + (v & 1) * 8, bdesc, idesc);
          }
          tc_commit(acc_full + bars + 8 * k);
          if (last) {
            tc_commit(ta_empty + 8 * rt.slot);
            tc_commit(act_empty + 8 * ra.slot);
          }
        }
        __syncwarp();
      };
      for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
        const TcUnit it = tc_unit(p, u);
        since = wait_start();
        for (int i = 0; i < 2 * it.nst; ++i) {
          if (JOINT) {
            block(w, true, true);
          } else {
            block(0, true, false);
            block(1, false, true);
          }
          e_ph ^= 1u;
          rt.next();
          ra.next();
          if (since == WAIT_OVER) break;
        }
        if (since == WAIT_OVER) {
          if (lane == 0) tc_report(p.status, 2130, 0, it.nst);
          ok = false;
        }
      }
    }
  } else if (warp < Cfg::DRAIN_WARP0) {
    // ------------------------------------------------------------ converters: int8 smem -> fp16 TMEM
    regs_dec<Cfg::REGS_CONV>();
    const int qd = warp & 3;
    const uint32_t row = qd * 32 + lane;
    const uint32_t t_lane = tmem_base + ((uint32_t)(qd * 32) << 16);
    uint32_t off[4];   // chunks of the row's first half, see above
#pragma unroll
    for (int c = 0; c < 4; ++c) off[c] = raw + swz128(row, c);
    Ring<RAW_SLOTS> r;
    Ring<TA_SLOTS, 2> a(0, 1u);   // a stage takes slots a and a + 1
    for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
      const TcUnit it = tc_unit(p, u);
      since = wait_start();
      for (int i = 0; i < it.nst && since != WAIT_OVER; ++i) {
        mbar_wait3_ready(raw_full + 8 * r.slot, r.ph, ta_empty + 8 * a.slot, a.ph, ta_empty + 8 * (a.slot + 1), a.ph, &since);
        tc_fence_after();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint4 wv[4];
#pragma unroll
          for (int c = 0; c < 4; ++c) wv[c] = lds_v4((off[c] ^ (h ? 64u : 0u)) + r.slot * RAW_BYTES);
          convert_half<TILED>(wv, t_lane + (a.slot + h) * TA_SLOT_COLS);
        }
        mbar_arrive_if(raw_empty + 8 * r.slot, lane == 0);
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        mbar_arrive_if(ta_full + 8 * a.slot, lane == 0);
        mbar_arrive_if(ta_full + 8 * (a.slot + 1), lane == 0);
        a.next();
        r.next();
      }
      if (since == WAIT_OVER) {
        if (lane == 0) tc_report(p.status, 2140, 0, it.nst);
        ok = false;
      }
    }
    for (int i = 0; i < TA_SLOTS / 2 && ok; ++i) {   // as for the activations
      mbar_wait2(ta_empty + 8 * a.slot, a.ph, ta_empty + 8 * (a.slot + 1), a.ph, &since);
      a.next();
    }
  } else {
    // ------------------------------------------------------------ drain + epilogue
    regs_inc<Cfg::REGS_DRAIN>();
    const int qd = warp & 3;
    const int g = (warp - Cfg::DRAIN_WARP0) >> 2;   // which half of the tokens
    const uint32_t row = qd * 32 + lane;
    const uint32_t col0 = tmem_base + ((uint32_t)(qd * 32) << 16) + Cfg::ACC_COL0 + g * T;
    const uint32_t bars = JOINT ? 0u : 8u * Cfg::ENTRIES * g;
    const uint32_t s_row = scl + row * 16;
    constexpr int CH = T == 96 ? 48 : 32;           // columns of a load
    int rc = 0;                                     // scale slot of the stage
    uint32_t ph = 0;                                // of both entries
    pdl_wait();  // before any write to global memory (nothing to drain before the activations are in anyway)
    for (int u = blockIdx.x; u < units; u += gridDim.x) {
      const TcUnit it = tc_unit(p, u);
      since = wait_start();
      float2 acc[T / 2];
#pragma unroll
      for (int x = 0; x < T / 2; ++x) acc[x] = make_float2(0.f, 0.f);
      for (int i = 0; i < it.nst && since != WAIT_OVER; ++i) {
        float s[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {               // the stage's blocks
          const uint32_t bar = bars + 8 * (k & 1);
          mbar_wait_ready(acc_full + bar, ph, &since);
          tc_fence_after();
#pragma unroll
          for (int c = 0; c < T / CH; ++c) {
            uint32_t b[CH];
            tc_ld_cols<CH>(col0 + (k & 1) * 2 * T + c * CH, b);
            if (k == 0 && c == 0) {
              const uint4 sc = lds_v4(s_row + rc * SC_BYTES);
              s[0] = __uint_as_float(sc.x); s[1] = __uint_as_float(sc.y); s[2] = __uint_as_float(sc.z); s[3] = __uint_as_float(sc.w);
            }
            tc_loaded(b);
            if (c == T / CH - 1) {
              tc_fence_before();
              __syncwarp();
              mbar_arrive_if(acc_empty + bar, lane == 0);
            }
            add_cols<CH>(acc + c * (CH / 2), s[k], b);
          }
          if (k & 1) ph ^= 1u;
        }
        if (++rc == SC_SLOTS) rc = 0;
      }
      if (since == WAIT_OVER) {
        if (lane == 0) tc_report(p.status, 2150, 0, it.nst);
        break;
      }
      store_tile<T>(p, acc, it.split, (int64_t)it.tile * TC_ROWS + row, (int64_t)(it.mtile * 2 + g) * T, lane);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 3) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// ---------------------------------------------------------------- host side
// What a tensor map is a function of: address, extents, pitches and box.  Maps are encoded once and kept.
struct MapKey {
  const void* base;
  uint64_t d0, d1, d2, d3, p1, p2, p3;
  uint32_t b0, b1, b2, b3, elem, swizzle;
  bool operator==(const MapKey& o) const {
    return base == o.base && d0 == o.d0 && d1 == o.d1 && d2 == o.d2 && d3 == o.d3 && p1 == o.p1 && p2 == o.p2 && p3 == o.p3 &&
           b0 == o.b0 && b1 == o.b1 && b2 == o.b2 && b3 == o.b3 && elem == o.elem && swizzle == o.swizzle;
  }
};
struct MapKeyHash {
  size_t operator()(const MapKey& k) const {
    uint64_t h = reinterpret_cast<uint64_t>(k.base);
    for (uint64_t v : {k.d0, k.d1, k.d2, k.d3, k.p1, k.p2, k.p3, ((uint64_t)k.b0 << 32) | k.b1, ((uint64_t)k.b2 << 32) | k.b3,
                       ((uint64_t)k.elem << 32) | k.swizzle})
      h = h * 0x9E3779B97F4A7C15ull + v;
    return (size_t)(h ^ (h >> 29));
  }
};

logos_status_t map_cached(CUtensorMap* out, const MapKey& key, CUtensorMapDataType dt) {   // d2 == 0: two dimensions
  static std::mutex mu;
  static std::unordered_map<MapKey, CUtensorMap, MapKeyHash> cache;
  {
    std::lock_guard<std::mutex> lk(mu);
    auto it = cache.find(key);
    if (it != cache.end()) {
      *out = it->second;
      return LOGOS_OK;
    }
  }
  if (key.d2 == 0) {
    LOGOS_TRY(make_tensor_map_2d(out, key.base, dt, key.elem, key.d0, key.d1, key.p1, key.b0, key.b1, (CUtensorMapSwizzle)key.swizzle));
  } else {
    const uint64_t dims[4] = {key.d0, key.d1, key.d2, key.d3}, pitch[3] = {key.p1, key.p2, key.p3};
    const uint32_t box[4] = {key.b0, key.b1, key.b2, key.b3};
    LOGOS_TRY(make_tensor_map_4d(out, key.base, dt, key.elem, dims, pitch, box, (CUtensorMapSwizzle)key.swizzle));
  }
  std::lock_guard<std::mutex> lk(mu);
  if (cache.size() > 8192) cache.clear();
  cache[key] = *out;
  return LOGOS_OK;
}

}  // namespace

logos_status_t cached_map(CUtensorMap* out, const void* base, CUtensorMapDataType dt, uint32_t elem, uint64_t d0,
                          uint64_t d1, uint64_t pitch1, uint32_t box0, uint32_t box1, CUtensorMapSwizzle swizzle) {
  return map_cached(out, MapKey{base, d0, d1, 0, 0, pitch1, 0, 0, box0, box1, 0, 0, elem, (uint32_t)swizzle}, dt);
}

namespace {

logos_status_t cached_map_4d(CUtensorMap* out, const void* base, CUtensorMapDataType dt, uint64_t d0, uint64_t d1, uint64_t d2,
                             uint64_t d3, uint64_t p1, uint64_t p2, uint64_t p3, uint32_t b1, uint32_t b2, uint32_t b3) {
  return map_cached(out, MapKey{base, d0, d1, d2, d3, p1, p2, p3, (uint32_t)d0, b1, b2, b3, 2, (uint32_t)CU_TENSOR_MAP_SWIZZLE_128B}, dt);
}

}  // namespace

namespace {

// How a product is cut up: tokens per tile, K splits, and the row tiles that run in pairs and alone.
struct TcPlan {
  int t, splits, pairs, solos;
  bool wide;   // the wide form: 2 t tokens a tile, row tiles alone
};

// Cycles of one K stage of a pair and of a single tile, by tokens per tile, of the pipeline fill plus the last
// epilogue, and of a unit's epilogue.  They decide only who computes what: the order of a sum depends on the K splits
// alone.  The table was made with an earlier form of this kernel; timed again (calls in a row, by the slope between
// K = 4096 and 12288, at 1965 MHz, one plane / two): singles 879/861, 879/1051, 1150/1574, 1620/2119, pairs
// 1967/1917, 1804/2092, 2338/3018, 2914/3676.  From 64 tokens on it stands between what one plane and two cost; whether a table
// for each makes better choices has not been tried.
struct TcCost {
  int t, pair, solo, unit;
};
constexpr TcCost kCosts[] = {{16, 1760, 1065, 700}, {32, 1900, 1090, 700}, {64, 2550, 1400, 700}, {96, 3300, 1900, 700}};
// Units of the wide form on the same scale, fitted to 74 shapes timed with each form (m 70 to 4096, n 896 to 55296, K 512 to 8192,
// one plane and two): what the costs choose is 0.1 % slower than the best of the three in the mean, 4 % at worst.  Bf16 / f32, us,
// the other form -> 128 tokens a unit, 192: 128 x 18944 x 3584 38.0 -> 30.8, 36.1 / 49.4 -> 39.8, 47.3; 192 50.0 -> 55.8, 38.3 / 64.4
// -> 73.7, 52.0; 1024 248 -> 210, 207 / 324 -> 287, 275; few row tiles, 1024 x 896 x 4864: 28.6 -> 36.5, 44.6 / 32.8 -> 41.5, 47.8.
// Up to 64 tokens half of a wide unit would be empty.
constexpr TcCost kWideCosts[] = {{64, 0, 1880, 1200}, {96, 0, 2380, 2100}};
constexpr int kFillCycles = 8000;

// The slowest CTA's time when `pairs` pair items and `solos` single tiles run round robin on g CTAs.
int64_t plan_cycles(const TcCost& c, int64_t pairs, int64_t solos, int64_t sp, int64_t mt, int64_t stages, int64_t g) {
  const int64_t pu = pairs * sp * mt, total = (pairs + solos) * sp * mt;
  const int64_t per = (stages + sp - 1) / sp;
  const int64_t tp = per * c.pair + c.unit, ts = per * c.solo + c.unit;
  int64_t worst = 0;
  for (int64_t cta : {(int64_t)0, pu % g, pu % g - 1, total % g - 1}) {
    if (cta < 0 || cta >= g) continue;
    const int64_t np = pu > cta ? (pu - cta + g - 1) / g : 0, nt = total > cta ? (total - cta + g - 1) / g : 0;
    worst = std::max(worst, np * tp + (nt - np) * ts);
  }
  return worst + kFillCycles;
}

TcPlan make_plan(int64_t m, int64_t n, int64_t k, int64_t sp, int sms, int64_t* cycles = nullptr) {
  const int64_t tl = (n + TC_ROWS - 1) / TC_ROWS, stages = (k + TC_KSTAGE - 1) / TC_KSTAGE;
  TcPlan best{16, (int)sp, 0, (int)tl, false};
  int64_t best_cost = INT64_MAX;
  for (const TcCost& c : kCosts) {
    // fewer tokens than half a larger tile never pay for it
    if (c.t < 64 && m > c.t) continue;
    if (c.t > 16 && m <= c.t / 2 && c.t <= 64) continue;
    if (c.t == 96 && m <= 64) continue;
    const int64_t mt = (m + c.t - 1) / c.t;
    const int64_t full_rounds = tl * sp * mt / (2 * sms);
    const int64_t cand[3] = {0, tl / 2, std::min<int64_t>(tl / 2, full_rounds * sms / (sp * mt))};
    for (int64_t pairs : cand) {
      const int64_t cost = plan_cycles(c, pairs, tl - 2 * pairs, sp, mt, stages, sms);
      if (cost < best_cost) {
        best_cost = cost;
        best = TcPlan{c.t, (int)sp, (int)pairs, (int)(tl - 2 * pairs), false};
      }
    }
  }
  if (m > 64) {
    for (const TcCost& c : kWideCosts) {
      const int64_t cost = plan_cycles(c, 0, tl, sp, (m + 2 * c.t - 1) / (2 * c.t), stages, sms);
      if (cost < best_cost) {
        best_cost = cost;
        best = TcPlan{c.t, (int)sp, 0, (int)tl, true};
      }
    }
  }
  if (cycles) *cycles = best_cost;
  return best;
}

// See gemm_many_splits.  The fold of the splits on the costs' scale: its launch (unless the consumer folds), and writing and
// reading the partial sums.  Where the consumer folds, prompts of 40 to 1536 rows of three model shapes (hidden 896, 3584, 5120) take 0.91 to
// 1.04 of their time with the best count from 1 to 12 for o_proj and down_proj alike.
int make_splits(int64_t m, int64_t n, int64_t k, int sms, bool folded) {
  const int64_t stages = k / TC_KSTAGE, most = std::min<int64_t>(stages / 4, 16);
  int best = 1;
  int64_t best_cost = INT64_MAX;
  for (int64_t sp = 1; sp <= std::max<int64_t>(most, 1); ++sp) {
    if (sp > 1 && sp * m * n > (16ll << 20)) break;
    int64_t cost;
    make_plan(m, n, k, sp, sms, &cost);
    if (sp > 1) cost += folded ? 1500 + sp * m * n / 600 : 6000 + sp * m * n / 333;
    if (cost < best_cost) {
      best_cost = cost;
      best = (int)sp;
    }
  }
  return best;
}

// Plans are pure functions of the shape: the last ones of a thread are kept.
TcPlan plan_for(int64_t m, int64_t n, int64_t k, int64_t splits, int device) {
  struct Entry {
    int64_t m = -1, n = 0, k = 0, sp = 0;
    int device = 0;
    TcPlan plan{};
  };
  thread_local Entry cache[64];
  const uint64_t h = ((uint64_t)m * 0x9E3779B97F4A7C15ull) ^ ((uint64_t)n * 0xBF58476D1CE4E5B9ull) ^ ((uint64_t)k * 0x94D049BB133111EBull) ^
                     (uint64_t)splits;
  Entry& e = cache[(h ^ (h >> 29)) >> 7 & 63];
  if (e.m != m || e.n != n || e.k != k || e.sp != splits || e.device != device) {
    e.m = m; e.n = n; e.k = k; e.sp = splits; e.device = device;
    e.plan = make_plan(m, n, k, splits, sm_count(device));
  }
  return e.plan;
}

template <int T, int LIMBS, bool WIDE = false>
logos_status_t launch_t(const GemmArgs& g, const TcPlan& plan, cudaStream_t st) {
  using Cfg = std::conditional_t<WIDE, WideCfg<T, LIMBS>, TcCfg<T, LIMBS>>;
  constexpr int TOKENS = WIDE ? 2 * T : T;   // of a token tile
  CUtensorMap mq, ma, ms;
  const int64_t stages = (g.k + TC_KSTAGE - 1) / TC_KSTAGE, tiles = (g.n + TC_ROWS - 1) / TC_ROWS;
  if (g.q_tiled) {
    const uint64_t rows = (uint64_t)tiles * (uint64_t)stages * TC_ROWS;
    LOGOS_TRY(cached_map(&mq, g.q, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, TC_KSTAGE, rows, TC_KSTAGE, TC_KSTAGE, TC_ROWS));
  } else {
    LOGOS_TRY(cached_map(&mq, g.q, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, (uint64_t)g.k, (uint64_t)g.n, (uint64_t)g.k, TC_KSTAGE, TC_ROWS));
  }
  // [planes][halves of a stage][tokens][64]: the planes lie at any multiple of 16 bytes from each other
  LOGOS_TRY(cached_map_4d(&ma, g.a, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 64, (uint64_t)g.m, (uint64_t)(2 * stages), LIMBS,
                          (uint64_t)g.lda * 2, 128, LIMBS == 2 ? (uint64_t)(reinterpret_cast<const char*>(g.a_lo) - static_cast<const char*>(g.a)) : 128,
                          TOKENS, WIDE ? 1 : 2, LIMBS));
  ms = ma;
  const bool s_tiled = g.q_tiled || g.s_tiled;
  if (!s_tiled)
    LOGOS_TRY(cached_map(&ms, g.s, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, (uint64_t)(g.k / 32), (uint64_t)g.n, (uint64_t)(g.k / 32) * 4, 4,
                         TC_ROWS, CU_TENSOR_MAP_SWIZZLE_NONE));
  TcParams p{};
  p.s = g.s; p.n = g.n; p.m = g.m;
  p.c = g.c; p.c_dtype = g.c_dtype; p.c_act = g.c_act; p.ldc = g.ldc; p.aux = g.aux; p.epilogue = g.epilogue;
  p.partials = g.partials;
  p.splits = plan.splits;
  p.stages_total = (int)stages;
  p.s_tiled = s_tiled;
  p.wait_scales = g.s_tiled;
  if (g.epilogue == EPI_RESIDUAL && g.c_dtype != LOGOS_BF16) return fail(LOGOS_ERROR, "q8_gemm: a residual goes with bf16 results");
  const int64_t mtiles = (g.m + TOKENS - 1) / TOKENS;
  const int64_t units = (int64_t)(plan.pairs + plan.solos) * plan.splits * mtiles;
  if (units > INT32_MAX / 4 || tiles * stages > INT32_MAX / TC_ROWS) return fail(LOGOS_OUT_OF_BOUNDS, "q8_gemm: too many work units");
  p.pairs = plan.pairs;
  p.solos = plan.solos;
  p.mtiles = (int)mtiles;
  // about 12 token tiles x 12 pairs of row tiles run side by side, of the wide form 8 x 18 row tiles
  const int64_t most = WIDE ? 8 : 12, groups = (mtiles + most - 1) / most;
  p.group = (int)((mtiles + groups - 1) / groups);
  p.stream_once = mtiles == 1;
  p.status = kernel_status_ptr(g.device);
  if (!p.status) return fail(LOGOS_ERROR, "q8_gemm: no kernel status word");
  if (p.splits > p.stages_total) return fail(LOGOS_ERROR, "q8_gemm: more K splits than 128-column stages");

  void (*kernel)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const TcParams);
  if constexpr (WIDE) kernel = g.q_tiled ? q8_gemm_wide_kernel<T, LIMBS, true> : q8_gemm_wide_kernel<T, LIMBS, false>;
  else kernel = g.q_tiled ? q8_gemm_tc_kernel<T, LIMBS, true> : q8_gemm_tc_kernel<T, LIMBS, false>;
  LOGOS_TRY(allow_smem(reinterpret_cast<const void*>(kernel), g.device, (int)Cfg::SMEM));
  // persistent CTAs: one per SM at most, each takes units blockIdx.x, blockIdx.x + gridDim.x, ...
  const int sms = sm_count(g.device);
  dim3 grid((unsigned)(units < sms ? units : sms), 1u, 1u);
  LOGOS_CUDA_TRY(launch_kernel(kernel, grid, dim3(Cfg::THREADS), Cfg::SMEM, st, mq, ma, ms, p));
  count_launch(LK_GEMM_TC);
  return check_launch("q8_gemm_tc_kernel");
}

template <int LIMBS>
logos_status_t launch_plan(const GemmArgs& g, const TcPlan& plan, cudaStream_t st) {
  if (plan.wide) return plan.t == 64 ? launch_t<64, LIMBS, true>(g, plan, st) : launch_t<96, LIMBS, true>(g, plan, st);
  switch (plan.t) {
    case 16: return launch_t<16, LIMBS>(g, plan, st);
    case 32: return launch_t<32, LIMBS>(g, plan, st);
    case 64: return launch_t<64, LIMBS>(g, plan, st);
    default: return launch_t<96, LIMBS>(g, plan, st);
  }
}

}  // namespace

bool gemm_tc_applicable(const GemmArgs& g) {
  if (g.a_dtype != LOGOS_F16) return false;
  if (g.k < TC_KSTAGE || g.k % 32) return false;
  // K of whole stages, or scales in the tile-major form: the row-major box needs rows of 16-byte multiples
  if (g.k % TC_KSTAGE && !g.q_tiled && !g.s_tiled) return false;
  if (g.m < 1 || g.n < 1) return false;
  if (g.lda % 8 || g.lda < (g.k + TC_KSTAGE - 1) / TC_KSTAGE * TC_KSTAGE) return false;   // whole stages, zero past K
  if (g.a_lo && reinterpret_cast<uintptr_t>(g.a_lo) <= reinterpret_cast<uintptr_t>(g.a)) return false;
  if ((reinterpret_cast<uintptr_t>(g.a) & 15u) || (reinterpret_cast<uintptr_t>(g.a_lo) & 15u) ||
      (reinterpret_cast<uintptr_t>(g.q) & 15u) || (reinterpret_cast<uintptr_t>(g.s) & 15u))
    return false;
  return true;
}

int gemm_many_splits(int64_t m, int64_t n, int64_t k, int device, bool folded) {
  if ((n + TC_ROWS - 1) / TC_ROWS >= sm_count(device)) return 1;
  struct Entry {
    int64_t m = -1, n = 0, k = 0;
    int device = 0, splits = 1;
    bool folded = false;
  };
  thread_local Entry cache[64];   // a pure function of the shape, as the plans are
  const uint64_t h = ((uint64_t)m * 0x9E3779B97F4A7C15ull) ^ ((uint64_t)n * 0xBF58476D1CE4E5B9ull) ^ ((uint64_t)k * 0x94D049BB133111EBull);
  Entry& e = cache[(h ^ (h >> 29)) >> 7 & 63];
  if (e.m != m || e.n != n || e.k != k || e.device != device || e.folded != folded)
    e = Entry{m, n, k, device, make_splits(m, n, k, sm_count(device), folded), folded};
  return e.splits;
}

int gemm_wide_tokens(int64_t m, int64_t n, int64_t k, int device) {
  const TcPlan plan = plan_for(m, n, k, 1, device);
  return plan.wide ? 2 * plan.t : 0;
}

logos_status_t launch_q8_gemm_tc(const GemmArgs& g, cudaStream_t st) {
  const TcPlan plan = plan_for(g.m, g.n, g.k, g.splits > 1 ? g.splits : 1, g.device);
  return g.a_lo ? launch_plan<2>(g, plan, st) : launch_plan<1>(g, plan, st);
}

}  // namespace logos
