// Thin inline-PTX layer for sm_100a: mbarriers with bounded waits, TMA tile
// loads, ldmatrix / mma.sync, tcgen05 (TMEM alloc, MMA, commit, ld/st).
// Every wait is bounded: after the limit the caller gets `false`, records a
// status code and leaves; nothing here spins for ever.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"

namespace logos {
namespace ptx {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(pred));
  return pred != 0;
}

// ------------------------------------------------------------ mbarrier
// The forms on a 32-bit address take the shared-window address: code that walks rings keeps such
// addresses, since deriving them from generic pointers at every wait costs more than the wait.
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) { mbar_init(smem_u32(bar), count); }
__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// this thread's writes to shared memory come before what the async proxy (TMA) does there after a later barrier
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_if(uint32_t bar, bool on) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\t@p mbarrier.arrive.shared::cta.b64 _, [%0];\n\t}" ::"r"(bar),
               "r"((uint32_t)on)
               : "memory");
}
// arrives `COUNT` times at once
template <int COUNT>
__device__ __forceinline__ void mbar_arrive_n_if(uint32_t bar, bool on) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\t@p mbarrier.arrive.shared::cta.b64 _, [%0], %2;\n\t}" ::"r"(bar),
               "r"((uint32_t)on), "n"(COUNT)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  mbar_arrive_expect_tx(smem_u32(bar), bytes);
}
// Bounded waits: one to two periods of the upper half of the SM clock, two to four and a half seconds at 1.9 GHz.  The
// limit is of time, since a poll that finds its phase open takes anything from 65 cycles to the 7800 for which
// the hardware suspends the thread (measured on a B200): a number of polls that outlasts the short ones bounds the
// long ones by minutes.  The clock is read once in 32 failed polls: an arrival that does not end the phase wakes the
// thread too, and reading it after every poll cost the GEMM 1 to 1.5 %.
//
// The forms with `since` share one limit, counted from wait_start(): once it has passed, *since is WAIT_OVER, and this
// and every later wait of the thread return after a poll, so that a loop can look at it once a round instead of
// after every wait.  What is done in between works on stale data; the caller drops it and reports.  A warp that
// waits takes issue slots from the warps it waits for: the loop is as few instructions as it can be.
constexpr uint32_t WAIT_OVER = 31;
// The clock's upper half in units of 32; the low five bits count failed polls.  At least two units, so that no valid
// value is WAIT_OVER or what a failed poll makes of it.
__device__ __forceinline__ uint32_t wait_start() {
  uint32_t t;
  asm volatile("mov.u32 %0, %%clock_hi;" : "=r"(t));
  return (t < 2 ? 2u : t) << 5;
}
#define LOGOS_MBAR_TRY(P, BAR, PH) "mbarrier.try_wait.parity.shared::cta.b64 " P ", [" BAR "], " PH ";\n\t"
#define LOGOS_MBAR_REGS "{\n\t.reg .pred p, q, r, s;\n\t.reg .u32 t;\n"
#define LOGOS_MBAR_AGAIN                                                                                     \
  "@p bra DONE;\n\t"                                                                                         \
  "add.u32 %0, %0, 1;\n\t"                                                                                   \
  "and.b32 t, %0, 31;\n\t"                                                                                   \
  "setp.ne.u32 s, t, 0;\n\t"                                                                                 \
  "@s bra POLL;\n\t"                                                                                         \
  "setp.eq.u32 s, %0, 32;\n\t"                                                                               \
  "@s bra OVER;\n\t"                                                                                         \
  "add.u32 %0, %0, -32;\n\t"                                                                                 \
  "mov.u32 t, %%clock_hi;\n\t"                                                                               \
  "shl.b32 t, t, 5;\n\t"                                                                                     \
  "sub.s32 t, t, %0;\n\t"                                                                                    \
  "setp.lt.s32 s, t, 64;\n\t"                                                                                \
  "@s bra POLL;\n"                                                                                           \
  "OVER:\n\tmov.u32 %0, 31;\n"                                                                              \
  "DONE:\n\t}"
__device__ __forceinline__ void mbar_wait(uint32_t bar, uint32_t parity, uint32_t* since) {
  asm volatile(LOGOS_MBAR_REGS "POLL:\n\t" LOGOS_MBAR_TRY("p", "%1", "%2") LOGOS_MBAR_AGAIN
               : "+r"(*since)
               : "r"(bar), "r"(parity)
               : "memory");
}
// Two or three barriers polled together: their latencies overlap.
__device__ __forceinline__ void mbar_wait2(uint32_t bar0, uint32_t ph0, uint32_t bar1, uint32_t ph1, uint32_t* since) {
  asm volatile(LOGOS_MBAR_REGS "POLL:\n\t" LOGOS_MBAR_TRY("p", "%1", "%2") LOGOS_MBAR_TRY("q", "%3", "%4")
               "and.pred p, p, q;\n\t" LOGOS_MBAR_AGAIN
               : "+r"(*since)
               : "r"(bar0), "r"(ph0), "r"(bar1), "r"(ph1)
               : "memory");
}
__device__ __forceinline__ void mbar_wait3(uint32_t bar0, uint32_t ph0, uint32_t bar1, uint32_t ph1, uint32_t bar2, uint32_t ph2,
                                           uint32_t* since) {
  asm volatile(LOGOS_MBAR_REGS "POLL:\n\t" LOGOS_MBAR_TRY("p", "%1", "%2") LOGOS_MBAR_TRY("q", "%3", "%4")
               LOGOS_MBAR_TRY("r", "%5", "%6") "and.pred p, p, q;\n\tand.pred p, p, r;\n\t" LOGOS_MBAR_AGAIN
               : "+r"(*since)
               : "r"(bar0), "r"(ph0), "r"(bar1), "r"(ph1), "r"(bar2), "r"(ph2)
               : "memory");
}
// The same for a converged warp and a barrier that is mostly ready when it is asked: one poll and a vote first, without a
// loop.  A taken branch costs the loop above 30 of its 110 cycles on a ready barrier; where waits are long
// (q8_gemm_tc_kernel at 64 tokens) the extra poll costs more than it saves, 1 to 3 %.
__device__ __forceinline__ uint32_t mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\t" LOGOS_MBAR_TRY("p", "%1", "%2") "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok;
}
__device__ __forceinline__ void mbar_wait_ready(uint32_t bar, uint32_t parity, uint32_t* since) {
  if (__builtin_expect(!__all_sync(0xffffffffu, mbar_try(bar, parity)), 0)) mbar_wait(bar, parity, since);
}
__device__ __forceinline__ void mbar_wait3_ready(uint32_t bar0, uint32_t ph0, uint32_t bar1, uint32_t ph1, uint32_t bar2, uint32_t ph2,
                                                 uint32_t* since) {
  const uint32_t ready = mbar_try(bar0, ph0) & mbar_try(bar1, ph1) & mbar_try(bar2, ph2);
  if (__builtin_expect(!__all_sync(0xffffffffu, ready), 0)) mbar_wait3(bar0, ph0, bar1, ph1, bar2, ph2, since);
}
// A single wait with a limit of its own, counted from its 32nd failed poll; false when it gave up.
#define LOGOS_MBAR_SINGLE(TRY)                \
  "{\n\t.reg .pred p, s;\n\t.reg .u32 n, t, e;\n\tmov.u32 n, 0;\n" \
  "POLL:\n\t" TRY                             \
  "@p bra DONE;\n\t"                          \
  "add.u32 n, n, 1;\n\t"                      \
  "and.b32 t, n, 31;\n\t"                     \
  "setp.ne.u32 s, t, 0;\n\t"                  \
  "@s bra POLL;\n\t"                          \
  "mov.u32 t, %%clock_hi;\n\t"                \
  "setp.eq.u32 s, n, 32;\n\t"                 \
  "@s mov.u32 e, t;\n\t"                      \
  "sub.u32 t, t, e;\n\t"                      \
  "setp.lt.u32 s, t, 2;\n\t"                  \
  "@s bra POLL;\n"                            \
  "DONE:\n\tselp.u32 %0, 1, 0, p;\n\t}"
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(LOGOS_MBAR_SINGLE(LOGOS_MBAR_TRY("p", "%1", "%2")) : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return ok != 0;
}

// ------------------------------------------------------------ clusters
// A wait for what other CTAs of the cluster pushed into this one's shared memory: a push releases at cluster scope, and
// only an acquire of that scope sees what it wrote (the plain form's is the CTA).
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(LOGOS_MBAR_SINGLE("mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t")
               : "=r"(ok)
               : "r"(smem_u32(bar)), "r"(parity)
               : "memory");
  return ok != 0;
}
// Returns once every thread of the cluster that has not ended is here.  Threads of a warp may come one by one.
__device__ __forceinline__ void cluster_meet() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// the address of this CTA's `addr` in the CTA of a rank
__device__ __forceinline__ uint32_t smem_of_rank(uint32_t addr, int rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
  return a;
}
// 16 or 8 bytes into another CTA's shared memory, counted on a barrier there
__device__ __forceinline__ void push16(uint32_t addr, float4 v, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
               ::"r"(addr), "r"(__float_as_uint(v.x)), "r"(__float_as_uint(v.y)), "r"(__float_as_uint(v.z)), "r"(__float_as_uint(v.w)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void push8(uint32_t addr, float2 v, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];"
               ::"r"(addr), "r"(__float_as_uint(v.x)), "r"(__float_as_uint(v.y)), "r"(bar)
               : "memory");
}

__device__ __forceinline__ uint4 lds_v4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}

// ------------------------------------------------------------ TMA (tile mode, no multicast)
__device__ __forceinline__ void prefetch_tensormap(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}
// x = innermost coordinate (elements); x * element size must be a multiple of 16 bytes.
__device__ __forceinline__ void tma_load_2d(uint32_t smem_dst, const CUtensorMap* m, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_dst), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* m, uint64_t* bar, int x, int y) {
  tma_load_2d(smem_u32(smem_dst), m, smem_u32(bar), x, y);
}
__device__ __forceinline__ void tma_load_2d_hint(uint32_t smem_dst, const CUtensorMap* m, uint32_t bar, int x, int y,
                                                 uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint "
      "[%0], [%1, {%3, %4}], [%2], %5;"
      ::"r"(smem_dst), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(x), "r"(y), "l"(policy)
      : "memory");
}
__device__ __forceinline__ void tma_load_4d_hint(uint32_t smem_dst, const CUtensorMap* m, uint32_t bar, int x, int y, int z, int w,
                                                 uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cta.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint "
      "[%0], [%1, {%3, %4, %5, %6}], [%2], %7;"
      ::"r"(smem_dst), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(x), "r"(y), "r"(z), "r"(w), "l"(policy)
      : "memory");
}
__device__ __forceinline__ uint64_t policy_evict_first() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t policy_evict_normal() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t policy_evict_last() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}

// Byte offset of 16-byte chunk `chunk` of row `row` inside a tile whose rows
// are 128 bytes and which TMA wrote with the 128-byte swizzle (tile base
// 1024-byte aligned): the chunk index is XORed with the row index mod 8.
__device__ __forceinline__ uint32_t swz128(uint32_t row, uint32_t chunk) {
  return row * 128u + ((chunk ^ (row & 7u)) << 4);
}

// ------------------------------------------------------------ legacy tensor path (attention)
__device__ __forceinline__ void ldmatrix_x4(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3,
                                                  uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}
// D(16x8,f32) += A(16x16,f16) * B(16x8,f16)
__device__ __forceinline__ void mma_f16_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// ------------------------------------------------------------ tcgen05 / TMEM
// Allocation is per CTA, by one full warp; the base address lands in shared memory.
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_result, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)),
               "r"(cols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// All MMAs this thread issued so far arrive on `bar` when they complete.
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem desc]; kind::f16 (f16/bf16 inputs, f32 accumulate)
template <bool ACCUMULATE>
__device__ __forceinline__ void tc_mma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "n"(ACCUMULATE ? 1 : 0)
      : "memory");
}
// D[tmem] = A[tmem] * B[smem desc] + D * 2^-SHIFT   (scale-input-d form, f16/tf32 kinds only)
template <int SHIFT>
__device__ __forceinline__ void tc_mma_f16_ts_scaled_d(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc,
                                                       uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, 1, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%4, %4, %4, %4}, p, %5;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(0), "n"(SHIFT)
      : "memory");
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// 32 lanes x 32-bit, N consecutive columns: thread t of the warp gets lane
// (taddr.lane + t), register j = column (taddr.col + j).
__device__ __forceinline__ void tc_ld_32x32b_x32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tc_ld_32x32b_x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tc_ld_32x32b_x8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tc_ld_32x32b_x4(uint32_t taddr, uint32_t (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tc_st_32x32b_x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
        "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]),
        "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
// Shared-memory matrix descriptor for a K-major operand tile stored with the
// 128-byte swizzle (rows of 128 bytes, 8-row groups of 1024 bytes):
//   bits [0,14)  start address >> 4          bits [16,30) leading byte offset >> 4 (unused here: 1)
//   bits [32,46) stride byte offset >> 4 (1024 B between 8-row groups)
//   bits [46,48) descriptor version = 1      bits [61,64) layout type 2 = SWIZZLE_128B
__device__ __forceinline__ uint64_t make_desc_sw128(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

// kind::f16 instruction descriptor: f32 accumulate, A/B formats (0 = f16, 1 =
// bf16), both K-major, N>>3 at bit 17, M>>4 at bit 24.
__host__ __device__ constexpr uint32_t make_idesc_f16(int a_fmt, int b_fmt, int m, int n) {
  return (1u << 4) | ((uint32_t)a_fmt << 7) | ((uint32_t)b_fmt << 10) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(m >> 4) << 24);
}

}  // namespace ptx

// Host side: tensor-map encoding through the driver entry point (no libcuda link).
logos_status_t make_tensor_map_2d(CUtensorMap* out, const void* base, CUtensorMapDataType dtype, uint32_t elem_bytes,
                                  uint64_t inner, uint64_t outer, uint64_t row_pitch_bytes, uint32_t box_inner,
                                  uint32_t box_outer, CUtensorMapSwizzle swizzle);
// Four dimensions: d[0] innermost (contiguous), pitches of d[1] to d[3] in bytes.
logos_status_t make_tensor_map_4d(CUtensorMap* out, const void* base, CUtensorMapDataType dtype, uint32_t elem_bytes,
                                  const uint64_t (&d)[4], const uint64_t (&pitch_bytes)[3], const uint32_t (&box)[4],
                                  CUtensorMapSwizzle swizzle);

}  // namespace logos
