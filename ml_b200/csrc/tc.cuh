// Blackwell (sm_100a) primitives as inline PTX: mbarrier, TMA tiled loads (each CTA fetches its own tiles),
// tcgen05 MMA / TMEM alloc / TMEM load, and the shared-memory + instruction descriptors they take.
#pragma once
#include "common.cuh"
#include <cuda.h>  // CUtensorMap (types only; the encoder is fetched through the runtime's driver entry point)

namespace tc {

// ------------------------------------------------------------------ addresses
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// ------------------------------------------------------------------ mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Bounded wait: gives up after ~4 s of wall time, records MLB_ERR_MBAR_TIMEOUT and returns false so the
// caller can unwind (free TMEM, return) instead of hanging the GPU.
#ifndef MLB_MBAR_TIMEOUT_NS
#define MLB_MBAR_TIMEOUT_NS 4000000000ull
#endif
// (As few instructions as it can be, here and below: a kernel has dozens of waits, and what they hold besides the first probe pushes its
// loops out of the SM's instruction cache.  A probe sleeps in hardware for a while, so reading the clock after each costs nothing.)
// Lanes may leave in different rounds: a whole warp that waits is brought together (__syncwarp, or a vote where the answer decides) before
// it touches tensor memory, stores matrices or meets at a named barrier.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int where = 0) {
  if (mbar_try(bar, parity)) return true;
  const uint64_t t0 = globaltimer_ns();
#pragma unroll 1
  while (!mbar_try(bar, parity)) {
    if (globaltimer_ns() - t0 > MLB_MBAR_TIMEOUT_NS) {
      mlb_set_error(MLB_ERR_MBAR_TIMEOUT, where);
      return false;
    }
  }
  return true;
}
// The same for a CTA that gives up as one: a wait that runs out leaves its number (not 0) in *given_up (shared memory, 0 before), and from then on others
// return false instead of waiting.  Of waits that run out within a probe of each other the last one's number stays: a compare-and-swap that kept the first
// made bidirectional attention slower (32 x 197 tokens, 12 heads, forward + backward 96.6 -> 97.0 us).  The CTA reports the number at its end
// (report_given_up, one thread, behind a barrier of all).
template <unsigned long long LIMIT_NS = MLB_MBAR_TIMEOUT_NS>
__device__ __forceinline__ bool mbar_wait_sticky(uint64_t* bar, uint32_t parity, int where, volatile int* given_up) {
  if (mbar_try(bar, parity)) return true;
  const uint64_t t0 = globaltimer_ns();
#pragma unroll 1
  do {
    if (*given_up) return false;
    if (mbar_try(bar, parity)) return true;
  } while (globaltimer_ns() - t0 <= LIMIT_NS);
  *given_up = where;
  return false;
}
__device__ __forceinline__ void report_given_up(volatile int* given_up) {
  if (*given_up) mlb_set_error(MLB_ERR_MBAR_TIMEOUT, *given_up);
}

// Same bound, but the polling thread sleeps between probes so that it does not compete for issue slots with warps that
// share its scheduler (for waits that are expected to last hundreds of cycles or more).
__device__ __forceinline__ bool mbar_wait_sleep(uint64_t* bar, uint32_t parity, int where = 0, unsigned ns = 40) {
  if (mbar_try(bar, parity)) return true;
  uint64_t t0 = globaltimer_ns();
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 1024; i++) {
      __nanosleep(ns);
      if (mbar_try(bar, parity)) return true;
    }
    if (globaltimer_ns() - t0 > MLB_MBAR_TIMEOUT_NS) {
      mlb_set_error(MLB_ERR_MBAR_TIMEOUT, where);
      return false;
    }
  }
}

// ------------------------------------------------------------------ fences
__device__ __forceinline__ void fence_async_smem() {  // generic-proxy smem writes -> visible to TMA / tcgen05
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// ------------------------------------------------------------------ TMA (2D tiled, CTA-local destination)
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}
// shared -> global tiled store / fp32 add-reduce (bulk async-group completion); out-of-range parts of the box are clipped.
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, const void* smem_src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(map), "r"(smem_u32(smem_src)),
               "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ void tma_reduce_add_2d(const CUtensorMap* map, const void* smem_src, int x, int y) {
  asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.bulk_group [%0, {%2, %3}], [%1];" ::"l"(map),
               "r"(smem_u32(smem_src)), "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ void tma_commit_group() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void tma_wait_group_read() {  // at most N groups still reading their shared-memory source
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
template <int N>
__device__ __forceinline__ void tma_wait_group() {
  asm volatile("cp.async.bulk.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}

// ------------------------------------------------------------------ TMEM
// One full warp allocates `ncols` (power of two, 32..512) columns; the base address lands in *smem_slot.
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_slot)), "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// Warp-collective: lane i of warp w (w = warp index mod 4) reads TMEM lane 32*w+i, 32 consecutive fp32 columns.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// Warp-collective store: lane i writes 16 consecutive 32-bit columns of TMEM lane 32*w+i.
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// A tcgen05.ld's registers hold their values once wait::ld has returned, and the wait names no registers: with the two in separate
// statements nothing keeps the compiler from moving arithmetic on the registers in front of the wait.  So load and wait are one
// statement, whose outputs are defined when it is over (early clobber where a later load's address is still to be read).
__device__ __forceinline__ void tmem_ld16_wait(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld32_wait(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
        "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld32x2_wait(uint32_t taddr_a, uint32_t (&a)[32], uint32_t taddr_b, uint32_t (&b)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%64];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%32, %33, %34, %35, %36, %37, %38, %39, %40, %41, %42, %43, %44, %45, %46, %47, "
      "%48, %49, %50, %51, %52, %53, %54, %55, %56, %57, %58, %59, %60, %61, %62, %63}, [%65];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=&r"(a[0]), "=&r"(a[1]), "=&r"(a[2]), "=&r"(a[3]), "=&r"(a[4]), "=&r"(a[5]), "=&r"(a[6]), "=&r"(a[7]), "=&r"(a[8]),
        "=&r"(a[9]),
        "=&r"(a[10]), "=&r"(a[11]), "=&r"(a[12]), "=&r"(a[13]), "=&r"(a[14]), "=&r"(a[15]), "=&r"(a[16]), "=&r"(a[17]), "=&r"(a[18]),
        "=&r"(a[19]), "=&r"(a[20]), "=&r"(a[21]), "=&r"(a[22]), "=&r"(a[23]), "=&r"(a[24]), "=&r"(a[25]), "=&r"(a[26]), "=&r"(a[27]),
        "=&r"(a[28]), "=&r"(a[29]), "=&r"(a[30]), "=&r"(a[31]), "=&r"(b[0]), "=&r"(b[1]), "=&r"(b[2]), "=&r"(b[3]), "=&r"(b[4]),
        "=&r"(b[5]), "=&r"(b[6]), "=&r"(b[7]), "=&r"(b[8]), "=&r"(b[9]), "=&r"(b[10]), "=&r"(b[11]), "=&r"(b[12]), "=&r"(b[13]),
        "=&r"(b[14]), "=&r"(b[15]), "=&r"(b[16]), "=&r"(b[17]), "=&r"(b[18]), "=&r"(b[19]), "=&r"(b[20]), "=&r"(b[21]), "=&r"(b[22]),
        "=&r"(b[23]), "=&r"(b[24]), "=&r"(b[25]), "=&r"(b[26]), "=&r"(b[27]), "=&r"(b[28]), "=&r"(b[29]), "=&r"(b[30]), "=&r"(b[31])
      : "r"(taddr_a), "r"(taddr_b)
      : "memory");
}
// Fragments: 32 columns of the warp's 32 rows, spread as a matrix instruction's accumulator is.  r[h][4 j + 2 v + x] is row 16 h + 8 v + lane / 4,
// column 8 j + 2 (lane % 4) + x: a thread has two adjacent columns of each eight, for four rows, so that what belongs to a column is
// read from shared memory once for four rows and by a quarter of the lanes.
__device__ __forceinline__ void tmem_ld_frag_wait(uint32_t taddr, uint32_t (&r)[2][16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%32];\n\t"
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
      "{%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%33];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=&r"(r[0][0]), "=&r"(r[0][1]), "=&r"(r[0][2]), "=&r"(r[0][3]), "=&r"(r[0][4]), "=&r"(r[0][5]), "=&r"(r[0][6]), "=&r"(r[0][7]),
        "=&r"(r[0][8]), "=&r"(r[0][9]), "=&r"(r[0][10]), "=&r"(r[0][11]), "=&r"(r[0][12]), "=&r"(r[0][13]), "=&r"(r[0][14]),
        "=&r"(r[0][15]), "=&r"(r[1][0]), "=&r"(r[1][1]), "=&r"(r[1][2]), "=&r"(r[1][3]), "=&r"(r[1][4]), "=&r"(r[1][5]), "=&r"(r[1][6]),
        "=&r"(r[1][7]), "=&r"(r[1][8]), "=&r"(r[1][9]), "=&r"(r[1][10]), "=&r"(r[1][11]), "=&r"(r[1][12]), "=&r"(r[1][13]),
        "=&r"(r[1][14]), "=&r"(r[1][15])
      : "r"(taddr), "r"(taddr + (16u << 16))
      : "memory");
}
// The same 32 columns packed in pairs (bf16 of columns 2 c, 2 c + 1 in 32-bit column c): w[h][2 j + v] is row 16 h + 8 v + lane / 4, column
// 4 j + lane % 4 of the sixteen.
__device__ __forceinline__ void tmem_st_frag(uint32_t taddr, const uint32_t (&w)[2][8]) {
  asm volatile("tcgen05.st.sync.aligned.16x128b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(w[0][0]), "r"(w[0][1]),
               "r"(w[0][2]), "r"(w[0][3]), "r"(w[0][4]), "r"(w[0][5]), "r"(w[0][6]), "r"(w[0][7])
               : "memory");
  asm volatile("tcgen05.st.sync.aligned.16x128b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr + (16u << 16)), "r"(w[1][0]),
               "r"(w[1][1]), "r"(w[1][2]), "r"(w[1][3]), "r"(w[1][4]), "r"(w[1][5]), "r"(w[1][6]), "r"(w[1][7])
               : "memory");
}
// 64 columns of 16 rows (the address's lane: the first), the first 32 in a, the others in b: fragments as above of one h.
__device__ __forceinline__ void tmem_ld_frag16x2_wait(uint32_t taddr, uint32_t (&a)[16], uint32_t (&b)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%32];\n\t"
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
      "{%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%33];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=&r"(a[0]), "=&r"(a[1]), "=&r"(a[2]), "=&r"(a[3]), "=&r"(a[4]), "=&r"(a[5]), "=&r"(a[6]), "=&r"(a[7]), "=&r"(a[8]), "=&r"(a[9]),
        "=&r"(a[10]), "=&r"(a[11]), "=&r"(a[12]), "=&r"(a[13]), "=&r"(a[14]), "=&r"(a[15]), "=&r"(b[0]), "=&r"(b[1]), "=&r"(b[2]),
        "=&r"(b[3]), "=&r"(b[4]), "=&r"(b[5]), "=&r"(b[6]), "=&r"(b[7]), "=&r"(b[8]), "=&r"(b[9]), "=&r"(b[10]), "=&r"(b[11]),
        "=&r"(b[12]), "=&r"(b[13]), "=&r"(b[14]), "=&r"(b[15])
      : "r"(taddr), "r"(taddr + 32)
      : "memory");
}
// Twice 16 columns of the warp's 32 rows: a[h][4 j + 2 v + x] is row 16 h + 8 v + lane / 4, column 8 j + 2 (lane % 4) + x.
__device__ __forceinline__ void tmem_ld_pairs_wait(uint32_t taddr_a, uint32_t (&a)[2][8], uint32_t taddr_b, uint32_t (&b)[2][8]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%32];\n\t"
      "tcgen05.ld.sync.aligned.16x256b.x2.b32 {%8, %9, %10, %11, %12, %13, %14, %15}, [%33];\n\t"
      "tcgen05.ld.sync.aligned.16x256b.x2.b32 {%16, %17, %18, %19, %20, %21, %22, %23}, [%34];\n\t"
      "tcgen05.ld.sync.aligned.16x256b.x2.b32 {%24, %25, %26, %27, %28, %29, %30, %31}, [%35];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=&r"(a[0][0]), "=&r"(a[0][1]), "=&r"(a[0][2]), "=&r"(a[0][3]), "=&r"(a[0][4]), "=&r"(a[0][5]), "=&r"(a[0][6]), "=&r"(a[0][7]),
        "=&r"(a[1][0]), "=&r"(a[1][1]), "=&r"(a[1][2]), "=&r"(a[1][3]), "=&r"(a[1][4]), "=&r"(a[1][5]), "=&r"(a[1][6]), "=&r"(a[1][7]),
        "=&r"(b[0][0]), "=&r"(b[0][1]), "=&r"(b[0][2]), "=&r"(b[0][3]), "=&r"(b[0][4]), "=&r"(b[0][5]), "=&r"(b[0][6]), "=&r"(b[0][7]),
        "=&r"(b[1][0]), "=&r"(b[1][1]), "=&r"(b[1][2]), "=&r"(b[1][3]), "=&r"(b[1][4]), "=&r"(b[1][5]), "=&r"(b[1][6]), "=&r"(b[1][7])
      : "r"(taddr_a), "r"(taddr_a + (16u << 16)), "r"(taddr_b), "r"(taddr_b + (16u << 16))
      : "memory");
}
// Four 8 x 8 bf16 matrices of such a fragment to shared memory: lane l gives the 16 bytes of row l % 8 of matrix l / 8.
__device__ __forceinline__ void stmatrix_x4(uint32_t saddr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(saddr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// 128 consecutive columns
__device__ __forceinline__ void tmem_ld32x4_wait(uint32_t taddr, uint32_t (&r)[4][32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%128];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%32, %33, %34, %35, %36, %37, %38, %39, %40, %41, %42, %43, %44, %45, %46, %47, "
      "%48, %49, %50, %51, %52, %53, %54, %55, %56, %57, %58, %59, %60, %61, %62, %63}, [%129];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%64, %65, %66, %67, %68, %69, %70, %71, %72, %73, %74, %75, %76, %77, %78, %79, "
      "%80, %81, %82, %83, %84, %85, %86, %87, %88, %89, %90, %91, %92, %93, %94, %95}, [%130];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%96, %97, %98, %99, %100, %101, %102, %103, %104, %105, %106, %107, %108, %109, %110, %111, "
      "%112, %113, %114, %115, %116, %117, %118, %119, %120, %121, %122, %123, %124, %125, %126, %127}, [%131];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=&r"(r[0][0]), "=&r"(r[0][1]), "=&r"(r[0][2]), "=&r"(r[0][3]), "=&r"(r[0][4]), "=&r"(r[0][5]), "=&r"(r[0][6]), "=&r"(r[0][7]),
        "=&r"(r[0][8]), "=&r"(r[0][9]), "=&r"(r[0][10]), "=&r"(r[0][11]), "=&r"(r[0][12]), "=&r"(r[0][13]), "=&r"(r[0][14]),
        "=&r"(r[0][15]), "=&r"(r[0][16]), "=&r"(r[0][17]), "=&r"(r[0][18]), "=&r"(r[0][19]), "=&r"(r[0][20]), "=&r"(r[0][21]),
        "=&r"(r[0][22]), "=&r"(r[0][23]), "=&r"(r[0][24]), "=&r"(r[0][25]), "=&r"(r[0][26]), "=&r"(r[0][27]), "=&r"(r[0][28]),
        "=&r"(r[0][29]), "=&r"(r[0][30]), "=&r"(r[0][31]), "=&r"(r[1][0]), "=&r"(r[1][1]), "=&r"(r[1][2]), "=&r"(r[1][3]),
        "=&r"(r[1][4]), "=&r"(r[1][5]), "=&r"(r[1][6]), "=&r"(r[1][7]), "=&r"(r[1][8]), "=&r"(r[1][9]), "=&r"(r[1][10]),
        "=&r"(r[1][11]), "=&r"(r[1][12]), "=&r"(r[1][13]), "=&r"(r[1][14]), "=&r"(r[1][15]), "=&r"(r[1][16]), "=&r"(r[1][17]),
        "=&r"(r[1][18]), "=&r"(r[1][19]), "=&r"(r[1][20]), "=&r"(r[1][21]), "=&r"(r[1][22]), "=&r"(r[1][23]), "=&r"(r[1][24]),
        "=&r"(r[1][25]), "=&r"(r[1][26]), "=&r"(r[1][27]), "=&r"(r[1][28]), "=&r"(r[1][29]), "=&r"(r[1][30]), "=&r"(r[1][31]),
        "=&r"(r[2][0]), "=&r"(r[2][1]), "=&r"(r[2][2]), "=&r"(r[2][3]), "=&r"(r[2][4]), "=&r"(r[2][5]), "=&r"(r[2][6]), "=&r"(r[2][7]),
        "=&r"(r[2][8]), "=&r"(r[2][9]), "=&r"(r[2][10]), "=&r"(r[2][11]), "=&r"(r[2][12]), "=&r"(r[2][13]), "=&r"(r[2][14]),
        "=&r"(r[2][15]), "=&r"(r[2][16]), "=&r"(r[2][17]), "=&r"(r[2][18]), "=&r"(r[2][19]), "=&r"(r[2][20]), "=&r"(r[2][21]),
        "=&r"(r[2][22]), "=&r"(r[2][23]), "=&r"(r[2][24]), "=&r"(r[2][25]), "=&r"(r[2][26]), "=&r"(r[2][27]), "=&r"(r[2][28]),
        "=&r"(r[2][29]), "=&r"(r[2][30]), "=&r"(r[2][31]), "=&r"(r[3][0]), "=&r"(r[3][1]), "=&r"(r[3][2]), "=&r"(r[3][3]),
        "=&r"(r[3][4]), "=&r"(r[3][5]), "=&r"(r[3][6]), "=&r"(r[3][7]), "=&r"(r[3][8]), "=&r"(r[3][9]), "=&r"(r[3][10]),
        "=&r"(r[3][11]), "=&r"(r[3][12]), "=&r"(r[3][13]), "=&r"(r[3][14]), "=&r"(r[3][15]), "=&r"(r[3][16]), "=&r"(r[3][17]),
        "=&r"(r[3][18]), "=&r"(r[3][19]), "=&r"(r[3][20]), "=&r"(r[3][21]), "=&r"(r[3][22]), "=&r"(r[3][23]), "=&r"(r[3][24]),
        "=&r"(r[3][25]), "=&r"(r[3][26]), "=&r"(r[3][27]), "=&r"(r[3][28]), "=&r"(r[3][29]), "=&r"(r[3][30]), "=&r"(r[3][31])
      : "r"(taddr), "r"(taddr + 32), "r"(taddr + 64), "r"(taddr + 96)
      : "memory");
}
// The wait by itself, for a load that other work goes on under: the empty statements behind it take the loaded registers in and out
// again, and all uses come after them (a copy of each register, so only where the overlap is worth more).
template <int N>
__device__ __forceinline__ void tmem_ld_tie(uint32_t (&r)[N]) {
  static_assert(N % 8 == 0, "whole groups of eight");
#pragma unroll
  for (int i = 0; i < N; i += 8)
    asm volatile("" : "+r"(r[i]), "+r"(r[i + 1]), "+r"(r[i + 2]), "+r"(r[i + 3]), "+r"(r[i + 4]), "+r"(r[i + 5]), "+r"(r[i + 6]), "+r"(r[i + 7]));
}
// r: every array loaded since the last wait
template <typename... R>
__device__ __forceinline__ void tmem_ld_wait(R&... r) {
  static_assert(sizeof...(R) > 0, "name the loaded registers");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
  (tmem_ld_tie(r), ...);
}

// ------------------------------------------------------------------ descriptors
// Shared-memory matrix descriptor, 128-byte swizzle (the layout TMA writes with CU_TENSOR_MAP_SWIZZLE_128B;
// tiles must start on a 1024-byte boundary).  Offsets are in bytes; the hardware fields drop the low 4 bits.
//   K-major tile  (rows = M or N index, 64 bf16 of K per 128-byte row):
//       lbo unused (set 16), sbo = 1024 (eight rows); step K by 16 elements = +32 bytes on the start address.
//   MN-major tile (rows = K index, 64 bf16 of M or N per 128-byte row, successive 64-wide MN chunks `lbo` bytes apart):
//       sbo = 1024 (eight K rows); step K by 16 rows = +2048 bytes on the start address.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version for sm_100
  d |= (uint64_t)2 << 61;  // SWIZZLE_128B
  return d;
}
// Instruction descriptor for kind::f16 with bf16 A/B, fp32 accumulate, dense.
// a_mn / b_mn: 0 = K-major operand, 1 = MN-major operand.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N, int a_mn, int b_mn) {
  return (1u << 4)            // D format fp32
         | (1u << 7)          // A bf16
         | (1u << 10)         // B bf16
         | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// Instruction descriptor for kind::f8f6f4 with E4M3 A / B (format code 0), fp32 accumulate, dense, both operands K-major.
// One instruction covers K = 32 elements (32 bytes per operand row).
__host__ __device__ constexpr uint32_t idesc_e4m3(int M, int N) {
  return (1u << 4)            // D format fp32
         | (0u << 7)          // A e4m3
         | (0u << 10)         // B e4m3
         | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// D[tmem] (+)= A[smem] * B[smem]; issued by ONE thread.
__device__ __forceinline__ void mma_bf16_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Same with the A operand in TMEM: [128 lanes = M rows] x K, bf16 pairs packed into 32-bit columns (k even in the low
// half), i.e. 8 columns per K = 16 step; always K-major.
__device__ __forceinline__ void mma_bf16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrive on `bar` once every tcgen05.mma issued so far by this thread has completed.
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// ------------------------------------------------------------------ CTA pairs (cta_group::2)
// Two CTAs of a cluster (ranks 2i and 2i+1, the even one is the leader) share one MMA: the leader's thread issues
// tcgen05.mma with M = 256; each CTA stages its 128 rows of A and its half of B's N rows in its own shared memory
// (same offsets in both) and owns 128 TMEM lanes x N accumulator columns.  Each CTA loads its own operand halves
// (no multicast) and reports the bytes to the LEADER's full barrier.
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_id_x() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%clusterid.x;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_nctarank() {      // CTAs of this cluster
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
// 16 bytes of the shared memory of any CTA of the cluster
__device__ __forceinline__ void ld_cluster_f32x4(uint32_t cluster_addr, float* x) {
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3]) : "r"(cluster_addr) : "memory");
}
__device__ __forceinline__ uint32_t cluster_count_x() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%nclusterid.x;" : "=r"(r));
  return r;
}
// shared::cluster address of the same shared-memory offset in CTA `rank` of this cluster
__device__ __forceinline__ uint32_t mapa_u32(uint32_t saddr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
  return r;
}
// All threads of all CTAs of the cluster.
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Arrival on a barrier of any CTA of the cluster, released at CTA scope: what it hands over are reads of tensor memory that have completed
// (tcgen05.wait), not writes.  Released at cluster scope it waits until the L2 has taken the stores before it, which in
// a GEMM's epilogue is ~3000 cycles of every tile (stamps, 16384 x 4096 x 768).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cta.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// Tiled loads into THIS CTA's shared memory whose completion bytes go to an mbarrier that may live in the peer CTA.
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* map, uint32_t bar_cluster_addr, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(map), "r"(bar_cluster_addr), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(void* smem_dst, const CUtensorMap* map, uint32_t bar_cluster_addr, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(map), "r"(bar_cluster_addr), "r"(x), "r"(y), "r"(z)
      : "memory");
}
// One full warp in EACH CTA of the pair (same warp index) runs these.
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_slot)), "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// D[tmem of both CTAs] (+)= A * B over the pair; issued by ONE thread of the leader CTA.
__device__ __forceinline__ void mma_bf16_ss_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                                 uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// The same with 8-bit (E4M3) operands: K = 32 per instruction, twice the multiply rate of kind::f16.
__device__ __forceinline__ void mma_e4m3_ss_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                                 uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrive on the mbarrier at this shared-memory offset in BOTH CTAs of the pair once the MMAs issued so far are done.
__device__ __forceinline__ void mma_commit_pair(uint64_t* bar) {
  const uint16_t mask = 3;
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
               "h"(mask)
               : "memory");
}

// One lane of a whole, converged warp, the same each time.  The threads that issue tcgen05.mma are chosen by it and not by `lane == 0`: only behind
// an election does the compiler know that one thread is there, and keeps descriptors in uniform registers; behind a comparison every MMA
// costs its thread 49 cycles and more whatever its size (back to back, M = 128, K = 16, A in TMEM: N = 64 48.8 -> 32.0 cycles, the
// tensor core's rate).  Attention forward + backward, us: 16 x 1024 tokens, 12 heads of 64 268.5 -> 263.5; 8 x 2048, 16 heads of 128
// 1017 -> 992; 32 x 197 without a mask 110.8 -> 101.7; forward 3 x 1000 28.6 -> 27.3.
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(pred));
  return pred != 0;
}

}  // namespace tc

// ------------------------------------------------------------------ host: tensor maps
// 2D row-major bf16 tensor [rows, cols] with `pitch_elems` elements between rows; box = [box_rows, 64 cols]
// (64 bf16 = one 128-byte swizzle row).  Requires 16-byte aligned base and pitch.  Returns false if the
// driver entry point is unavailable or the encode is rejected.
// `elem_bytes` = 2 (bf16), 4 (fp32; box_cols is then 32 so that a box row is still 128 bytes) or 1 (8-bit; box_cols 128).
bool mlb_make_tmap(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint64_t pitch_elems,
                   uint32_t box_rows, uint32_t box_cols, int elem_bytes);
// MN-major operand stored [k_rows, mn_cols] (mn contiguous, mn_cols a multiple of 64): a 3-D view
// {64 columns, k rows (pitch), mn_cols/64 chunks (128 bytes apart)} whose box {64, 64, chunks} lands in shared memory as
// `chunks` consecutive [64 rows x 128 B] swizzled blocks: the MN-major UMMA layout, fetched by ONE TMA instruction.
// Returns nullptr if the shape does not allow it or the driver rejects the map (callers fall back to 2-D boxes).
const CUtensorMap* mlb_tmap_mn3d_cached(const void* base, uint64_t k_rows, uint64_t mn_cols, uint64_t pitch_elems, uint32_t chunks);
// Cached lookup (key = all arguments); the returned pointer stays valid for the life of the process.
const CUtensorMap* mlb_tmap_cached(const void* base, uint64_t rows, uint64_t cols, uint64_t pitch_elems,
                                   uint32_t box_rows, uint32_t box_cols = 64, int elem_bytes = 2);
// [seqs][rows][cols] bf16, contiguous, box {64 columns, 64 rows, 1 sequence}, 128-byte swizzle: rows past a sequence's end read as
// zeros instead of the next sequence's.  Needs a 16-byte aligned base and cols a multiple of 8.
const CUtensorMap* mlb_tmap_seq3d_cached(const void* base, uint64_t seqs, uint64_t rows, uint64_t cols);
