// tcgen05 / TMA / cluster wrappers shared by the tensor-core GEMM kernels.
#pragma once

#include <cuda.h>

#include "rdq_common.cuh"

namespace rdq {

// ---- shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row groups 1024 B apart
__device__ __forceinline__ uint64_t make_desc_sw128(uint32_t smem_addr) {
  uint64_t d = (smem_addr & 0x3ffffu) >> 4;
  d |= 1ull << 16;                                  // leading byte offset (unused for swizzled K-major)
  d |= static_cast<uint64_t>(1024 >> 4) << 32;      // stride byte offset
  d |= 1ull << 46;                                  // version
  d |= 2ull << 61;                                  // SWIZZLE_128B
  return d;
}

// ---- TMA
__device__ __forceinline__ void prefetch_tensormap(const CUtensorMap *map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::
          "r"(dst),
      "l"(map), "r"(x), "r"(y), "r"(bar)
      : "memory");
}
// The box into L2 only.  That may run ahead of the grid-dependency wait whatever the kernel before writes:
// L2 is where its writes go, and the load that follows the wait reads them there.
__device__ __forceinline__ void tma_prefetch_2d(const CUtensorMap *map, int x, int y) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(map), "r"(x), "r"(y) : "memory");
}
// into this CTA's shared memory, completing on a barrier of either CTA of the pair
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3}], "
      "[%4];" ::"r"(dst),
      "l"(map), "r"(x), "r"(y), "r"(bar)
      : "memory");
}

// ---- clusters
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// ... in two halves, by every thread of the cluster
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ uint32_t mapa_u32(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ bool mbar_try_cluster(uint32_t bar, uint32_t parity, uint32_t ns) {
  uint32_t ok;
  asm volatile(
      "{\n.reg .pred p;\n"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n"
      "selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(ns)
      : "memory");
  return ok != 0;
}

// Wait on a barrier unless the CTA is aborting; raises the abort flag when about a second passed.  That
// second is for this launch's own work: what waits may wait for the launch before as well, which can take
// longer, so after a millisecond the wait goes on behind pdl_wait(), which has no limit of its own.
// The first try carries no time hint: it returns 40 cycles sooner when the phase is complete.
__device__ __forceinline__ bool mbar_try_now(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n.reg .pred p;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool gemm_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag) {
  if (mbar_try_now(smem_u32(bar), parity)) return true;
  for (int i = 0; i < 20000; ++i) {
    if (mbar_try(smem_u32(bar), parity, 50000u)) return true;
    if (*abort_flag) return false;
    if (i == 20) pdl_wait();
  }
  *abort_flag = 1;
  return false;
}
// ... with what the other CTA of the pair wrote before its arrival made visible
__device__ __forceinline__ bool gemm_wait_cluster(uint64_t *bar, uint32_t parity, volatile int *abort_flag) {
  for (int i = 0; i < 20000; ++i) {
    if (mbar_try_cluster(smem_u32(bar), parity, 50000u)) return true;
    if (*abort_flag) return false;
  }
  *abort_flag = 1;
  return false;
}
// The bounded wait as one asm block without branches that the compiler could see: 0 when it ran out
// (20000 tries of up to 50 us; the launch before has to be complete).
__device__ __forceinline__ uint32_t wait_bounded(uint32_t bar, uint32_t parity) {
  uint32_t left;
  asm volatile(
      "{\n.reg .pred p, q;\n"
      "mov.u32 %0, 20000;\n"
      "WAIT_%=:\n"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
      "@p bra DONE_%=;\n"
      "sub.u32 %0, %0, 1;\n"
      "setp.ne.u32 q, %0, 0;\n"
      "@q bra WAIT_%=;\n"
      "DONE_%=:\n}\n"
      : "=&r"(left)
      : "r"(bar), "r"(parity), "r"(50000u)
      : "memory");
  return left;
}
// ---- tiles whose k range several CTAs share
// Each of the `parts` CTAs leaves FP32 sums in the workspace and its four epilogue warps count themselves
// in a word of the tile (arrive_global).  When all are there, each CTA adds and stores a share of the
// tile's tokens.  That must not rely on the CTAs running at the same time -- kernels of another stream
// may hold the SMs that some of them need until these here give theirs up -- so a CTA that has waited for
// long leaves without doing anything (await_parts).  Nobody leaves once all have arrived, and the CTA
// that arrives last need not wait (its own warps have arrived when it asks): at least one is present then, and those present do the WHOLE tile
// when anyone has left.  The sums and their order are the same, so several doing it changes nothing.
// The word: warps arrived (bits 0-11), CTAs that left (12-21), CTAs done waiting (22-31).
constexpr int kPatience = 500;  // about half a millisecond: CTAs of a launch start within a few microseconds
constexpr uint32_t kMostParts = 1000;

// How many CTAs left, once all parts are there; -1: this CTA is to leave.
__device__ __forceinline__ int await_parts(uint32_t *word, uint32_t parts, int patience) {
  for (int i = 0;; ++i) {  // (ends: beyond the patience a failed exchange means that another CTA changed the word)
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(word) : "memory");
    if ((v & 0xfffu) == 4 * parts) return static_cast<int>((v >> 12) & 0x3ffu);
    if (i >= patience && atomicCAS(word, v, v + (1u << 12)) == v) return -1;
    if (i > 64) __nanosleep(100);
  }
}
// The CTAs present count themselves once they are done waiting; the last of them puts the word back to
// zero (later, when the answer has come).
__device__ __forceinline__ uint32_t pass_parts(uint32_t *word) { return atomicAdd(word, 1u << 22) >> 22; }
__device__ __forceinline__ void clear_parts(uint32_t *word, uint32_t passed, int left, uint32_t parts) {
  if (passed + 1 + left == parts) asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(word), "r"(0u) : "memory");
}
__device__ __forceinline__ void arrive_global(uint32_t *word) {
  asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(word) : "memory");
}

// One lane of a converged warp.  Loops that issue tcgen05 or TMA instructions run with the whole warp
// and issue under this predicate: behind `lane == 0` the compiler treats their operands as divergent
// and an MMA takes 97 cycles to issue (measured; 16 to 128 by shape under the predicate).
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile(
      "{\n.reg .pred p;\n"
      "elect.sync _|p, 0xffffffff;\n"
      "selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(p));
  return p != 0;
}

// ---- tcgen05
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// D(tensor memory) (+)= A(smem) . B(smem)^T, one CTA
__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
      "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}
// ... a pair of CTAs: each holds half of A's rows, half of B's rows and half of D's rows
__device__ __forceinline__ void umma_f16_pair(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
      "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// arrives on the barrier at this offset in both CTAs of the pair
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
      "h"(static_cast<uint16_t>(3))
      : "memory");
}
__device__ __forceinline__ void tmem_alloc(uint32_t dst, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst), "r"(cols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t tmem, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t dst, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst), "r"(cols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t tmem, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// 32 consecutive columns of the 32 lanes of this warp's quarter
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}

// ---- host: tensor map of a row-major matrix [rows, cols], boxes of box_cols x box_rows, 128-byte swizzle
int encode_2d(CUtensorMap *map, CUtensorMapDataType type, int elem_bytes, const void *base, int cols, int rows, int box_cols,
              int box_rows);
inline int encode_f16_2d(CUtensorMap *map, const void *base, int cols, int rows, int box_cols, int box_rows) {
  return encode_2d(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, base, cols, rows, box_cols, box_rows);
}

}  // namespace rdq
