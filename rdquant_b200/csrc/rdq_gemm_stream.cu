// Weight-streaming GEMM for a few dozen to a few hundred activation rows: packed weights go from
// shared memory through the format converters straight into TENSOR MEMORY, where tcgen05.mma takes
// them as its first operand.
//
//   y[M, N] = x[M, K] . W[N, K]^T * scale (+ bias)
//
// Bound: HBM (packed weight bytes) up to about a hundred rows, the tensor pipe and the activation
// traffic above.  Weights are the rows of the MMA (128 permuted rows of ONE format per tile) and
// tokens its columns (a multiple of 16 up to 128), so few rows cost few tensor cycles, and the
// converted weights never pass through shared memory: a converter thread owns one weight row, reads
// its packed bytes with conflict-free 16-byte loads and writes them as tensor-memory columns.
//
// Work: every tile is a run of 16 KB chunks (128 rows x 128 packed bytes = 256 / 128 / 64 k of
// NVFP4 / FP8 / FP16), all chunks of the layer are numbered in tile order and each CTA takes a
// contiguous range of equal cost (make_plan).  A tile inside one range is finished by its CTA.  The
// CTAs that share a tile cut by range borders leave FP32 partial sums in the workspace, wait for a while
// until all parts of the tile are there, and each adds and stores a share of its tokens, parts in CTA
// order: the result does not depend on timing (await_parts: those that leave, and who does their share).  A second kernel for these sums cost
// 4-7 us per layer, and one CTA per tile adding them up to 13 us.
//
// A stage of the pipeline is one chunk: up to 128 tensor-memory columns of weights and up to four
// 64-k activation boxes, on one barrier.  Every barrier wait of the issuing warp costs about 190 cycles
// and every hand-over of a converter group 300 to 1000, whatever the number of tokens: with 64-k
// stages the issuing warp needed 640 cycles per 64 k, with 128-k stages the converters 300, and a
// CTA's share of the HBM rate asks for 64 k every 250.
//
// Roles of a CTA's warps:
//   0        TMA of weight chunks (128 x 128 B boxes out of the row-major tensors, 128B swizzle)
//   1        TMA of activation boxes (tokens x 64 k)
//   2        MMA issue; tensor-memory allocation
//   3        block scales of NVFP4 chunks by cp.async, on the chunk's barrier
//   4-7      epilogue: tcgen05.ld, channel scale + bias, stores to y[token, perm[row]]
//   8-       converters, a group of four warps (a warp per 32 tensor-memory lanes) per stage: three
//            groups and stages of a chunk for up to 64 tokens; above, where the accumulators take more
//            tensor memory and a k block's MMAs longer, four groups and stages of half a chunk (two
//            of a whole one left the MMAs waiting: 1930 cycles per NVFP4 chunk of 128 tokens, whose
//            MMAs take 1024)
// Every launch is programmatic: it overlaps the end of the kernel before.  With RDQ_GEMV_PDL the
// weight and scale loads start before the grid-dependency wait.  Without it the first chunks are asked into
// L2 ahead of the wait and loaded from there behind it: with every thread waiting before the set-up, the
// first MMA came 1.7 us later than with the flag (2.6 us after the wait, 2560 -> 6144 at 32 rows).
//
// Reference behaviour replaced: 2 x marlin_gemm + F.linear + cat + index_select
// (rdquant/inference.py:620-677).
#include <cuda.h>

#include <algorithm>
#include <type_traits>
#include <unordered_map>

#include "rdq_gemm_common.cuh"
#include "rdq_kernels.cuh"

namespace rdq {

namespace {

// tokens per tile -> k blocks of 64 per stage, pipeline stages = converter groups: two accumulators of
// that many columns and 32 columns per k block of a stage share the 512 columns
template <int NT>
constexpr int kBlocks = NT == 64 ? 4 : 2;
template <int NT>
constexpr int kStages = (512 - 2 * NT) / (32 * kBlocks<NT>);
template <int NT>
constexpr int kThreads = (8 + 4 * kStages<NT>) * 32;
// (bounds for the compiler: 88 registers, so that 256 threads of a kernel with 32 fit beside the CTA)
template <int NT>
constexpr int kThreadBound = NT == 64 ? 736 : kThreads<NT>;
constexpr int kFinishThreads = 512;
constexpr int kChunkBytes = 128 * 128;
constexpr int kScaleBytes = 128 * 16;
constexpr int kMaxRing = 8;
constexpr int kSmemMax = 222 * 1024;
constexpr int kMaxTokens = 128;   // per token tile
constexpr int kMaxCtas = RDQ_LINEAR_WORDS;
static_assert(kMaxCtas <= kMostParts, "fields of a shared tile's word");

// Chunks of the layer in processing order: NVFP4 tiles, FP8 tiles, FP16 tiles; inside a channel tile
// its token tiles one after another.
struct StreamSched {
  int mt, nt, M;            // token tiles, tokens per tile
  int S[3];                 // chunks per tile
  int E[3];                 // end of each format's chunk range
  int nkb;                  // k blocks of 64
  int G;                    // CTAs
  int bnd[kMaxCtas + 1];    // first chunk of each CTA
};
struct Segment {
  int fmt, row_tile, m_tile;  // 128-row tile inside the format group, token tile
  int c0, c1;                 // chunks of the tile
  int start;                  // global index of the tile's first chunk
};
__device__ __forceinline__ Segment segment_at(const StreamSched &s, int chunk, int end) {
  Segment g;
  g.fmt = chunk < s.E[0] ? 0 : (chunk < s.E[1] ? 1 : 2);
  const int base = g.fmt == 0 ? 0 : s.E[g.fmt - 1];
  const int S = s.S[g.fmt];
  const int t = (chunk - base) / S;
  g.start = base + t * S;
  g.row_tile = t / s.mt;
  g.m_tile = t - g.row_tile * s.mt;
  g.c0 = chunk - g.start;
  g.c1 = min(S, end - g.start);
  return g;
}

struct StreamArgs {
  const uint8_t *s4;
  const float *s8;
  float global4;
  const int32_t *perm;
  const __half *bias;
  void *y;
  int n4, n8, n16, K, N;
  float *partial;    // [2 * CTA + (0 first, 1 last segment)][token][128 rows]
  uint32_t *arrived;  // [CTA in which a cut tile starts]: its word (await_parts)
  int patience;
  int nw;             // weight chunks in flight
  int early;          // weights may be read before the kernel before this one has finished
  int scale_bytes;  // a block-scale row is copied 16, 8 or 4 bytes at a time
  int test_timeout;
};

// output column, scale and bias of a row
struct Row {
  bool live;
  int col;
  float scl, bia;
};
struct StreamSmem {
  Row cut[2][128];  // rows of the range's first and last tile, for finish_shared
  uint64_t w_full[kMaxRing], w_empty[kMaxRing];
  uint64_t full[4], empty[4];
  uint64_t d_full[2], d_empty[2];
  uint64_t never;
  uint32_t tmem_base;
  int abort_flag;
  int left[2];  // finish_shared: what await_parts answered
};

// position in a ring
// the CTAs that hold a cut tile: `from` holds its start
__device__ __forceinline__ int first_cta(const StreamSched &s, int b, int tile_start) {
  while (s.bnd[b] > tile_start) --b;
  return b;
}
__device__ __forceinline__ int last_cta(const StreamSched &s, int b, int tile_end) {
  while (s.bnd[b + 1] < tile_end) ++b;
  return b;
}
// workspace slot of CTA c's part of the tile that starts in CTA `from`: a range's first segment goes
// to the even slot, its last to the odd one
__device__ __forceinline__ long long part_slot(const StreamSched &s, int c, int from, int tile_start) {
  return 2ll * c + (c == from && s.bnd[c] < tile_start ? 1 : 0);
}

struct Cursor {
  int i = 0;
  uint32_t ph = 0;
  __device__ __forceinline__ void next(int n) {
    if (++i == n) {
      i = 0;
      ph ^= 1;
    }
  }
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(uint32_t dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_arrive(uint32_t bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ uint4 lds16(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
// 16 tensor-memory columns (32 k) of this warp's 32 lanes
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// D (+)= A(tensor memory) . B(smem)^T.  The descriptor comes in halves: only the low one changes from
// MMA to MMA, and every operand that changes costs the issuing warp a register move.
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint32_t db_lo, uint32_t db_hi, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\n.reg .b64 db;\nsetp.ne.b32 p, %5, 0;\nmov.b64 db, {%2, %3};\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n}\n" ::"r"(tmem_d),
      "r"(tmem_a), "r"(db_lo), "r"(db_hi), "r"(idesc), "r"(accumulate)
      : "memory");
}
// MMAs FROM .. TO - 1 of a stage (four to a k block of 64)
template <int FROM, int TO>
__device__ __forceinline__ void issue_mmas(uint32_t acc, uint32_t wa, uint32_t dx, uint32_t dx_hi, uint32_t box, uint32_t idesc,
                                           uint32_t accumulate) {
#pragma unroll
  for (int i = 0; i < TO; ++i) {
    if (i >= FROM) umma_f16_ts(acc, wa + 8 * i, dx + 2 * (i & 3), dx_hi, idesc, i == 0 ? accumulate : 1u);
    if ((i & 3) == 3) dx += box;
  }
}

// half a k block (32 k) of one weight row -> 16 tensor-memory columns
__device__ __forceinline__ void convert_fp4(const uint4 &q, uint32_t scales, uint32_t (&o)[16]) {
  const uint32_t s2 = cvt_e4m3x2(scales);
  const uint32_t s0 = __byte_perm(s2, 0u, 0x1010u), s1 = __byte_perm(s2, 0u, 0x3232u);
  cvt_e2m1x8(q.x, o[0], o[1], o[2], o[3]);
  cvt_e2m1x8(q.y, o[4], o[5], o[6], o[7]);
  cvt_e2m1x8(q.z, o[8], o[9], o[10], o[11]);
  cvt_e2m1x8(q.w, o[12], o[13], o[14], o[15]);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    o[i] = hmul2_u32(o[i], s0);
    o[8 + i] = hmul2_u32(o[8 + i], s1);
  }
}
__device__ __forceinline__ void convert_fp8(const uint4 &a, const uint4 &b, uint32_t (&o)[16]) {
  cvt_e4m3x4(a.x, o[0], o[1]);
  cvt_e4m3x4(a.y, o[2], o[3]);
  cvt_e4m3x4(a.z, o[4], o[5]);
  cvt_e4m3x4(a.w, o[6], o[7]);
  cvt_e4m3x4(b.x, o[8], o[9]);
  cvt_e4m3x4(b.y, o[10], o[11]);
  cvt_e4m3x4(b.z, o[12], o[13]);
  cvt_e4m3x4(b.w, o[14], o[15]);
}

// row r of a segment's tile
__device__ __forceinline__ Row row_of(const StreamArgs &a, const Segment &g, int r, bool wanted) {
  Row w;
  const int row = g.row_tile * 128 + r;  // row inside the format group
  const int rows = g.fmt == 0 ? a.n4 : (g.fmt == 1 ? a.n8 : a.n16);
  const int prow = row + (g.fmt == 0 ? 0 : (g.fmt == 1 ? a.n4 : a.n4 + a.n8));
  w.live = row < rows;
  w.col = 0;
  w.scl = 0.f;
  w.bia = 0.f;
  if (w.live && wanted) {
    w.col = a.perm ? a.perm[prow] : prow;
    w.scl = g.fmt == 0 ? a.global4 : (g.fmt == 1 ? a.s8[row] : 1.f);
    w.bia = a.bias ? __half2float(a.bias[w.col]) : 0.f;
  }
  return w;
}

template <bool BF16>
__device__ __forceinline__ void store_row(void *y, long long i, float v) {
  if (BF16) static_cast<__nv_bfloat16 *>(y)[i] = __float2bfloat16_rn(v);
  else static_cast<__half *>(y)[i] = __float2half_rn(v);
}

// Half of the first 512 threads: waits until all parts of the segment's tile are in the workspace,
// then adds and stores this CTA's share of its tokens, or all of them when CTAs have left.  `sub` (0, 1) and r (row) identify the thread.
// kPart parts of kTok tokens are read at a time: four of eight for narrow token tiles (a small layer's
// tile has three or four parts), two of sixteen for wide ones.
template <bool BF16, int kPart, int kTok>
__device__ __forceinline__ void finish_shared(const StreamArgs &a, const StreamSched &sc, const Segment &g, const Row &row, int r,
                                              int sub, int bar_id, volatile int *answer) {
  const int b0 = first_cta(sc, blockIdx.x, g.start), b1 = last_cta(sc, blockIdx.x, g.start + sc.S[g.fmt]);
  const int parts = b1 - b0 + 1;
  const int tok0 = g.m_tile * sc.nt;
  const int ntok = min(sc.nt, sc.M - tok0);
  if (r == 0 && sub == 0) *answer = await_parts(a.arrived + b0, parts, a.patience);
  asm volatile("bar.sync %0, %1;" ::"r"(bar_id), "n"(kFinishThreads / 2) : "memory");
  const int left = *answer;
  if (left < 0) return;
  const uint32_t passed = r == 0 && sub == 0 ? pass_parts(a.arrived + b0) : 0u;
  const int share = static_cast<int>(blockIdx.x) - b0;
  const int lo = left ? 0 : ntok * share / parts, hi = left ? ntok : ntok * (share + 1) / parts;
  constexpr int kSub = 2;
#pragma unroll 1
  for (int t0 = lo + sub; t0 < hi; t0 += kTok * kSub) {
    float v[kTok];
#pragma unroll
    for (int e = 0; e < kTok; ++e) v[e] = 0.f;
#pragma unroll 1
    for (int b = b0; b <= b1; b += kPart) {
      // the loads of kPart parts in flight
      float p[kPart][kTok];
#pragma unroll
      for (int i = 0; i < kPart; ++i) {
        const float *src = a.partial + (part_slot(sc, min(b + i, b1), b0, g.start) * sc.nt + t0) * 128 + r;
#pragma unroll
        for (int e = 0; e < kTok; ++e) p[i][e] = t0 + e * kSub < hi && b + i <= b1 ? __ldcg(src + e * kSub * 128) : 0.f;
      }
#pragma unroll
      for (int i = 0; i < kPart; ++i)
#pragma unroll
        for (int e = 0; e < kTok; ++e) v[e] += p[i][e];
    }
    if (row.live) {
#pragma unroll
      for (int e = 0; e < kTok; ++e)
        if (t0 + e * kSub < hi)
          store_row<BF16>(a.y, 1ll * (tok0 + t0 + e * kSub) * a.N + row.col, fmaf(v[e], row.scl, row.bia));
    }
  }
  if (r == 0 && sub == 0) clear_parts(a.arrived + b0, passed, left, parts);
}

// NT: most tokens per tile (64 or 128)
template <int NT, bool BF16>
__global__ void __launch_bounds__(kThreadBound<NT>, 1)
gemm_stream_kernel(const __grid_constant__ CUtensorMap w4map, const __grid_constant__ CUtensorMap w8map,
                   const __grid_constant__ CUtensorMap w16map, const __grid_constant__ CUtensorMap xmap,
                   const __grid_constant__ StreamArgs a, const __grid_constant__ StreamSched sc, int *status) {
  constexpr int NS = kStages<NT>, KB = kBlocks<NT>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ StreamSmem S;
  const uint32_t w_ring = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t x_ring = w_ring + a.nw * kChunkBytes;
  const uint32_t x_bytes = static_cast<uint32_t>(sc.nt) * 128;  // one 64-k box
  const uint32_t s_ring = x_ring + NS * KB * x_bytes;
  // (from lane 0, so that the compiler keeps the roles' branches and loops in uniform registers)
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int begin = sc.bnd[blockIdx.x], end = sc.bnd[blockIdx.x + 1];
  auto wmap = [&](int fmt) { return fmt == 0 ? &w4map : (fmt == 1 ? &w8map : &w16map); };
  auto load_chunk = [&](const Segment &g, int c, int slot) {
    const uint32_t bar = smem_u32(&S.w_full[slot]);
    mbar_arrive_expect_tx(bar, kChunkBytes);
    tma_load_2d(w_ring + slot * kChunkBytes, wmap(g.fmt), c * (g.fmt == 2 ? 64 : 128), g.row_tile * 128, bar);
  };
  // The first weight chunks are on their way before anything else is set up; without leave to read weights
  // early, on their way into L2.
  const int ahead = min(a.nw, end - begin), early = a.early ? ahead : 0;
  if (threadIdx.x == 0) {
    for (int i = 0; i < a.nw; ++i) {
      mbar_init(smem_u32(&S.w_full[i]), 1 + 32);  // the TMA thread and the scale warp's lanes
      mbar_init(smem_u32(&S.w_empty[i]), 16 / KB);  // the groups that convert a chunk of four k blocks
    }
    mbar_init_fence();
    Segment g = segment_at(sc, begin, end);
    for (int i = 0; i < ahead; ++i) {
      if (begin + i == g.start + g.c1) g = segment_at(sc, begin + i, end);
      if (a.early) load_chunk(g, begin + i - g.start, i);
      else tma_prefetch_2d(wmap(g.fmt), (begin + i - g.start) * (g.fmt == 2 ? 64 : 128), g.row_tile * 128);
    }
  }
  if (threadIdx.x == 32) {
    for (int i = 0; i < NS; ++i) {
      mbar_init(smem_u32(&S.full[i]), 1 + 4);  // the activation loads and the group's warps
      mbar_init(smem_u32(&S.empty[i]), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&S.d_full[i]), 1);
      mbar_init(smem_u32(&S.d_empty[i]), 4);
    }
    mbar_init(smem_u32(&S.never), 1);
    S.abort_flag = 0;
    mbar_init_fence();
  }
  if (warp == 2) tmem_alloc(smem_u32(&S.tmem_base), 512);
  if (warp == 3 && lane == 0) prefetch_tensormap(&xmap);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = S.tmem_base;
  const uint32_t tmem_a = tmem + 2 * NT;

  // stages of a range: its NVFP4 chunks (they come first) take several each above 64 tokens
  constexpr int split = 4 / KB;
  const int n4 = max(0, min(end, sc.E[0]) - begin);
  const int stages = split * n4 + (end - begin - n4);

  if (warp == 0) {
    // ---------------------------------------------------------------- weight chunks
    const bool leader = elect_one();
    if (!a.early) pdl_wait();
    Cursor w;
    if (early == a.nw) w.ph ^= 1;
    else w.i = early;
    Segment g = segment_at(sc, begin, end);
    for (int i = begin + early; i < end; ++i) {
      if (i >= g.start + g.c1) g = segment_at(sc, i, end);
      if (!gemm_wait(&S.w_empty[w.i], w.ph ^ 1, &S.abort_flag)) break;
      if (leader) load_chunk(g, i - g.start, w.i);
      w.next(a.nw);
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- activation boxes
    const bool leader = elect_one();
    pdl_wait();
    pdl_launch_dependents();
    Cursor x;
    Segment g = segment_at(sc, begin, end);
    for (int i = begin; i < end; ++i) {
      if (i >= g.start + g.c1) g = segment_at(sc, i, end);
      const int per = 4 >> g.fmt;  // k blocks of 64 per chunk
      const int kb0 = (i - g.start) * per, blocks = min(per, sc.nkb - kb0);
      bool ok = true;
      for (int b = 0; b < per && ok; b += KB) {  // stages of the chunk; past K a stage can be empty
        ok = gemm_wait(&S.empty[x.i], x.ph ^ 1, &S.abort_flag);
        if (ok && leader) {
          const uint32_t bar = smem_u32(&S.full[x.i]);
          const uint32_t dst = x_ring + x.i * KB * x_bytes;
          const int nb = min(KB, blocks - b);
          if (nb > 0) mbar_arrive_expect_tx(bar, nb * x_bytes);
          else mbar_arrive(bar);
          for (int j = 0; j < nb; ++j) tma_load_2d(dst + j * x_bytes, &xmap, (kb0 + b + j) * 64, g.m_tile * sc.nt, bar);
        }
        x.next(NS);
      }
      if (!ok) break;
    }
  } else if (warp == 2) {
    // ---------------------------------------------------------------- MMA issue
    // The inner loop is kept to a wait in one asm block, the MMAs and a commit: with anything that can
    // diverge in it, every MMA's operands are moved to uniform registers again and an MMA takes 60
    // cycles to issue instead of 20.
    const bool leader = elect_one();
    pdl_wait();  // (it needs the activations in any case, and its bounded waits are for this launch's own work)
    const uint32_t idesc = (1u << 4) | (static_cast<uint32_t>(sc.nt >> 3) << 17) | (8u << 24);
    const uint64_t desc0 = make_desc_sw128(x_ring);
    const uint32_t dx0 = static_cast<uint32_t>(desc0), dx_hi = static_cast<uint32_t>(desc0 >> 32), box = x_bytes >> 4;
    const uint32_t full0 = smem_u32(&S.full[0]), empty0 = smem_u32(&S.empty[0]);
    uint32_t stage = 0, ph = 0;
    Cursor d;
    int left = stages;
    uint32_t ok = NT > 64 ? wait_bounded(full0, 0) : 1u;
    tc_fence_after();
    for (int ck = begin; ck < end && ok;) {
      const Segment g = segment_at(sc, ck, end);
      const int per = 4 >> g.fmt;
      if (!gemm_wait(&S.d_empty[d.i], d.ph ^ 1, &S.abort_flag)) break;
      tc_fence_after();
      const uint32_t acc = tmem + d.i * NT;
      const int bps = min(per, KB);                                    // k blocks of a stage
      const int blocks = min(g.c1 * per, sc.nkb) - g.c0 * per;
      const int whole = blocks / bps, rest = blocks - whole * bps;     // stages with all of them
      const int none = (g.c1 - g.c0) * (per / bps) - whole - (rest > 0);  // stages past K
      uint32_t accumulate = 0;
      // Above 64 tokens the next stage is waited for ahead of the last two MMAs of the present one: the
      // tensor pipe takes an MMA when the one before last is done, so that a wait between stages is a
      // gap of 140 cycles in its work (1700 -> 1540 cycles per NVFP4 chunk of 128 tokens).
      auto run = [&](auto blocks, int count) {
        constexpr int n = 4 * decltype(blocks)::value, head = NT == 64 ? 0 : (n > 2 ? n - 2 : 0);
#pragma unroll 1
        for (int i = 0; i < count; ++i) {
          const uint32_t wa = tmem_a + stage * (32 * KB), dx = dx0 + stage * KB * box, empty = empty0 + stage * 8;
          if (NT == 64) {  // (with few columns the weights are what a stage waits for, and its release must not)
            ok = wait_bounded(full0 + stage * 8, ph);
            if (!ok) break;
            tc_fence_after();
          } else if (leader) {
            issue_mmas<0, head>(acc, wa, dx, dx_hi, box, idesc, accumulate);
          }
          stage = stage + 1 == NS ? 0 : stage + 1;
          ph ^= stage == 0;
          if (NT > 64) {
            if (--left > 0) ok = wait_bounded(full0 + stage * 8, ph);
            tc_fence_after();
          }
          if (leader) {
            issue_mmas<head, n>(acc, wa, dx, dx_hi, box, idesc, accumulate);
            umma_commit(empty);
          }
          accumulate = 1;
          if (!ok) break;
        }
      };
      if (bps == 4) run(std::integral_constant<int, 4>(), whole);
      else if (bps == 2) run(std::integral_constant<int, 2>(), whole);
      else run(std::integral_constant<int, 1>(), whole);
      if (rest == 3) run(std::integral_constant<int, 3>(), 1);
      else if (rest == 2) run(std::integral_constant<int, 2>(), 1);
      else if (rest == 1) run(std::integral_constant<int, 1>(), 1);
      run(std::integral_constant<int, 0>(), none);
      if (ok && leader) umma_commit(smem_u32(&S.d_full[d.i]));
      d.next(2);
      ck = g.start + g.c1;
    }
    if (!ok) S.abort_flag = 1;
    __syncwarp();
  } else if (warp == 3) {
    // ------------------------------------------------------------------ block scales
    // (a row's address once per tile: with it computed per chunk this warp was late at times; 8192 -> 57344 at 16 rows 56.3 us, now 55.3)
    if (!a.early) pdl_wait();
    Cursor w;
    const int pitch = a.K >> 4;
    Segment g;
    g.start = g.c1 = 0;
    const uint8_t *src[4];
    int rows = 0;
    for (int i = begin; i < end; ++i) {
      if (i == begin || i >= g.start + g.c1) {
        g = segment_at(sc, i, end);
        rows = g.fmt != 0 ? 0 : 4;
#pragma unroll
        for (int u = 0; u < 4; ++u) src[u] = a.s4 + 1ll * min(g.row_tile * 128 + u * 32 + lane, a.n4 - 1) * pitch;
      }
      if (!gemm_wait(&S.w_empty[w.i], w.ph ^ 1, &S.abort_flag)) break;
      const int c = i - g.start;
      const uint32_t dst = s_ring + w.i * kScaleBytes + lane * 16;
      if (a.scale_bytes == 16) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (u < rows) cp_async16(dst + u * 512, src[u] + c * 16);
      } else {
        const int words = min(4, sc.nkb - 4 * c);
        for (int u = 0; u < 4; ++u) {
          if (u >= rows) break;
          const uint8_t *from = u == 0 ? src[0] : (u == 1 ? src[1] : (u == 2 ? src[2] : src[3]));
          for (int j = 0; j < words; j += a.scale_bytes >> 2) {
            if (a.scale_bytes == 8) cp_async8(dst + u * 512 + 4 * j, from + c * 16 + 4 * j);
            else cp_async4(dst + u * 512 + 4 * j, from + c * 16 + 4 * j);
          }
        }
      }
      cp_async_arrive(smem_u32(&S.w_full[w.i]));
      w.next(a.nw);
    }
  } else if (warp < 8) {
    // ------------------------------------------------------------------ epilogue
    const int q = warp & 3;
    const uint32_t lanes = static_cast<uint32_t>(q * 32) << 16;
    if (!a.early) pdl_wait();
    // constants of the rows that are finished together with other CTAs: fetched now, when nobody waits
    S.cut[0][q * 32 + lane] = row_of(a, segment_at(sc, begin, end), q * 32 + lane, true);
    S.cut[1][q * 32 + lane] = row_of(a, segment_at(sc, end - 1, end), q * 32 + lane, true);
    Cursor d;
    bool first = true;
    for (int ck = begin; ck < end;) {
      const Segment g = segment_at(sc, ck, end);
      const bool whole = g.c0 == 0 && g.c1 == sc.S[g.fmt];
      const Row row = row_of(a, g, q * 32 + lane, whole);
      const int tok0 = g.m_tile * sc.nt;
      const int ntok = min(sc.nt, sc.M - tok0);
      if (!gemm_wait(&S.d_full[d.i], d.ph, &S.abort_flag)) break;
      tc_fence_after();
      const uint32_t acc = tmem + d.i * NT + lanes;
      float *part = a.partial + (2ll * blockIdx.x + (first ? 0 : 1)) * sc.nt * 128 + q * 32 + lane;
      uint16_t *yp = static_cast<uint16_t *>(a.y) + 1ll * tok0 * a.N + row.col;
      // sixteen tokens at a time; the stores of one batch overlap the load of the next
      uint32_t v[2][16];
      tmem_ld16(acc, v[0]);
      auto batch = [&](uint32_t (&cur)[16], uint32_t (&nxt)[16], int c) {
        tmem_wait_ld();
        if (c + 16 < ntok) {
          tmem_ld16(acc + c + 16, nxt);
        } else {  // the accumulator is free once its last columns are read
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&S.d_empty[d.i]));
        }
        const int n = min(16, ntok - c);
        if (!whole) {
          if (n == 16) {
#pragma unroll
            for (int e = 0; e < 16; ++e) part[(c + e) * 128] = __uint_as_float(cur[e]);
          } else {
#pragma unroll
            for (int e = 0; e < 16; ++e)
              if (e < n) part[(c + e) * 128] = __uint_as_float(cur[e]);
          }
        } else if (row.live) {
          uint16_t *p = yp;
#pragma unroll
          for (int e = 0; e < 16; e += 2) {
            const uint32_t h = pack_y2(fmaf(__uint_as_float(cur[e]), row.scl, row.bia),
                                       fmaf(__uint_as_float(cur[e + 1]), row.scl, row.bia), BF16);
            if (e < n) p[0] = static_cast<uint16_t>(h);
            if (e + 1 < n) p[a.N] = static_cast<uint16_t>(h >> 16);
            p += 2 * a.N;
          }
          yp += 16ll * a.N;
        }
      };
      for (int c = 0; c < ntok; c += 32) {
        batch(v[0], v[1], c);
        if (c + 16 < ntok) batch(v[1], v[0], c + 16);
      }
      if (!whole) {
        __threadfence();
        __syncwarp();
        if (lane == 0) arrive_global(a.arrived + first_cta(sc, blockIdx.x, g.start));
      }
      first = false;
      d.next(2);
      ck = g.start + g.c1;
    }
  } else {
    // ------------------------------------------------------------------ converters
    // Group `grp` owns stage `grp` and takes every NS-th stage's worth of chunks: a part of an NVFP4
    // chunk (`split` to a chunk) or a whole chunk of the other formats.  It waits for the release of its
    // stage first: the MMAs have then consumed every stage up to NS before this one, so the parity it
    // tests on the chunk's barrier (used by chunk i - nw before, nw >= NS) cannot be a round old.
    const int q = warp & 3, grp = (warp - 8) >> 2;
    const int row = q * 32 + lane;
    const uint32_t rbase = row * 128, sw = row & 7;
    const uint32_t dst = tmem_a + grp * (32 * KB) + (static_cast<uint32_t>(q * 32) << 16);
    int slot = 0, last = begin;
    uint32_t w_ph = 0, ph = 0;
    Segment g;
    g.start = g.c1 = 0;
    for (int j = grp; j < stages; j += NS) {
      const int i = j < split * n4 ? begin + j / split : begin + n4 + (j - split * n4);
      const int part = j < split * n4 ? j % split : 0;
      slot += i - last;  // at most NS further
      last = i;
      if (slot >= a.nw) {
        slot -= a.nw;
        w_ph ^= 1;
      }
      if (j == grp || i >= g.start + g.c1) g = segment_at(sc, i, end);
      if (!gemm_wait(&S.empty[grp], ph ^ 1, &S.abort_flag)) break;
      if (!gemm_wait(&S.w_full[slot], w_ph, &S.abort_flag)) break;
      tc_fence_after();
      const uint32_t base = w_ring + slot * kChunkBytes + rbase;
      auto piece = [&](int p) { return lds16(base + ((p ^ sw) << 4)); };
      uint32_t o[16];
      if (g.fmt == 0) {
        // (k blocks beyond K convert the zero fill of the box; the MMAs do not read them)
        const uint4 s4 = lds16(s_ring + slot * kScaleBytes + row * 16);
        const uint32_t sc4[4] = {part ? s4.z : s4.x, part ? s4.w : s4.y, s4.z, s4.w};
        // Four pieces are read ahead of their conversion: one after the other, each waited for its own read.
        uint4 v[4] = {piece(2 * KB * part), piece(2 * KB * part + 1), piece(2 * KB * part + 2), piece(2 * KB * part + 3)};
#pragma unroll
        for (int h = 0; h < 2 * KB; ++h) {
          convert_fp4(v[h & 3], sc4[h >> 1] >> (16 * (h & 1)), o);
          if (h + 4 < 2 * KB) v[h & 3] = piece(2 * KB * part + h + 4);
          tmem_st16(dst + 16 * h, o);
        }
      } else if (g.fmt == 1) {
        uint4 v[4] = {piece(0), piece(1), piece(2), piece(3)};
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          convert_fp8(v[2 * (h & 1)], v[2 * (h & 1) + 1], o);
          if (h < 2) {
            v[2 * h] = piece(2 * h + 4);
            v[2 * h + 1] = piece(2 * h + 5);
          }
          tmem_st16(dst + 16 * h, o);
        }
      } else {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
#pragma unroll
          for (int p = 0; p < 4; ++p) {
            const uint4 v = piece(4 * h + p);
            o[4 * p] = v.x;
            o[4 * p + 1] = v.y;
            o[4 * p + 2] = v.z;
            o[4 * p + 3] = v.w;
          }
          tmem_st16(dst + 16 * h, o);
        }
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(smem_u32(&S.full[grp]));
        mbar_arrive(smem_u32(&S.w_empty[slot]), g.fmt == 0 ? 1u : static_cast<uint32_t>(split));
      }
      ph ^= 1;
    }
  }

  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 2) tmem_dealloc(tmem, 512);
  // ---- tiles shared with other CTAs: half of 512 threads take the range's first segment, half its last
  if (!S.abort_flag && begin < end && threadIdx.x < kFinishThreads) {
    const int half = threadIdx.x >> 8;
    Segment g = segment_at(sc, begin, end);
    bool mine = half == 0;
    if (half == 1 && g.start + g.c1 < end) {
      mine = true;
      g = segment_at(sc, end - 1, end);
      g = segment_at(sc, max(g.start, begin), end);
    }
    if (mine && !(g.c0 == 0 && g.c1 == sc.S[g.fmt]))
      finish_shared<BF16, NT == 64 ? 4 : 2, NT == 64 ? 8 : 16>(a, sc, g, S.cut[half][threadIdx.x & 127], threadIdx.x & 127, (threadIdx.x >> 7) & 1, 1 + half, &S.left[half]);
  }
  __syncthreads();
  if (S.abort_flag) {
    linger(16000);  // let copies that are still in flight land before the shared memory is given up
    __syncthreads();
    if (threadIdx.x == 0) atomicExch(status, 1);
  }
  if (a.test_timeout && threadIdx.x == 0 && blockIdx.x == 0) {
    if (!mbar_wait(smem_u32(&S.never), 0, 3u)) atomicExch(status, 2);
  }
}

struct StreamPlan {
  StreamSched sc;
  int wide, nw, smem;  // wide: the variant for more than 64 tokens per tile
};

// Token tiles of equal width; a chunk costs what bounds it: its bytes at the SM's share of the HBM
// rate (23 B/clk; the other token tiles find it in L2), the conversion of its k blocks, or its stages
// in the tensor pipe.
StreamPlan make_plan(int n4, int n8, int n16, int M, int K) {
  StreamPlan p;
  StreamSched &s = p.sc;
  s.M = M;
  s.mt = (M + kMaxTokens - 1) / kMaxTokens;
  s.nt = ((M + s.mt - 1) / s.mt + 15) / 16 * 16;
  s.nkb = (K + 63) / 64;
  const int n[3] = {n4, n8, n16};
  const double bytes[3] = {kChunkBytes + kScaleBytes, kChunkBytes, kChunkBytes};
  int e = 0, u[3];
  long long w = 0, W[3];
  for (int f = 0; f < 3; ++f) {
    const int per = 4 >> f;
    s.S[f] = (s.nkb + per - 1) / per;
    // (measured on 128 x 128 tiles: 1540 / 825 / 581 cycles per NVFP4 / FP8 / FP16 chunk)
    const int bps = std::min(per, kBlocks<128>);
    const double conv = f == 0 ? 170 : (f == 1 ? 150 : 90);
    const double work = s.nt > 64 ? per / bps * (300 + 1.85 * bps * s.nt) : per * std::max(conv, 2.0 * s.nt);
    // the few FP16 channels lie far apart: every value of their tiles is a memory sector of its own,
    // 52000 cycles of stores for 128 x 128 of them (an FP16 CTA was 10 us late at 512 tokens)
    const double scattered = f == 2 && s.nt > 64 ? 410.0 * s.nt / s.S[f] : 0.0;
    u[f] = static_cast<int>(std::max(bytes[f] / (23.0 * s.mt), work) + scattered);
    const int chunks = (n[f] + 127) / 128 * s.mt * s.S[f];
    e += chunks;
    w += 1ll * chunks * u[f];
    s.E[f] = e;
    W[f] = w;
  }
  // A CTA's share is not below three of the most expensive chunks: tiles cut into more parts cost more
  // to put together than they gain (1024 x 2560, 32 rows: one chunk each 14.2 us, three 11.0).
  const long long least = 3ll * std::max({u[0], u[1], u[2]});
  s.G = static_cast<int>(std::min<long long>(std::min(sm_count(), kMaxCtas), std::max(1ll, w / least)));
  for (int b = 0; b < s.G; ++b) {
    const long long pos = w * b / s.G;
    s.bnd[b] = static_cast<int>(pos < W[0] ? pos / u[0]
                                           : (pos < W[1] ? s.E[0] + (pos - W[0]) / u[1] : s.E[1] + (pos - W[1]) / u[2]));
  }
  s.bnd[s.G] = e;
  p.wide = s.nt > 64;
  const int xb = (p.wide ? kStages<128> * kBlocks<128> : kStages<64> * kBlocks<64>) * s.nt * 128;
  p.nw = std::min(kMaxRing, (kSmemMax - 1024 - xb) / (kChunkBytes + kScaleBytes));
  p.smem = 1024 + xb + p.nw * (kChunkBytes + kScaleBytes);
  return p;
}

// the plans of the last few thousand (layer shape, rows) pairs of this thread
const StreamPlan &stream_plan(int n4, int n8, int n16, int M, int K) {
  struct Key {
    int v[6];
    bool operator==(const Key &o) const { return std::equal(v, v + 6, o.v); }
  };
  struct Hash {
    size_t operator()(const Key &k) const {
      size_t h = 1469598103934665603ull;
      for (int x : k.v) h = (h ^ static_cast<size_t>(x)) * 1099511628211ull;
      return h;
    }
  };
  static thread_local std::unordered_map<Key, StreamPlan, Hash> plans;
  const Key key{{n4, n8, n16, M, K, sm_count()}};
  auto it = plans.find(key);
  if (it == plans.end()) {
    if (plans.size() >= 4096) plans.clear();
    it = plans.emplace(key, make_plan(n4, n8, n16, M, K)).first;
  }
  return it->second;
}

int encode_u8_2d(CUtensorMap *map, const void *base, int cols, int rows) {
  return encode_2d(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, base, cols, rows, 128, 128);
}

}  // namespace

// 16-byte row pitches for TMA, whole 4-byte groups of block scales
bool gemm_stream_takes(int K) { return K % 64 == 0; }

size_t gemm_stream_workspace(int M, int K) {
  (void)K;
  const int mt = (M + kMaxTokens - 1) / kMaxTokens, nt = ((M + mt - 1) / mt + 15) / 16 * 16;
  return 2ull * std::min(sm_count(), kMaxCtas) * nt * 128 * sizeof(float);
}

int launch_gemm_stream(const GemmArgs &g, void *workspace, size_t workspace_bytes, bool pdl, cudaStream_t stream) {
  const StreamPlan &p = stream_plan(g.n4, g.n8, g.n16, g.M, g.K);
  RDQ_REQUIRE(workspace && workspace_bytes >= 2ull * p.sc.G * p.sc.nt * 128 * sizeof(float), RDQ_E_INVALID,
              "GEMM workspace too small");
  int *status = nullptr;
  int rc = gemm_status_ptr(&status);
  if (rc != RDQ_OK) return rc;
  CUtensorMap w4map, w8map, w16map, xmap;
  rc = encode_f16_2d(&xmap, g.x, g.K, g.M, 64, p.sc.nt);
  if (rc != RDQ_OK) return rc;
  w4map = w8map = w16map = xmap;  // maps of absent groups are never used
  if (g.n4 && (rc = encode_u8_2d(&w4map, g.w4, g.K / 2, g.n4)) != RDQ_OK) return rc;
  if (g.n8 && (rc = encode_u8_2d(&w8map, g.w8, g.K, g.n8)) != RDQ_OK) return rc;
  if (g.n16 && (rc = encode_f16_2d(&w16map, g.w16, g.K, g.n16, 64, 128)) != RDQ_OK) return rc;
  StreamArgs a;
  a.s4 = g.s4;
  a.s8 = g.s8;
  a.global4 = g.global4;
  a.perm = g.perm;
  a.bias = g.bias;
  a.y = g.y;
  a.n4 = g.n4;
  a.n8 = g.n8;
  a.n16 = g.n16;
  a.K = g.K;
  a.N = g.n4 + g.n8 + g.n16;
  a.partial = static_cast<float *>(workspace);
  a.arrived = reinterpret_cast<uint32_t *>(g.counters);
  a.nw = p.nw;
  a.early = pdl;
  a.scale_bytes = !aligned16(g.s4) ? 4 : (g.K % 256 == 0 ? 16 : (g.K % 128 == 0 ? 8 : 4));
  a.test_timeout = gemm_test_timeout() == 1;
  a.patience = gemm_test_timeout() == 2 ? 0 : kPatience;
  const StreamSched &sc = p.sc;

  static const void *const fns[4] = {
      reinterpret_cast<const void *>(gemm_stream_kernel<64, false>), reinterpret_cast<const void *>(gemm_stream_kernel<64, true>),
      reinterpret_cast<const void *>(gemm_stream_kernel<128, false>), reinterpret_cast<const void *>(gemm_stream_kernel<128, true>)};
  const int variant = p.wide * 2 + (g.y_bf16 ? 1 : 0);
  const void *fn = fns[variant];
  static std::atomic<bool> attr_done[4][64];
  int dev = 0;
  RDQ_CUDA(cudaGetDevice(&dev));
  std::atomic<bool> *done = dev >= 0 && dev < 64 ? &attr_done[variant][dev] : nullptr;
  if (!done || !done->load()) {
    RDQ_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax));
    if (done) done->store(true);
  }
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(sc.G));
  cfg.blockDim = dim3(p.wide ? kThreads<128> : kThreads<64>);
  cfg.dynamicSmemBytes = p.smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  void *params[7] = {&w4map, &w8map, &w16map, &xmap, &a, const_cast<StreamSched *>(&sc), &status};
  RDQ_CUDA(cudaLaunchKernelExC(&cfg, fn, params));
  return RDQ_OK;
}

}  // namespace rdq
