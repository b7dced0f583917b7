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
// Up to 256 tokens, where that is faster (best_plan), tiles are not cut: a tile has as many rows (8 to 128) as make all
// tiles cost the same bytes, and belongs to one cluster of one, two or four CTAs that share its k.  A chunk is 256 k of any format then (one, two or four boxes).  The
// CTAs of a cluster exchange FP32 sums through distributed shared memory (finish_in_cluster): each finishes a share of the tokens.
// They run at the same time by construction, and no word in global memory is involved.
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
#include <cmath>
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
constexpr int kMaxRing = 16;
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
  int R[3];                 // rows per tile
  int cluster;              // (whole tiles) CTAs that share a tile's k: E are tiles of rows then, bnd tiles, numbered token tile by token tile
  int G;                    // CTAs
  int bnd[kMaxCtas + 1];    // first chunk of each CTA
};
struct Segment {
  int fmt, row_tile, m_tile;  // 128-row tile inside the format group, token tile
  int c0, c1;                 // chunks of the tile
  int start;                  // global index of the tile's first chunk
};
// the same where `S` chunks of every tile are this CTA's, numbered through
template <bool MANY>
__device__ __forceinline__ Segment whole_segment_at(const StreamSched &s, int S, int chunk) {
  Segment g;
  const int t = chunk / S;
  int rt = t;
  g.m_tile = 0;
  while (MANY && rt >= s.E[2]) {
    rt -= s.E[2];
    ++g.m_tile;
  }
  g.fmt = rt < s.E[0] ? 0 : (rt < s.E[1] ? 1 : 2);
  g.row_tile = rt - (g.fmt == 0 ? 0 : s.E[g.fmt - 1]);
  g.start = t * S;
  g.c0 = chunk - g.start;
  g.c1 = S;
  return g;
}
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
  int w_pitch, s_pitch;  // bytes of a ring slot: weights, block scales
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
  uint64_t r_full[2][4], r_empty[2][4];  // sums from the cluster's other CTAs: [buffer][epilogue warp]
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
// ... and waits for it: the values pass through, so that no use of one moves ahead of the wait
__device__ __forceinline__ void tmem_wait_ld16(uint32_t (&r)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]),
                 "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
               :
               : "memory");
}
// 16 bytes to shared memory of another CTA of the cluster, counted on a barrier there: no fence on this side
__device__ __forceinline__ void st_async16(uint32_t addr, uint32_t bar, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%2,%3,%4,%5}, [%1];" ::"r"(addr), "r"(bar), "r"(a),
               "r"(b), "r"(c), "r"(d)
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

// row r of a segment's tile of `height` rows
__device__ __forceinline__ Row row_of(const StreamArgs &a, const Segment &g, int height, int r, bool wanted) {
  Row w;
  const int row = g.row_tile * height + r;  // row inside the format group
  const int rows = g.fmt == 0 ? a.n4 : (g.fmt == 1 ? a.n8 : a.n16);
  const int prow = row + (g.fmt == 0 ? 0 : (g.fmt == 1 ? a.n4 : a.n4 + a.n8));
  w.live = r < height && row < rows;
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

// a row's sums of up to 16 tokens from `tok` on
template <bool BF16>
__device__ __forceinline__ void store_tokens(const StreamSched &sc, const StreamArgs &a, const Row &row, const float (&v)[16], int tok,
                                             int count) {
  const int n = row.live ? min(count, sc.M - tok) : 0;
  uint16_t *y = static_cast<uint16_t *>(a.y) + 1ll * tok * a.N + row.col;
#pragma unroll
  for (int e = 0; e < 16; e += 2) {
    const uint32_t h = pack_y2(fmaf(v[e], row.scl, row.bia), fmaf(v[e + 1], row.scl, row.bia), BF16);
    if (e < n) y[0] = static_cast<uint16_t>(h);
    if (e + 1 < n) y[a.N] = static_cast<uint16_t>(h >> 16);
    y += 2 * a.N;
  }
}
// a tile that this CTA has alone
template <bool BF16>
__device__ __forceinline__ void finish_alone(const StreamSched &sc, const StreamArgs &a, const Row &row, uint32_t acc, int tok0, int ntok,
                                             bool dry) {
#pragma unroll 1
  for (int t = 0; t < ntok; t += 16) {
    uint32_t v[16];
    tmem_ld16(acc + t, v);
    tmem_wait_ld16(v);
    float o[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) o[e] = __uint_as_float(v[e]);
    store_tokens<BF16>(sc, a, row, o, tok0 + t, dry ? 0 : 16);
    if (dry) break;
  }
}

// Tiles whose k the CTAs of a cluster share: epilogue warp q sends its 32 rows' sums of the tokens that another CTA
// finishes to that CTA's warp q, waits for those of its own tokens and adds, in the order of the ranks.  `turn` counts the
// tiles in which the warp has rows, for its barriers complete a phase in those alone; two buffers take turns, `more` where
// the buffer will be used again.  Layout of a buffer: [rank][four tokens][128 rows][4].
template <bool BF16>
__device__ __forceinline__ void finish_in_cluster(StreamSmem &S, const StreamSched &sc, const StreamArgs &a, const Row &row, uint32_t acc,
                                                  uint32_t r_ring, int tok0, int rank, int q, int lane, int turn, bool more, bool dry) {
  const int C = sc.cluster, share = sc.nt / C;  // a multiple of four
  const uint32_t part = share * 512;            // bytes of a rank's sums
  const uint32_t buf = r_ring + (turn & 1) * C * part, at = (q * 32 + lane) * 16;
  const int parity = (turn >> 1) & 1;
  uint64_t *full = &S.r_full[turn & 1][q], *empty = &S.r_empty[turn & 1][q];
  if (!dry && turn >= 2 && !gemm_wait_cluster(empty, parity ^ 1, &S.abort_flag)) return;
  uint32_t v[16];
#pragma unroll 1
  for (int p = 1; p < C; ++p) {
    const int to = rank + p < C ? rank + p : rank + p - C;
    const uint32_t dst = mapa_u32(buf + rank * part + at, to), bar = mapa_u32(smem_u32(full), to);
#pragma unroll 1
    for (int t = 0; t < share; t += 16) {
      tmem_ld16(acc + to * share + t, v);
      tmem_wait_ld16(v);
#pragma unroll
      for (int e = 0; e < 16; e += 4)
        if (!dry && t + e < share) st_async16(dst + (t + e) * 512, bar, v[e], v[e + 1], v[e + 2], v[e + 3]);
    }
  }
  if (!dry && lane == 0) mbar_arrive_expect_tx(smem_u32(full), (C - 1) * share * 128);
#pragma unroll 1
  for (int t = 0; t < share; t += 16) {
    const int tok = rank * share + t;
    tmem_ld16(acc + tok, v);
    tmem_wait_ld16(v);
    if (!dry && t == 0 && !gemm_wait_cluster(full, parity, &S.abort_flag)) return;
    float o[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) o[e] = 0.f;
#pragma unroll 1
    for (int p = 0; p < C; ++p) {
#pragma unroll
      for (int e = 0; e < 16; e += 4) {
        uint4 w = make_uint4(v[e], v[e + 1], v[e + 2], v[e + 3]);
        if (p != rank && t + e < share) w = lds16(buf + p * part + (t + e) * 512 + at);
        o[e] += __uint_as_float(w.x);
        o[e + 1] += __uint_as_float(w.y);
        o[e + 2] += __uint_as_float(w.z);
        o[e + 3] += __uint_as_float(w.w);
      }
    }
    // This buffer of theirs is read; ahead of the stores, whose end the release would wait for.
    if (t + 16 >= share && more && !dry) {
      __syncwarp();
      if (lane < C) mbar_arrive_cluster(mapa_u32(smem_u32(empty), lane));
    }
    store_tokens<BF16>(sc, a, row, o, tok0 + tok, dry ? 0 : min(16, share - t));
  }
}

// NT: most tokens per tile (64 or 128).  WHOLE: every tile belongs to one cluster, a chunk has 256 k of any format (make_whole_plan).
// MANY: of several token tiles; without it their arithmetic, which every role does ahead of its first chunk, is not there (decode
// step of four blocks, 32 sequences at 600 tokens: 284 us with a division by their number, 277 with a loop, 269 without).
template <int NT, bool BF16, bool WHOLE, bool MANY = false>
__global__ void __launch_bounds__(kThreadBound<NT>, 1)
gemm_stream_kernel(const __grid_constant__ CUtensorMap w4map, const __grid_constant__ CUtensorMap w8map,
                   const __grid_constant__ CUtensorMap w16map, const __grid_constant__ CUtensorMap xmap,
                   const __grid_constant__ StreamArgs a, const __grid_constant__ StreamSched sc, int *status) {
  constexpr int NS = kStages<NT>, KB = kBlocks<NT>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ StreamSmem S;
  const uint32_t w_ring = (smem_u32(smem_raw) + 1023u) & ~1023u;
  // (tiles of 128 rows: constants)
  const uint32_t w_pitch = WHOLE ? a.w_pitch : kChunkBytes, s_pitch = WHOLE ? a.s_pitch : kScaleBytes;
  const uint32_t x_ring = w_ring + a.nw * w_pitch;
  const uint32_t x_bytes = static_cast<uint32_t>(sc.nt) * 128;  // one 64-k box
  const uint32_t s_ring = x_ring + NS * KB * x_bytes;
  const uint32_t r_ring = x_ring + NS * KB * x_bytes + a.nw * s_pitch + 512;
  // (from lane 0, so that the compiler keeps the roles' branches and loops in uniform registers)
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  // WHOLE: this CTA has the chunks lo .. lo + own - 1 of its cluster's tiles
  const uint32_t rank = WHOLE && sc.cluster > 1 ? cluster_ctarank() : 0u;
  const int worker = WHOLE ? static_cast<int>(blockIdx.x) / sc.cluster : static_cast<int>(blockIdx.x);
  const int lo = WHOLE ? sc.S[0] * static_cast<int>(rank) / sc.cluster : 0;
  const int own = WHOLE ? sc.S[0] * static_cast<int>(rank + 1) / sc.cluster - lo : 0;
  const int begin = sc.bnd[worker] * (WHOLE ? own : 1), end = sc.bnd[worker + 1] * (WHOLE ? own : 1);
  auto seg_at = [&](int chunk, int to) { return WHOLE ? whole_segment_at<MANY>(sc, own, chunk) : segment_at(sc, chunk, to); };
  auto wmap = [&](int fmt) { return fmt == 0 ? &w4map : (fmt == 1 ? &w8map : &w16map); };
  // the boxes of a chunk: one of 128 rows, or as many as 256 k take (those past K are left out)
  auto height_of = [&](int fmt) { return WHOLE ? sc.R[fmt] : 128; };
  auto boxes_of = [&](const Segment &g, int c) { return WHOLE ? min(1 << g.fmt, (sc.nkb - 4 * (lo + c) + (3 >> g.fmt)) >> (2 - g.fmt)) : 1; };
  auto box_x = [&](const Segment &g, int c, int j) { return ((WHOLE ? (lo + c) << g.fmt : c) + j) * (g.fmt == 2 ? 64 : 128); };
  auto load_chunk = [&](const Segment &g, int c, int slot) {
    const uint32_t bar = smem_u32(&S.w_full[slot]);
    const uint32_t box = height_of(g.fmt) * 128;
    const int boxes = boxes_of(g, c);
    mbar_arrive_expect_tx(bar, boxes * box);
    for (int j = 0; j < boxes; ++j)
      tma_load_2d(w_ring + slot * w_pitch + j * box, wmap(g.fmt), box_x(g, c, j), g.row_tile * height_of(g.fmt), bar);
  };
  auto blocks_of = [](int fmt) { return WHOLE ? 4 : 4 >> fmt; };  // k blocks of a chunk
  // The first weight chunks are on their way before anything else is set up; without leave to read weights
  // early, on their way into L2.
  const int ahead = min(a.nw, end - begin), early = a.early ? ahead : 0;
  if (threadIdx.x == 0) {
    for (int i = 0; i < a.nw; ++i) {
      mbar_init(smem_u32(&S.w_full[i]), 1 + 32);  // the TMA thread and the scale warp's lanes
      mbar_init(smem_u32(&S.w_empty[i]), 16 / KB);  // the groups that convert a chunk of four k blocks
    }
    mbar_init_fence();
    Segment g = seg_at(begin, end);
    for (int i = 0; i < ahead; ++i) {
      if (begin + i == g.start + g.c1) g = seg_at(begin + i, end);
      const int c = begin + i - g.start;
      if (a.early) load_chunk(g, c, i);
      else tma_prefetch_2d(wmap(g.fmt), box_x(g, c, 0), g.row_tile * height_of(g.fmt));
      for (int j = 1; WHOLE && !a.early && j < boxes_of(g, c); ++j)
        tma_prefetch_2d(wmap(g.fmt), box_x(g, c, j), g.row_tile * height_of(g.fmt));
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
    if (WHOLE) {
      for (int i = 0; i < 8; ++i) {
        mbar_init(smem_u32(&S.r_full[i >> 2][i & 3]), 1);
        mbar_init(smem_u32(&S.r_empty[i >> 2][i & 3]), sc.cluster);
      }
    }
    mbar_init(smem_u32(&S.never), 1);
    S.abort_flag = 0;
    mbar_init_fence();
  }
  if (warp == 2) tmem_alloc(smem_u32(&S.tmem_base), 512);
  if (warp == 3 && lane == 0) prefetch_tensormap(&xmap);
  tc_fence_before();
  __syncthreads();
  if (WHOLE && sc.cluster > 1) cluster_arrive();  // (waited for ahead of the first word to another CTA)
  tc_fence_after();
  const uint32_t tmem = S.tmem_base;
  const uint32_t tmem_a = tmem + 2 * NT;

  // stages of a range: its NVFP4 chunks (they come first) take several each above 64 tokens
  constexpr int split = 4 / KB;
  const int n4 = WHOLE ? 0 : max(0, min(end, sc.E[0]) - begin);
  const int stages = split * n4 + (end - begin - n4);

  if (warp == 0) {
    // ---------------------------------------------------------------- weight chunks
    const bool leader = elect_one();
    if (!a.early) pdl_wait();
    Cursor w;
    if (early == a.nw) w.ph ^= 1;
    else w.i = early;
    Segment g = seg_at(begin, end);
    for (int i = begin + early; i < end; ++i) {
      if (i >= g.start + g.c1) g = seg_at(i, end);
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
    Segment g = seg_at(begin, end);
    for (int i = begin; i < end; ++i) {
      if (i >= g.start + g.c1) g = seg_at(i, end);
      const int per = blocks_of(g.fmt);  // k blocks of 64 per chunk
      const int kb0 = (lo + i - g.start) * per, blocks = min(per, sc.nkb - kb0);
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
      const Segment g = seg_at(ck, end);
      const int per = blocks_of(g.fmt);
      if (!gemm_wait(&S.d_empty[d.i], d.ph ^ 1, &S.abort_flag)) break;
      tc_fence_after();
      const uint32_t acc = tmem + d.i * NT;
      const int bps = min(per, KB);                                    // k blocks of a stage
      const int blocks = min((lo + g.c1) * per, sc.nkb) - (lo + g.c0) * per;
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
    int rows = 0;  // of this lane
    for (int i = begin; i < end; ++i) {
      if (i == begin || i >= g.start + g.c1) {
        g = seg_at(i, end);
        const int height = height_of(0);
        rows = g.fmt != 0 ? 0 : (height - lane + 31) / 32;
#pragma unroll
        for (int u = 0; u < 4; ++u) src[u] = a.s4 + 1ll * min(g.row_tile * height + u * 32 + lane, a.n4 - 1) * pitch;
      }
      if (!gemm_wait(&S.w_empty[w.i], w.ph ^ 1, &S.abort_flag)) break;
      const int c = lo + i - g.start;
      const uint32_t dst = s_ring + w.i * s_pitch + lane * 16;
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
    if (!WHOLE) S.cut[0][q * 32 + lane] = row_of(a, seg_at(begin, end), 128, q * 32 + lane, true);
    if (!WHOLE) S.cut[1][q * 32 + lane] = row_of(a, seg_at(end - 1, end), 128, q * 32 + lane, true);
    Cursor d;
    bool first = true;
    // Tiles in which this warp has rows, so far and in all.  Tiles get lower from format to format: the last ones of a token
    // tile may have none, and the next token tile starts with high ones again.
    int turn = 0, turns = 0;
    if (WHOLE && sc.cluster > 1) {
      const int with = q * 32 < sc.R[2] ? sc.E[2] : (q * 32 < sc.R[1] ? sc.E[1] : (q * 32 < sc.R[0] ? sc.E[0] : 0));
      auto before = [&](int tile) {
        int n = 0;
        for (; MANY && tile >= sc.E[2]; tile -= sc.E[2]) n += with;
        return n + min(tile, with);
      };
      turns = before(sc.bnd[worker + 1]) - before(sc.bnd[worker]);
      cluster_wait();
    }
    // (whole tiles) The first turn of the loop, while nothing is there to be stored, runs through without a wait, a store or
    // an arrival: it brings the code into the instruction caches, 2000 cycles that would be spent behind the last MMA.
    bool dry = WHOLE;
    for (int ck = begin; ck < end;) {
      const Segment g = seg_at(ck, end);
      const bool whole = WHOLE || (g.c0 == 0 && g.c1 == sc.S[g.fmt]);
      const Row row = row_of(a, g, height_of(g.fmt), q * 32 + lane, whole);
      const int tok0 = g.m_tile * sc.nt;
      const int ntok = min(sc.nt, sc.M - tok0);
      if (!(WHOLE && dry)) {
        if (!gemm_wait(&S.d_full[d.i], d.ph, &S.abort_flag)) break;
        tc_fence_after();
      }
      const uint32_t acc = tmem + d.i * NT + lanes;
      float *part = a.partial + (2ll * blockIdx.x + (first ? 0 : 1)) * sc.nt * 128 + q * 32 + lane;
      uint16_t *yp = static_cast<uint16_t *>(a.y) + 1ll * tok0 * a.N + row.col;
      // sixteen tokens at a time; the stores of one batch overlap the load of the next
      uint32_t v[2][16];
      if (WHOLE) {
        if (q * 32 < sc.R[g.fmt]) {  // (else no rows)
          if (sc.cluster > 1) finish_in_cluster<BF16>(S, sc, a, row, acc, r_ring, tok0, static_cast<int>(rank), q, lane, turn, turn + 2 < turns, dry);
          else finish_alone<BF16>(sc, a, row, acc, tok0, ntok, dry);
          if (!dry) ++turn;
        }
        if (dry) {
          dry = false;
          continue;
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&S.d_empty[d.i]));
        d.next(2);
        ck = g.start + g.c1;
        continue;
      }
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
      if (j == grp || i >= g.start + g.c1) g = seg_at(i, end);
      if (!gemm_wait(&S.empty[grp], ph ^ 1, &S.abort_flag)) break;
      if (!gemm_wait(&S.w_full[slot], w_ph, &S.abort_flag)) break;
      tc_fence_after();
      const uint32_t base = w_ring + slot * w_pitch + rbase;
      auto piece = [&](int p) { return lds16(base + ((p ^ sw) << 4)); };
      uint32_t o[16];
      if (WHOLE && q * 32 >= sc.R[g.fmt]) {
        // no rows: the MMAs read whatever these lanes hold, for sums that nobody reads
      } else if (WHOLE && g.fmt > 0) {
        const uint32_t box = sc.R[g.fmt] * 128;
        const int halves = 2 * min(4, sc.nkb - 4 * (lo + i - g.start));
#pragma unroll
        for (int h = 0; h < 8; ++h) {  // 32 k at a time: of a box of 128 or 64 k
          if (h >= halves) break;
          const uint32_t at = base + (g.fmt == 1 ? h >> 2 : h >> 1) * box;
          auto part = [&](int p) { return lds16(at + ((p ^ sw) << 4)); };
          if (g.fmt == 1) {
            convert_fp8(part(2 * (h & 3)), part(2 * (h & 3) + 1), o);
          } else {
#pragma unroll
            for (int p = 0; p < 4; ++p) {
              const uint4 v = part(4 * (h & 1) + p);
              o[4 * p] = v.x;
              o[4 * p + 1] = v.y;
              o[4 * p + 2] = v.z;
              o[4 * p + 3] = v.w;
            }
          }
          tmem_st16(dst + 16 * h, o);
        }
      } else if (g.fmt == 0) {
        // (k blocks beyond K convert the zero fill of the box; the MMAs do not read them)
        const uint4 s4 = lds16(s_ring + slot * s_pitch + row * 16);
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
  if (WHOLE && sc.cluster > 1 && (warp < 4 || warp >= 8)) cluster_wait();  // (the epilogue's warps have)
  tc_fence_before();
  __syncthreads();
  if (WHOLE && sc.cluster > 1) cluster_arrive_relaxed();  // nobody leaves while another CTA may write to it
  if (warp == 2) tmem_dealloc(tmem, 512);
  // ---- tiles shared with other CTAs: half of 512 threads take the range's first segment, half its last
  if (!WHOLE && !S.abort_flag && begin < end && threadIdx.x < kFinishThreads) {
    const int half = threadIdx.x >> 8;
    Segment g = seg_at(begin, end);
    bool mine = half == 0;
    if (half == 1 && g.start + g.c1 < end) {
      mine = true;
      g = seg_at(end - 1, end);
      g = seg_at(max(g.start, begin), end);
    }
    if (!WHOLE && mine && !(g.c0 == 0 && g.c1 == sc.S[g.fmt]))
      finish_shared<BF16, NT == 64 ? 4 : 2, NT == 64 ? 8 : 16>(a, sc, g, S.cut[half][threadIdx.x & 127], threadIdx.x & 127, (threadIdx.x >> 7) & 1, 1 + half, &S.left[half]);
  }
  if (!WHOLE) __syncthreads();
  if (WHOLE && sc.cluster > 1) cluster_wait();
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
  int whole, w_pitch, s_pitch;
  double us;     // estimated time
  double share;  // (cut tiles) a CTA's cycles
  int parts;     // (cut tiles) CTAs that share a tile, at most
  int each;      // (whole tiles) tiles of a cluster, at most
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
    s.R[f] = 128;
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
  // Fitted to 40 layers at 72 to 512 rows (6 % off on average, 49 % at worst): a CTA's share and the parts that the most
  // divided tile is put together from.
  const double share = static_cast<double>(w) / s.G;
  double parts = 0;
  for (int f = 0; f < 3; ++f)
    if (n[f]) parts = std::max(parts, std::ceil(s.S[f] * u[f] / share));
  p.us = 7.6 + 0.672e-3 * share + 0.22 * parts + 0.32 * M / 128;
  p.share = share;
  p.parts = static_cast<int>(parts);
  p.each = 0;
  p.nw = std::min(p.nw, 8);
  p.smem = 1024 + xb + p.nw * (kChunkBytes + kScaleBytes);
  p.whole = 0;
  s.cluster = 1;
  p.w_pitch = kChunkBytes;
  p.s_pitch = kScaleBytes;
  return p;
}

// clusters of that many CTAs (1, 2, 4) that run at the same time: fewer than the SMs would make where an SM of a group
// is left over; 0 when the device cannot say
int clusters_at_once(int size) {
  const int sms = std::min(sm_count(), kMaxCtas);
  if (size == 1) return sms;
  static std::atomic<int> cached[64][2];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  std::atomic<int> &known = cached[dev][size / 4];
  if (known.load() == 0) {
    const void *fn = reinterpret_cast<const void *>(gemm_stream_kernel<64, false, true>);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(size);
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(sms / size * size));
    cfg.blockDim = dim3(kThreads<64>);
    cfg.dynamicSmemBytes = kSmemMax;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, fn, &cfg) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    known.store(n > 0 ? std::min(n, sms / size) : -1);
  }
  return std::max(0, known.load());
}

// Whole tiles: each belongs to one cluster alone, whose CTAs share its k, so that nothing is put together through global
// memory.  Rows per tile by the bytes of a row, so that all tiles cost the same.
bool make_whole_plan(int n4, int n8, int n16, int M, int K, int cluster, StreamPlan *out) {
  const int workers = clusters_at_once(cluster);
  if (workers == 0 || (K + 255) / 256 < cluster) return false;
  StreamPlan p;
  StreamSched &s = p.sc;
  s.M = M;
  s.mt = (M + 63) / 64;
  s.nt = ((M + s.mt - 1) / s.mt + 15) / 16 * 16;
  s.nkb = (K + 63) / 64;
  s.cluster = cluster;
  const int n[3] = {n4, n8, n16};
  const double bytes[3] = {0.5625, 1.0, 2.0};
  int least = 0;
  for (int f = 0; f < 3; ++f) least += (n[f] + 127) / 128;
  const int most = std::max(1, (least * s.mt + workers - 1) / workers);  // tiles of a cluster
  int tiles = 0;
  for (double t = 4.5;; t += 0.5) {
    tiles = 0;
    for (int f = 0; f < 3; ++f) {
      s.R[f] = std::max(8, std::min(128, static_cast<int>(t / bytes[f] / 8) * 8));
      tiles += (n[f] + s.R[f] - 1) / s.R[f];
    }
    if (tiles * s.mt <= most * workers) break;  // (holds at the latest where all tiles have 128 rows)
  }
  int e = 0;
  double heaviest = 0;
  for (int f = 0; f < 3; ++f) {
    s.S[f] = (s.nkb + 3) / 4;
    e += (n[f] + s.R[f] - 1) / s.R[f];
    s.E[f] = e;
    if (n[f]) heaviest = std::max(heaviest, s.R[f] * bytes[f]);
  }
  const int items = tiles * s.mt;
  s.G = std::min(workers, items);
  for (int b = 0; b <= s.G; ++b) s.bnd[b] = static_cast<int>(1ll * items * b / s.G);
  const int each = (items + s.G - 1) / s.G;
  p.wide = 0;
  p.whole = 1;
  p.each = each;
  p.share = 0;
  p.parts = 0;
  p.w_pitch = std::max({n4 ? s.R[0] : 0, n8 ? 2 * s.R[1] : 0, n16 ? 4 * s.R[2] : 0}) * 128;
  p.s_pitch = s.R[0] * 16;
  const int xb = kStages<64> * kBlocks<64> * s.nt * 128 + (cluster > 1 ? std::min(2, each) * s.nt * 512 : 0);
  // (a warp reads the rows of all its lanes: 512 bytes behind the last slot's block scales)
  p.nw = std::min(kMaxRing, (kSmemMax - 1024 - 512 - xb) / (p.w_pitch + p.s_pitch));
  if (p.nw < (each > 1 ? kStages<64> + 1 : kStages<64>)) return false;
  p.smem = 1024 + 512 + xb + p.nw * (p.w_pitch + p.s_pitch);
  // Fitted to calls one after another on 40 layers (0.4 to 350 MB, K 1024 to 16384, 9 to 64 rows): the faster of the
  // clusters is picked but for 0.5 % on average, 9 % at worst.
  const double steps = each * ((s.S[0] + cluster - 1) / cluster) * (0.181 + 0.0035 * s.nt);
  const double memory = heaviest * K / cluster * each / 43e3 * 0.484;
  p.us = 4.9 + std::max(steps, memory) + 1.35 * std::min(steps, memory) + (cluster > 1 ? 1.2 : 0.0) + (cluster > 2 ? 0.25 : 0.0);
  *out = p;
  return true;
}

// What whole tiles of up to 64 tokens take more than cut ones, in microseconds.  Whole ones cost by their steps of 256 k and
// by the exchange, cut ones by a CTA's share and by the parts of a tile.  Where a row of block scales is no
// multiple of 16 bytes the warp that copies them 8 bytes at a time bounds both, whole tiles by their rows of NVFP4.
// Fitted to the difference of both on 190 layers (1 to 150 MB, K 1024 to 16384, 50 to 90 % NVFP4) at 9 to 64 rows.  Of 1800
// points, layers without FP16, with odd channels and K of 64 times an odd number among them, the choice is 0.13 % behind the faster on
// average, 10 % at worst (4096 -> 5120 at 9 rows); always whole is 0.6 % behind, 23 % at worst.
double whole_minus_cut(const StreamPlan &whole, const StreamPlan &cut, int n4, int K) {
  const StreamSched &s = whole.sc;
  const bool narrow = n4 > 0 && K % 256 != 0;
  const int steps = whole.each * ((s.S[0] + s.cluster - 1) / s.cluster);
  const double exchange = s.cluster == 1 ? 0.0 : (s.cluster == 2 ? (narrow ? 1.2 : 1.5) : 1.5 * whole.each);
  return steps * (narrow ? 0.143 * ((s.R[0] + 31) / 32) : 0.32) + exchange -
         (1.2 + (narrow ? 0.74e-3 : 0.4e-3) * cut.share + 0.09 * cut.parts + 0.02 * s.nt);
}

// Up to 64 tokens: the CTAs that share a cut tile spend 7000 cycles behind the last MMA (partial sums, fence,
// arrival, sums, each a round trip to L2 by code that is run once), a cluster 1700 and a CTA alone 1000.  32 rows, calls
// one after another, us of cut tiles and of whole ones: 2560 -> 6144 10.6, 8.3; 4096 -> 2560 10.6, 7.7; 9728 -> 2560 12.5, 10.6;
// 1024 -> 1024 8.0, 6.0; 8192 -> 8192 15.5, 13.7.  But a tile that no cluster of four has room for, of a long K, takes
// longer than its shares: 13312 -> 4608 15.4, 17.6; 8192 -> 4224 at 9 rows 12.5, 13.7; 12288 -> 4096 at 64 rows 16.0, 18.6.  From 150 MB on
// tiles are cut: the tail is short beside the rest, and they use the MMA's 128 rows (10496 -> 21760, 163 MB, at 9 and 32 rows 32.8,
// 34.3 cut, 32.2, 33.9 at best whole; 8192 -> 57344, 292 MB, at 48 rows 73.6, 76.2).  Narrow copies of block scales are the
// exception that is not made: 7552 -> 55424, 297 MB, at 32 rows 84.9, 68.9.
//
// More tokens come in tiles of 64, each work of its own: the weights are converted for each, where cut tiles convert them for 128
// at a time, so that it pays where a CTA's share is small beside the tail.  The estimates decide; the margin covers theirs
// (12416 -> 896 at 192 rows, 0.89 by them, is 20.8 us whole and 17.1 cut).  Over 40 layers, against
// cut tiles and the GEMM over decoded weights, 20 % less time at 72 to 128 rows and 12 % at 160 to 256 (2560 -> 1024 at 128
// rows 11.2 us, now 7.6; 2560 -> 6144 16.5, 11.4; 4096 -> 2560 at 192 rows 14.6, 11.6).  Beyond, 7 % would be left.
StreamPlan best_plan(int n4, int n8, int n16, int M, int K) {
  const StreamPlan cut = make_plan(n4, n8, n16, M, K);
  if (M > 256 || (n4 * 0.5625 + n8 + 2.0 * n16) * K >= 150e6) return cut;
  StreamPlan best = cut;
  double least = M <= 64 ? 1e30 : 0.88 * cut.us;
  for (int cluster = 4; cluster >= 1; cluster /= 2) {
    StreamPlan p;
    if (!make_whole_plan(n4, n8, n16, M, K, cluster, &p)) continue;
    // (up to 64 tokens a further tile costs a cluster of four a microsecond that the estimate does not have: 8064 -> 9984 at
    // 24 rows, three each, 24.6 us, alone 21.3)
    const double us = p.us + (M <= 64 && cluster == 4 ? p.each - 1 : 0);
    if (us >= least) continue;
    best = p;
    least = us;
  }
  return best.whole && M <= 64 && whole_minus_cut(best, cut, n4, K) > 0 ? cut : best;
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
    it = plans.emplace(key, best_plan(n4, n8, n16, M, K)).first;
  }
  return it->second;
}

int encode_u8_2d(CUtensorMap *map, const void *base, int cols, int rows, int box_rows) {
  return encode_2d(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, base, cols, rows, 128, box_rows);
}

}  // namespace

// 16-byte row pitches for TMA, whole 4-byte groups of block scales
bool gemm_stream_takes(int K) { return K % 64 == 0; }

// Partial sums of cut tiles.  Whole tiles have none; not 0 all the same, by which callers tell a decode kernel.
size_t gemm_stream_workspace(int n4, int n8, int n16, int M, int K) {
  const StreamPlan &p = stream_plan(n4, n8, n16, M, K);
  return p.whole ? 256 : 2ull * p.sc.G * p.sc.nt * 128 * sizeof(float);
}
double gemm_stream_estimate(int n4, int n8, int n16, int M, int K) {
  const StreamPlan &p = stream_plan(n4, n8, n16, M, K);
  return p.whole ? p.us : 0.0;
}
bool gemm_stream_uses_words(int n4, int n8, int n16, int M, int K) { return !stream_plan(n4, n8, n16, M, K).whole; }

int launch_gemm_stream(const GemmArgs &g, void *workspace, size_t workspace_bytes, bool pdl, cudaStream_t stream) {
  const StreamPlan &p = stream_plan(g.n4, g.n8, g.n16, g.M, g.K);
  RDQ_REQUIRE(p.whole || (workspace && g.counters && workspace_bytes >= 2ull * p.sc.G * p.sc.nt * 128 * sizeof(float)), RDQ_E_INVALID,
              "GEMM workspace too small");
  int *status = nullptr;
  int rc = gemm_status_ptr(&status);
  if (rc != RDQ_OK) return rc;
  CUtensorMap w4map, w8map, w16map, xmap;
  rc = encode_f16_2d(&xmap, g.x, g.K, g.M, 64, p.sc.nt);
  if (rc != RDQ_OK) return rc;
  w4map = w8map = w16map = xmap;  // maps of absent groups are never used
  if (g.n4 && (rc = encode_u8_2d(&w4map, g.w4, g.K / 2, g.n4, p.sc.R[0])) != RDQ_OK) return rc;
  if (g.n8 && (rc = encode_u8_2d(&w8map, g.w8, g.K, g.n8, p.sc.R[1])) != RDQ_OK) return rc;
  if (g.n16 && (rc = encode_f16_2d(&w16map, g.w16, g.K, g.n16, 64, p.sc.R[2])) != RDQ_OK) return rc;
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
  a.w_pitch = p.w_pitch;
  a.s_pitch = p.s_pitch;
  a.early = pdl;
  a.scale_bytes = !aligned16(g.s4) ? 4 : (g.K % 256 == 0 ? 16 : (g.K % 128 == 0 ? 8 : 4));
  a.test_timeout = gemm_test_timeout() == 1;
  a.patience = gemm_test_timeout() == 2 ? 0 : kPatience;
  const StreamSched &sc = p.sc;

  static const void *const fns[8] = {
      reinterpret_cast<const void *>(gemm_stream_kernel<64, false, false>), reinterpret_cast<const void *>(gemm_stream_kernel<64, true, false>),
      reinterpret_cast<const void *>(gemm_stream_kernel<128, false, false>), reinterpret_cast<const void *>(gemm_stream_kernel<128, true, false>),
      reinterpret_cast<const void *>(gemm_stream_kernel<64, false, true>), reinterpret_cast<const void *>(gemm_stream_kernel<64, true, true>),
      reinterpret_cast<const void *>(gemm_stream_kernel<64, false, true, true>), reinterpret_cast<const void *>(gemm_stream_kernel<64, true, true, true>)};
  const int variant = (p.whole ? (sc.mt > 1 ? 6 : 4) : p.wide * 2) + (g.y_bf16 ? 1 : 0);
  const void *fn = fns[variant];
  static std::atomic<bool> attr_done[8][64];
  int dev = 0;
  RDQ_CUDA(cudaGetDevice(&dev));
  std::atomic<bool> *done = dev >= 0 && dev < 64 ? &attr_done[variant][dev] : nullptr;
  if (!done || !done->load()) {
    RDQ_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax));
    if (done) done->store(true);
  }
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = static_cast<unsigned>(sc.cluster);
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(sc.G * sc.cluster));
  cfg.blockDim = dim3(p.wide ? kThreads<128> : kThreads<64>);
  cfg.dynamicSmemBytes = p.smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = sc.cluster > 1 ? 2 : 1;
  void *params[7] = {&w4map, &w8map, &w16map, &xmap, &a, const_cast<StreamSched *>(&sc), &status};
  RDQ_CUDA(cudaLaunchKernelExC(&cfg, fn, params));
  return RDQ_OK;
}

}  // namespace rdq
