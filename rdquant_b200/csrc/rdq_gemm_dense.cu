// Prefill GEMM for long prompts: the layer's weights are decoded ONCE per call into an f16 scratch
// (original channel order), then a persistent two-SM tcgen05 GEMM multiplies the activations with it.
//
//   y[M, N] = x[M, K] . W[N, K]^T * scale[N] (+ bias)
//
// Why two passes: decoding inside the GEMM repeats the conversion for every token tile and adds the
// converters' shared-memory writes to a kernel that shared-memory bandwidth bounds already.  The
// scratch costs 2 N K bytes written and read once per call (it mostly stays in the 126 MB L2) and
// leaves a GEMM whose operands both arrive by TMA.
//
// Decoding pass (decode_rows_kernel), HBM-bound: a warp per piece of an output channel, a lane per 8 k --
// loads of 128 / 256 / 512 contiguous bytes and stores of 512 contiguous bytes per warp instruction, up to five
// of them in flight.  (A warp per channel left layers of few long rows with too few warps: see
// rdq_dequant.cu.)  NVFP4 is scaled by its block scale (exact in f16), FP8 stays unscaled: channel
// scale and NVFP4 global scale go into scale[N] and are applied to the FP32 sum.
//
// GEMM (gemm_pair_kernel): a cluster of two CTAs computes 256 channels x up to 256 tokens with
// tcgen05.mma.cta_group::2 (M = 256: 128 channels per CTA).  Channels are the rows of the MMA and
// tokens its columns, so the number of tokens per tile follows the prompt in steps of 32 instead of
// padding it to 256.  Each CTA loads its 128 x 64 weight block and its half of the tokens; the MMA
// reads both halves, so that per k block of 64 an SM's shared memory is written 16 + 16 KB and read
// 16 + 16 KB in the 512 cycles of the MMAs: below the 128 B/clk that bounds a single-CTA tile.
//   warp 0      TMA loads into a ring of six 32 KB stages, completing on the even CTA's barrier
//   warp 1      MMA issue (even CTA); tensor-memory allocation (512 columns = two accumulators)
//   warps 2-5   epilogue: tcgen05.ld (a thread holds one channel: scale and bias are registers),
//               f16 / bf16, transposition through shared memory, 64-byte stores per token.  It
//               works on one accumulator while the MMAs fill the other.
// Tiles are walked in groups of eight token tiles so that concurrent tiles share operands in L2.
// Tiles beyond the last full wave are split along k: every part leaves its FP32 sums in the
// workspace, waits for a while for the others -- they mostly run at the same time, as the last work of
// their CTAs -- and adds and stores its share of the tile's tokens, in the order of the parts
// (await_parts: those that leave, and who does their share).
//
// Reference behaviour replaced: F.linear over a materialised FP16 weight copy
// (rdquant/inference.py:679-687).
#include <cuda.h>

#include "rdq_gemm_common.cuh"
#include "rdq_kernels.cuh"

namespace rdq {

namespace {

// ------------------------------------------------------------------------------- decoding pass
struct DecodeArgs {
  const uint8_t *w4, *s4, *w8, *w16;
  const float *s8;
  float global4;
  const int32_t *inv_perm;
  __half *out;    // [N, K]
  float *scale;   // [N]
  int *counters;  // zeroed for the GEMM
  int n_counters;
  int n4, n8, N, K;
  int segs, len;        // pieces of a row, vectors of eight in a piece
  const uint4 *x_bf16;  // bf16 activations to round to f16 on the way (or null), in vectors of eight
  uint4 *x;
  long long x_vecs;
};

constexpr int kDecodeUnroll = 5;

__global__ void __launch_bounds__(256) decode_rows_kernel(DecodeArgs a) {
  pdl_launch_dependents();  // (launched in stream order: everything before it is complete)
  const int lane = threadIdx.x & 31;
  const long long gid = 1ll * blockIdx.x * blockDim.x + threadIdx.x;
  for (long long i = gid; i < a.n_counters; i += 1ll * gridDim.x * blockDim.x) a.counters[i] = 0;
  if (a.x_bf16) {  // (a launch of its own for these took 3 us)
    const long long stride = 1ll * gridDim.x * blockDim.x;
    for (long long i = gid; i < a.x_vecs; i += 4 * stride) {
      uint4 v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (i + q * stride < a.x_vecs) v[q] = a.x_bf16[i + q * stride];
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (i + q * stride < a.x_vecs)
          a.x[i + q * stride] =
              make_uint4(bf16x2_to_f16x2(v[q].x), bf16x2_to_f16x2(v[q].y), bf16x2_to_f16x2(v[q].z), bf16x2_to_f16x2(v[q].w));
    }
  }
  const int K = a.K;
  const unsigned task = static_cast<unsigned>(gid >> 5), segs = a.segs;
  const int j = static_cast<int>(task / segs), first = static_cast<int>(task - j * segs) * a.len + lane;
  const int nvec = min(K >> 3, first - lane + a.len);  // end of the piece (the launcher requires K % 8 == 0)
  if (j < a.N) {
    const int r = a.inv_perm ? a.inv_perm[j] : j;
    __half *orow = a.out + 1ll * j * K;
    if (r < a.n4) {
      const uint8_t *wrow = a.w4 + 1ll * r * (K >> 1);
      const uint8_t *srow = a.s4 + 1ll * r * (K >> 4);
      if (first == 0) a.scale[j] = a.global4;
      uint32_t q[kDecodeUnroll], s[kDecodeUnroll];
#pragma unroll
      for (int u = 0; u < kDecodeUnroll; ++u) {
        const int v = first + 32 * u;
        if (v < nvec) {
          q[u] = __ldg(reinterpret_cast<const uint32_t *>(wrow) + v);
          s[u] = __ldg(srow + (v >> 1));
        }
      }
#pragma unroll
      for (int u = 0; u < kDecodeUnroll; ++u) {
        const int v = first + 32 * u;
        if (v < nvec) {
          const uint32_t scl = __byte_perm(cvt_e4m3x2(s[u]), 0u, 0x1010u);
          uint4 o;
          cvt_e2m1x8(q[u], o.x, o.y, o.z, o.w);
          o.x = hmul2_u32(o.x, scl);
          o.y = hmul2_u32(o.y, scl);
          o.z = hmul2_u32(o.z, scl);
          o.w = hmul2_u32(o.w, scl);
          reinterpret_cast<uint4 *>(orow)[v] = o;
        }
      }
    } else if (r < a.n4 + a.n8) {
      const int rr = r - a.n4;
      const uint8_t *wrow = a.w8 + 1ll * rr * K;
      if (first == 0) a.scale[j] = a.s8[rr];
      uint2 q[kDecodeUnroll];
#pragma unroll
      for (int u = 0; u < kDecodeUnroll; ++u) {
        const int v = first + 32 * u;
        if (v < nvec) q[u] = __ldg(reinterpret_cast<const uint2 *>(wrow) + v);
      }
#pragma unroll
      for (int u = 0; u < kDecodeUnroll; ++u) {
        const int v = first + 32 * u;
        if (v < nvec) {
          uint4 o;
          cvt_e4m3x4(q[u].x, o.x, o.y);
          cvt_e4m3x4(q[u].y, o.z, o.w);
          reinterpret_cast<uint4 *>(orow)[v] = o;
        }
      }
    } else {
      const uint4 *wrow = reinterpret_cast<const uint4 *>(a.w16 + 2ll * (r - a.n4 - a.n8) * K);
      if (first == 0) a.scale[j] = 1.f;
      uint4 q[kDecodeUnroll];
#pragma unroll
      for (int u = 0; u < kDecodeUnroll; ++u)
        if (first + 32 * u < nvec) q[u] = __ldg(wrow + first + 32 * u);
#pragma unroll
      for (int u = 0; u < kDecodeUnroll; ++u)
        if (first + 32 * u < nvec) reinterpret_cast<uint4 *>(orow)[first + 32 * u] = q[u];
    }
  }
}

// ----------------------------------------------------------------------------------------- GEMM
constexpr int kStages = 6;
constexpr int kBytesW = 128 * 64 * 2;         // weight block of one CTA and k block
constexpr int kStageBytes = 2 * kBytesW;      // + up to 128 tokens
constexpr int kEpiPitch = 64 + 16;            // staging row: 32 channels of one token, skewed
constexpr int kEpiBytes = 4 * 32 * kEpiPitch;
constexpr int kPairSmem = kStages * kStageBytes + kEpiBytes + 1024;
constexpr int kPairThreads = 192;
constexpr int kMaxParts = 4;

struct PairArgs {
  int M, N, kblocks;
  int nt;                // tokens per tile, a multiple of 32 up to 256
  int m_tiles, n_tiles;  // token tiles, 256-channel tiles
  int full;              // tiles [0, full) are done whole, later ones in `parts` parts of k
  int parts;
  const float *scale;
  const __half *bias;
  void *y;
  float *partial;  // [tile - full][part][CTA][token][128 channels]
  uint32_t *counters;  // [tile - full][CTA]: the tile's word (await_parts)
  int patience;
  int test_timeout;
};

struct PairSmem {
  uint64_t full[kStages];
  uint64_t empty[kStages];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint64_t never;
  uint32_t tmem_base;
  int abort_flag;
  int left;  // finish_shared: what await_parts answered
};

struct WorkItem {
  int m, n;          // tile coordinates
  int kb0, kb1;      // k blocks
  int rem, part;     // remainder-tile index (-1: whole tile) and part
};
__device__ __forceinline__ WorkItem work_item(const PairArgs &a, int item) {
  WorkItem w;
  int tile = item;
  w.rem = -1;
  w.part = 0;
  w.kb0 = 0;
  w.kb1 = a.kblocks;
  if (item >= a.full) {
    w.rem = (item - a.full) / a.parts;
    w.part = (item - a.full) - w.rem * a.parts;
    tile = a.full + w.rem;
    w.kb0 = w.part * a.kblocks / a.parts;
    w.kb1 = (w.part + 1) * a.kblocks / a.parts;
    if (a.parts == 1) w.rem = -1;
  }
  constexpr int G = 8;
  const int per_group = G * a.n_tiles;
  const int g = tile / per_group, r = tile - g * per_group;
  const int gsz = min(G, a.m_tiles - g * G);
  w.n = r / gsz;
  w.m = g * G + (r - w.n * gsz);
  return w;
}

// The four epilogue warps: wait for all parts of a split tile, add and store this part's tokens (all of
// them when CTAs have left).  A
// warp takes every fourth token, a lane four channels, with the loads of four tokens in flight.
template <bool BF16>
__device__ __forceinline__ void finish_shared(const PairArgs &a, const WorkItem &w, uint32_t rank, int q, int lane,
                                              volatile int *answer) {
  const int ch = w.n * 256 + static_cast<int>(rank) * 128 + lane * 4;
  float scl[4], bia[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    scl[e] = ch + e < a.N ? a.scale[ch + e] : 0.f;
    bia[e] = ch + e < a.N && a.bias ? __half2float(a.bias[ch + e]) : 0.f;
  }
  uint32_t *const word = a.counters + w.rem * 2 + rank;
  asm volatile("bar.sync 1, 128;" ::: "memory");  // this CTA's warps have all arrived: the last CTA to arrive does not leave
  if (q == 0 && lane == 0) *answer = await_parts(word, a.parts, a.patience);
  asm volatile("bar.sync 1, 128;" ::: "memory");
  const int left = *answer;
  if (left < 0) return;
  const uint32_t passed = q == 0 && lane == 0 ? pass_parts(word) : 0u;
  const int tok0 = w.m * a.nt, ntok = min(a.nt, a.M - tok0);
  const int lo = left ? 0 : ntok * w.part / a.parts, hi = left ? ntok : ntok * (w.part + 1) / a.parts;
  const long long part_stride = 2ll * a.nt * 128;
  const float *src = a.partial + (1ll * w.rem * a.parts * 2 + rank) * a.nt * 128 + lane * 4;
  const bool vec = (a.N & 3) == 0 && ch + 4 <= a.N;
  constexpr int kTok = 4;
#pragma unroll 1
  for (int t0 = lo + q; t0 < hi; t0 += 4 * kTok) {
    float4 p[kMaxParts][kTok];
#pragma unroll
    for (int b = 0; b < kMaxParts; ++b)
#pragma unroll
      for (int e = 0; e < kTok; ++e)
        p[b][e] = b < a.parts && t0 + 4 * e < hi
                      ? __ldcg(reinterpret_cast<const float4 *>(src + b * part_stride + (t0 + 4 * e) * 128))
                      : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int e = 0; e < kTok; ++e) {
      if (t0 + 4 * e >= hi) break;
      float4 v = p[0][e];
#pragma unroll
      for (int b = 1; b < kMaxParts; ++b) {
        v.x += p[b][e].x;
        v.y += p[b][e].y;
        v.z += p[b][e].z;
        v.w += p[b][e].w;
      }
      const uint32_t h0 = pack_y2(fmaf(v.x, scl[0], bia[0]), fmaf(v.y, scl[1], bia[1]), BF16);
      const uint32_t h1 = pack_y2(fmaf(v.z, scl[2], bia[2]), fmaf(v.w, scl[3], bia[3]), BF16);
      uint16_t *dst = static_cast<uint16_t *>(a.y) + 1ll * (tok0 + t0 + 4 * e) * a.N + ch;
      if (vec) {
        *reinterpret_cast<uint2 *>(dst) = make_uint2(h0, h1);
      } else {
        const uint16_t h[4] = {static_cast<uint16_t>(h0), static_cast<uint16_t>(h0 >> 16), static_cast<uint16_t>(h1),
                               static_cast<uint16_t>(h1 >> 16)};
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (ch + u < a.N) dst[u] = h[u];
      }
    }
  }
  if (q == 0 && lane == 0) clear_parts(word, passed, left, a.parts);
}

template <bool BF16>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap,
                 const __grid_constant__ PairArgs a, int *status) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ PairSmem S;
  const uint32_t stage0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t staging = stage0 + kStages * kStageBytes;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int cluster = blockIdx.x >> 1, nclusters = gridDim.x >> 1;
  const int items = a.full + (a.m_tiles * a.n_tiles - a.full) * a.parts;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(smem_u32(&S.full[i]), 1);
      mbar_init(smem_u32(&S.empty[i]), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&S.acc_full[i]), 1);
      mbar_init(smem_u32(&S.acc_empty[i]), 8);  // four epilogue warps of each CTA
    }
    mbar_init(smem_u32(&S.never), 1);
    S.abort_flag = 0;
    mbar_init_fence();
  }
  if (warp == 1) {
    tmem_alloc_pair(smem_u32(&S.tmem_base), 512);
    if (lane == 0) {
      prefetch_tensormap(&xmap);
      prefetch_tensormap(&wmap);
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();  // the partner's barriers exist
  tc_fence_after();
  const uint32_t tmem = S.tmem_base;
  pdl_wait();
  pdl_launch_dependents();

  if (warp == 0) {
    {
      // ------------------------------------------------------------------ TMA loads
      const bool leader = elect_one();
      const uint32_t xbytes = static_cast<uint32_t>(a.nt) * 64;  // this CTA's nt / 2 tokens
      int s = 0, ph = 0;
      bool alive = true;
      for (int item = cluster; item < items && alive; item += nclusters) {
        const WorkItem w = work_item(a, item);
        const int ch0 = w.n * 256 + static_cast<int>(rank) * 128;
        const int tok0 = w.m * a.nt + static_cast<int>(rank) * (a.nt >> 1);
        for (int kb = w.kb0; kb < w.kb1; ++kb) {
          alive = gemm_wait_cluster(&S.empty[s], (ph & 1) ^ 1, &S.abort_flag);
          if (!alive) break;
          if (leader) {
            const uint32_t bar = mapa_u32(smem_u32(&S.full[s]), 0);  // the even CTA's barrier
            if (rank == 0) mbar_arrive_expect_tx(smem_u32(&S.full[s]), 2 * (kBytesW + xbytes));
            const uint32_t dst = stage0 + s * kStageBytes;
            tma_load_2d_pair(dst, &wmap, kb * 64, ch0, bar);
            tma_load_2d_pair(dst + kBytesW, &xmap, kb * 64, tok0, bar);
          }
          if (++s == kStages) { s = 0; ++ph; }
        }
      }
      // On both the normal and the aborted path: let the copies in flight land before the CTA may
      // leave (every stage that was filled is released by the MMAs; bounded).
      for (int i = 0; i < kStages; ++i) {
        if (ph > 0 || i < s) {
          const int last_ph = i < s ? ph : ph - 1;  // round in which stage i was filled last
          for (int t = 0; t < (alive ? 20000 : 20); ++t)
            if (mbar_try(smem_u32(&S.empty[i]), last_ph & 1, 50000u)) break;
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (rank == 0) {
      // ------------------------------------------------------------------ MMA issue
      const bool leader = elect_one();
      const uint32_t idesc = (1u << 4) | (static_cast<uint32_t>(a.nt >> 3) << 17) | (16u << 24);
      int s = 0, ph = 0, it = 0;
      bool alive = true;
      for (int item = cluster; item < items && alive; item += nclusters, ++it) {
        const WorkItem w = work_item(a, item);
        const int buf = it & 1;
        alive = gemm_wait_cluster(&S.acc_empty[buf], ((it >> 1) & 1) ^ 1, &S.abort_flag);
        if (!alive) break;
        tc_fence_after();
        const uint32_t acc = tmem + buf * 256;
        for (int kb = w.kb0; kb < w.kb1; ++kb) {
          alive = gemm_wait_cluster(&S.full[s], ph & 1, &S.abort_flag);
          if (!alive) break;
          tc_fence_after();
          const uint64_t dw = make_desc_sw128(stage0 + s * kStageBytes);
          const uint64_t dx = make_desc_sw128(stage0 + s * kStageBytes + kBytesW);
          if (leader) {
#pragma unroll
            for (int k4 = 0; k4 < 4; ++k4) umma_f16_pair(acc, dw + 2 * k4, dx + 2 * k4, idesc, (kb != w.kb0 || k4 != 0) ? 1u : 0u);
            umma_commit_pair(smem_u32(&S.empty[s]));
          }
          if (++s == kStages) { s = 0; ++ph; }
        }
        if (alive && leader) umma_commit_pair(smem_u32(&S.acc_full[buf]));
      }
    }
    __syncwarp();
  } else {
    // -------------------------------------------------------------------- epilogue
    const int q = warp & 3;  // tensor-memory lanes this warp may read
    const uint32_t stg = staging + q * 32 * kEpiPitch;
    const uint32_t lanes = static_cast<uint32_t>(q * 32) << 16;
    const uint32_t empty_bar[2] = {mapa_u32(smem_u32(&S.acc_empty[0]), 0), mapa_u32(smem_u32(&S.acc_empty[1]), 0)};
    const bool vec = (a.N & 7) == 0;
    WorkItem shared;  // the part of a split tile this CTA did (at most one, its last item)
    shared.rem = -1;
    int it = 0;
    for (int item = cluster; item < items; item += nclusters, ++it) {
      const WorkItem w = work_item(a, item);
      const int buf = it & 1;
      const int ch_base = w.n * 256 + static_cast<int>(rank) * 128 + q * 32;  // first channel of this warp
      const int ch = ch_base + lane;
      float scl = 0.f, bia = 0.f;
      if (ch < a.N) {
        scl = a.scale[ch];
        bia = a.bias ? __half2float(a.bias[ch]) : 0.f;
      }
      if (!gemm_wait_cluster(&S.acc_full[buf], (it >> 1) & 1, &S.abort_flag)) break;
      tc_fence_after();
      const uint32_t acc = tmem + buf * 256 + lanes;
      const int tok0 = w.m * a.nt;
      const int ntok = min(a.nt, a.M - tok0);
      if (w.rem >= 0) {
        // leave this part's sums for finish_shared
        float *mine = a.partial + ((1ll * w.rem * a.parts + w.part) * 2 + rank) * a.nt * 128 + q * 32 + lane;
        for (int c = 0; c < ntok; c += 32) {
          uint32_t v[32];
          tmem_ld32(acc + c, v);
          tmem_wait_ld();
#pragma unroll
          for (int e = 0; e < 32; ++e)
            if (c + e < ntok) mine[(c + e) * 128] = __uint_as_float(v[e]);
        }
        tc_fence_before();
        __threadfence();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive_cluster(empty_bar[buf]);
          arrive_global(a.counters + w.rem * 2 + rank);
        }
        shared = w;
        continue;
      }
      for (int c = 0; c < ntok; c += 32) {
        uint32_t v[32];
        tmem_ld32(acc + c, v);
        tmem_wait_ld();
        if (c + 32 >= ntok) {  // the accumulator is free as soon as its last columns are read
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(empty_bar[buf]);
        }
        // [token][channel] in shared memory, then 64 contiguous bytes per token
#pragma unroll
        for (int e = 0; e < 32; e += 2) {
          const uint32_t h = pack_y2(fmaf(__uint_as_float(v[e]), scl, bia), fmaf(__uint_as_float(v[e + 1]), scl, bia), BF16);
          asm volatile("st.shared.u16 [%0], %1;" ::"r"(stg + e * kEpiPitch + lane * 2),
                       "h"(static_cast<uint16_t>(h)) : "memory");
          asm volatile("st.shared.u16 [%0], %1;" ::"r"(stg + (e + 1) * kEpiPitch + lane * 2),
                       "h"(static_cast<uint16_t>(h >> 16)) : "memory");
        }
        __syncwarp();
        if (vec && ch_base + 32 <= a.N) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int t = i * 8 + (lane >> 2), piece = lane & 3;
            uint4 val;
            asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                         : "=r"(val.x), "=r"(val.y), "=r"(val.z), "=r"(val.w)
                         : "r"(stg + t * kEpiPitch + piece * 16)
                         : "memory");
            if (c + t < ntok)
              *reinterpret_cast<uint4 *>(static_cast<uint16_t *>(a.y) + 1ll * (tok0 + c + t) * a.N + ch_base + piece * 8) = val;
          }
        } else if (ch < a.N) {
          for (int t = 0; t < 32 && c + t < ntok; ++t) {
            uint16_t val;
            asm volatile("ld.shared.u16 %0, [%1];" : "=h"(val) : "r"(stg + t * kEpiPitch + lane * 2) : "memory");
            static_cast<uint16_t *>(a.y)[1ll * (tok0 + c + t) * a.N + ch] = val;
          }
        }
        __syncwarp();
      }
    }
    if (shared.rem >= 0 && !S.abort_flag) finish_shared<BF16>(a, shared, rank, q, lane, &S.left);
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync();  // nothing of the pair is in flight towards either CTA any more
  if (warp == 1) tmem_dealloc_pair(tmem, 512);
  if (threadIdx.x == 0 && S.abort_flag) atomicExch(status, 1);
  if (a.test_timeout && threadIdx.x == 0 && blockIdx.x == 0) {
    if (!mbar_wait(smem_u32(&S.never), 0, 3u)) atomicExch(status, 2);
  }
}

struct PairPlan {
  double cycles;  // estimate
  int nt, m_tiles, n_tiles, clusters, full, parts;
};
// Chosen by estimated cycles among token tiles of equal width (a multiple of 32 up to 256).  A k block
// costs its MMAs or its loads (64 B/clk of L2 bandwidth per SM); whole tiles run in waves over all SM
// pairs; the tiles after the last full wave may be split along k into 2 .. 4 parts, whose FP32 sums
// are written and read once more: about 60 cycles per token of the tile and 4000 for the exchange
// (measured on tiles of 256 tokens: a split that leaves every part 20 k blocks gains nothing).
PairPlan make_pair_plan(int M, int N, int K) {
  PairPlan best{};
  double best_t = 0;
  const int pairs = std::max(1, sm_count() / 2), kblocks = (K + 63) / 64;
  const int lo = (M + 255) / 256, hi = std::max(lo, std::min((M + 95) / 96, lo + 12));
  for (int mt = lo; mt <= hi; ++mt) {
    PairPlan p;
    p.nt = ((M + mt - 1) / mt + 31) / 32 * 32;
    p.m_tiles = (M + p.nt - 1) / p.nt;
    p.n_tiles = (N + 255) / 256;
    const int tiles = p.m_tiles * p.n_tiles;
    const int waves = tiles / pairs, rem = tiles - waves * pairs;
    const double kb = std::max(2.0 * p.nt, 256.0 + p.nt);
    for (int parts = 1; parts <= kMaxParts; ++parts) {
      if (parts > 1 && (rem == 0 || rem * parts > pairs || kblocks / parts < 4)) break;
      const double t = waves * kblocks * kb + (rem ? (kblocks + parts - 1) / parts * kb + (parts > 1 ? 4000.0 + 60.0 * p.nt : 0.0) : 0.0);
      if (best_t == 0 || t < best_t) {
        best_t = t;
        p.cycles = t;
        p.parts = parts;
        p.full = parts > 1 ? waves * pairs : tiles;
        p.clusters = std::min(pairs, p.full + (tiles - p.full) * parts);
        best = p;
      }
    }
  }
  return best;
}
// (a call asks for its plan three times)
const PairPlan &pair_plan(int M, int N, int K) {
  static thread_local PairPlan plan;
  static thread_local int key[4] = {-1, -1, -1, -1};
  const int sms = sm_count();
  if (key[0] != M || key[1] != N || key[2] != K || key[3] != sms) {
    plan = make_pair_plan(M, N, K);
    key[0] = M;
    key[1] = N;
    key[2] = K;
    key[3] = sms;
  }
  return plan;
}

size_t up256(size_t v) { return (v + 255) & ~static_cast<size_t>(255); }

struct DenseLayout {
  size_t weights, scale, counters, partial, total;
};
DenseLayout dense_layout(const PairPlan &p, int N, int K) {
  DenseLayout d;
  const size_t rem = static_cast<size_t>(p.m_tiles) * p.n_tiles - p.full;
  d.weights = 0;
  d.scale = up256(2ull * N * K);
  d.counters = d.scale + up256(4ull * N);
  d.partial = d.counters + up256(rem * 2 * sizeof(int));
  d.total = d.partial + (p.parts > 1 ? rem * p.parts * 2 * p.nt * 128 * sizeof(float) : 0);
  return d;
}

}  // namespace

bool gemm_dense_takes(int K) { return K % 16 == 0; }  // 16-byte row pitch for TMA, whole runs of 8 k

double gemm_dense_estimate(int M, int N, int K) { return 5.1 + 0.545e-6 * N * K + pair_plan(M, N, K).cycles / 1500.0; }

size_t gemm_dense_workspace(int M, int N, int K) { return dense_layout(pair_plan(M, N, K), N, K).total; }

int launch_gemm_dense(const GemmArgs &g, void *workspace, size_t workspace_bytes, cudaStream_t stream) {
  const int N = g.n4 + g.n8 + g.n16;
  const PairPlan p = pair_plan(g.M, N, g.K);
  const DenseLayout lay = dense_layout(p, N, g.K);
  RDQ_REQUIRE(workspace && workspace_bytes >= lay.total, RDQ_E_INVALID, "GEMM workspace too small (%zu bytes needed)", lay.total);
  char *ws = static_cast<char *>(workspace);
  DecodeArgs d;
  d.w4 = g.w4;
  d.s4 = g.s4;
  d.w8 = g.w8;
  d.w16 = reinterpret_cast<const uint8_t *>(g.w16);
  d.s8 = g.s8;
  d.global4 = g.global4;
  d.inv_perm = g.inv_perm;
  d.out = reinterpret_cast<__half *>(ws + lay.weights);
  d.scale = reinterpret_cast<float *>(ws + lay.scale);
  d.counters = reinterpret_cast<int *>(ws + lay.counters);
  d.n_counters = p.parts > 1 ? (p.m_tiles * p.n_tiles - p.full) * 2 : 0;
  d.n4 = g.n4;
  d.n8 = g.n8;
  d.N = N;
  d.K = g.K;
  d.x_bf16 = static_cast<const uint4 *>(g.x_bf16);
  d.x = reinterpret_cast<uint4 *>(const_cast<__half *>(g.x));
  d.x_vecs = 1ll * g.M * g.K / 8;

  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.stream = stream;
  cfg.blockDim = dim3(256);
  const RowPieces cut = row_pieces(g.K, kDecodeUnroll);
  d.segs = cut.pieces;
  d.len = 32 * cut.len;
  cfg.gridDim = dim3(static_cast<unsigned>((1ll * N * d.segs + 7) / 8));
  // In stream order, not overlapping the kernel before: calls that follow one another would chain GEMMs
  // without an end, and with fewer clusters than SM pairs the next call's clusters start beside this
  // one's.  Such a chain of 200 rows x 4560 -> 7017 stopped making progress after some hundred calls.
  RDQ_CUDA(cudaLaunchKernelEx(&cfg, decode_rows_kernel, d));

  int *status = nullptr;
  int rc = gemm_status_ptr(&status);
  if (rc != RDQ_OK) return rc;
  CUtensorMap xmap, wmap;
  rc = encode_f16_2d(&xmap, g.x, g.K, g.M, 64, p.nt / 2);
  if (rc != RDQ_OK) return rc;
  rc = encode_f16_2d(&wmap, d.out, g.K, N, 64, 128);
  if (rc != RDQ_OK) return rc;
  PairArgs a;
  a.M = g.M;
  a.N = N;
  a.kblocks = (g.K + 63) / 64;
  a.nt = p.nt;
  a.m_tiles = p.m_tiles;
  a.n_tiles = p.n_tiles;
  a.full = p.full;
  a.parts = p.parts;
  a.scale = d.scale;
  a.bias = g.bias;
  a.y = g.y;
  a.partial = reinterpret_cast<float *>(ws + lay.partial);
  a.counters = reinterpret_cast<uint32_t *>(d.counters);
  a.test_timeout = gemm_test_timeout() == 1;
  a.patience = gemm_test_timeout() == 2 ? 0 : kPatience;

  const void *fn = g.y_bf16 ? reinterpret_cast<const void *>(gemm_pair_kernel<true>)
                            : reinterpret_cast<const void *>(gemm_pair_kernel<false>);
  static std::atomic<bool> attr_done[2][64];
  int dev = 0;
  RDQ_CUDA(cudaGetDevice(&dev));
  std::atomic<bool> *done = dev >= 0 && dev < 64 ? &attr_done[g.y_bf16 ? 1 : 0][dev] : nullptr;
  if (!done || !done->load()) {
    RDQ_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmem));
    if (done) done->store(true);
  }
  cfg.gridDim = dim3(static_cast<unsigned>(2 * p.clusters));
  cfg.blockDim = dim3(kPairThreads);
  cfg.dynamicSmemBytes = kPairSmem;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  void *params[4] = {&xmap, &wmap, &a, &status};
  RDQ_CUDA(cudaLaunchKernelExC(&cfg, fn, params));
  return RDQ_OK;
}

}  // namespace rdq
