// Kernel and launchers of rdq_gemv_tiled.cu (included at its end; see the header comment there).
namespace rdq {

namespace {

// Image schedule, identical on every CTA.  Images are numbered in storage order.
//
// Where K has only short chunks (images_per_run) the numbered images are runs of up to `run` stored ones of a tile: one copy,
// one ring slot and one turn of a warp group each, everything else below counts in them.
struct TSched {
  int ck;            // chunk length in NVFP4 elements
  int run, chunks;   // stored images per numbered one, of an NVFP4 tile
  int S4, S8, S16;   // images per tile in each group
  int t4, t8;        // tiles in the NVFP4 / FP8 groups
  int e4, e8, e16;   // end of each group's image range
  int img4, img8;    // image bytes (FP8 and FP16 images have the same size)
  int G;             // CTAs with images
  int bound[kMaxCtas + 1];  // first image of every CTA (computed by the launcher: three 64-bit divisions)

  __device__ __forceinline__ int boundary(int b) const { return bound[b < G ? b : G]; }
  __device__ __forceinline__ int tile_of_image(int s) const {
    if (s < e4) return s / S4;
    if (s < e8) return t4 + (s - e4) / S8;
    return t4 + t8 + (s - e8) / S16;
  }
  // byte offset of image s inside the tiled buffer
  __device__ __forceinline__ long long image_offset(int s) const {
    if (s < e4) return 1ll * s * img4;
    return 1ll * e4 * img4 + 1ll * (s - e4) * img8;
  }
  // the stored images of run s: their number, size and place
  __device__ __forceinline__ int run_at(int s, int &img, long long &offset) const {
    const int fmt = s < e4 ? 0 : (s < e8 ? 1 : 2);
    const int i = s - (fmt == 0 ? 0 : (fmt == 1 ? e4 : e8)), S = fmt == 0 ? S4 : (fmt == 1 ? S8 : S16);
    const int tile = i / S, first = (i - tile * S) * run, all = chunks << fmt;
    img = fmt == 0 ? img4 : img8;
    offset = (1ll * tile * all + first) * img;
    if (fmt > 0) offset += 1ll * chunks * t4 * img4;
    if (fmt > 1) offset += 2ll * chunks * t8 * img8;
    return min(run, all - first);
  }
};

// x is written by the preceding kernel: coherent loads, issued only after the PDL wait
__device__ __forceinline__ uint4 t_ldx16(const __half *p) {
  uint4 v;
  asm volatile("ld.global.L1::evict_last.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint2 t_ldx8(const __half *p) {
  uint2 v;
  asm volatile("ld.global.L1::evict_last.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t t_ldx4(const __half *p) {
  uint32_t v;
  asm volatile("ld.global.L1::evict_last.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ uint4 ldg_nc16(const void *p) {
  uint4 v;
  asm volatile("ld.global.nc.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ uint4 ldg_cg16(const void *p) {
  uint4 v;
  asm volatile("ld.global.cg.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}

constexpr uint32_t kIdle = 0xffffffffu;  // a workspace word that holds no partial sum
__device__ __forceinline__ uint4 ld_relaxed16(const float *p) {
  uint4 v;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}

constexpr int kRunBytes = 15872;  // NVFP4 bytes of a run: three slots fit beside 44 KB of activations and the hand-over slots of 16 rows
constexpr int kRunChunk = 512;   // longest chunk whose images travel in runs
constexpr int kAskAhead = 20 * 1024;  // bytes of weights per warp group that are asked into L2 before they may be read (12 and 40 KB: slower)
constexpr int kStageUnroll = 2;  // pair-loop unrolling of the NVFP4 / FP8 stages

struct TiledArgs {
  const __half *x;  // bf16 rows with xop == 3
  int M;
  const uint8_t *tiled;
  const float *s8;
  float global4;
  const int32_t *perm;
  const __half *bias;
  void *y;
  int y_bf16;
  int n4, n8, n16, K;
  float *workspace;
  int32_t *flags;  // one per CTA, then the status word at index status_idx
  int status_idx;
  int nstages;
  int slot_bytes;
  int fdepth;  // slots per hand-over ring
  int early;         // weights may be read before the kernel before this one has finished
  int opens;         // let the next kernel start only when that kernel has finished
  int beside;        // everything may be: wait for it at the end
  int test_timeout;  // self-test: CTA 0 ends with a wait that runs out
  // Peer mode (column-parallel layers): the outputs go to n_dst destinations -- one slice of a
  // gather buffer on every GPU of the node, this one included, written with plain stores over
  // NVLink -- instead of y; the last epilogue warp of the grid then raises this rank's flag on
  // every GPU.  n_dst == 0: off.
  int n_dst;
  __half *dst[kMaxPeers];
  int32_t *peer_flag[kMaxPeers];  // this rank's flag word on every GPU
  int32_t *peer_state;            // local: [0] epilogue warps done in this launch, [1] launches completed
  // Activation prologue (0: x is used as it is).  1: x_in = x (+ x_aux); the CTA's activation rows
  // are f16(x_in * rsqrt(mean(x_in^2) + eps)) * x_weight, and CTA 0 writes x_in to x_out (the
  // updated residual stream).  2: x is [M, 2 K] and the rows are silu(x[:, :K]) * x[:, K:].
  // 3: x is bf16 and the rows are its f16 rounding.
  int xop;
  const __half *x_aux;
  const __half *x_weight;
  __half *x_out;
  float x_eps;
};


// Activation fragment loads: from the shared-memory copy (XS) or from global memory.
// `base` is a shared-memory byte address (XS) or a generic pointer value.
template <bool XS>
__device__ __forceinline__ uint4 ldx16(uint64_t base, int byte_off) {
  uint4 v;
  if (XS) {
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(static_cast<uint32_t>(base) + byte_off) : "memory");
  } else {
    v = t_ldx16(reinterpret_cast<const __half *>(base + byte_off));
  }
  return v;
}
template <bool XS>
__device__ __forceinline__ uint2 ldx8(uint64_t base, int byte_off) {
  uint2 v;
  if (XS) {
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];"
                 : "=r"(v.x), "=r"(v.y) : "r"(static_cast<uint32_t>(base) + byte_off) : "memory");
  } else {
    v = t_ldx8(reinterpret_cast<const __half *>(base + byte_off));
  }
  return v;
}
template <bool XS>
__device__ __forceinline__ uint32_t ldx4(uint64_t base, int byte_off) {
  uint32_t v;
  if (XS) {
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(static_cast<uint32_t>(base) + byte_off) : "memory");
  } else {
    v = t_ldx4(reinterpret_cast<const __half *>(base + byte_off));
  }
  return v;
}
__device__ __forceinline__ uint32_t lds_u32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}

// multiply-accumulate one NVFP4 piece (16 rows x 32 k): raw words of rows g / g+8, the lane's block
// scales of the two rows (low and high half: the multiplies take either half of a register at no
// cost), the lane's 8 activations
template <int NT>
__device__ __forceinline__ void fp4_piece(float (&acc)[NT][2][4], uint32_t wg, uint32_t wg8, uint32_t scales,
                                          const uint4 (&xv)[NT]) {
  const __half2 sc = *reinterpret_cast<const __half2 *>(&scales);
  const __half2 lo = __low2half2(sc), hi = __high2half2(sc);
  const uint32_t sg = *reinterpret_cast<const uint32_t *>(&lo), sg8 = *reinterpret_cast<const uint32_t *>(&hi);
  uint32_t a0, a1, a2, a3, b0, b1, b2, b3;
  cvt_e2m1x8(wg, a0, a1, a2, a3);
  cvt_e2m1x8(wg8, b0, b1, b2, b3);
  a0 = hmul2_u32(a0, sg); a1 = hmul2_u32(a1, sg); a2 = hmul2_u32(a2, sg); a3 = hmul2_u32(a3, sg);
  b0 = hmul2_u32(b0, sg8); b1 = hmul2_u32(b1, sg8); b2 = hmul2_u32(b2, sg8); b3 = hmul2_u32(b3, sg8);
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    mma_16816(acc[n][0], a0, b0, a1, b1, xv[n].x, xv[n].y);
    mma_16816(acc[n][1], a2, b2, a3, b3, xv[n].z, xv[n].w);
  }
}

// Per-lane shared-memory addresses inside a stage, for the pair of pieces the warp starts with.
// A "pair" is two 16-byte pieces of every row = one ldmatrix.x4.
//
// ---- NVFP4 stage: pairs [lo, hi) of 16 rows x 64 k.  All loads of a pair are issued
// before its first use; addresses advance by constants.
template <int NT, bool XS>
__device__ __forceinline__ void stage_fp4(float (&acc)[NT][2][4], uint32_t lm_addr, uint32_t sc_addr,
                                          uint32_t sc8_addr, const uint64_t (&xb)[NT], int xoff, int npairs,
                                          uint32_t sel) {
#pragma unroll kStageUnroll
  for (int i = 0; i < npairs; ++i) {
    uint32_t w[4];
    ldmatrix_x4(lm_addr, w[0], w[1], w[2], w[3]);
    const uint32_t s_g = lds_u32(sc_addr);    // scale bytes of pieces (p, p+1) for row g
    const uint32_t s_g8 = lds_u32(sc8_addr);  // ... for row g + 8
    uint4 x0[NT], x1[NT];
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      x0[n] = ldx16<XS>(xb[n], xoff);
      x1[n] = ldx16<XS>(xb[n], xoff + 64);
    }
    uint32_t sc0, sc1;  // (row g, row g + 8) of pieces p and p + 1
    cvt_e4m3x4(__byte_perm(s_g, s_g8, sel), sc0, sc1);
    fp4_piece<NT>(acc, w[0], w[1], sc0, x0);
    fp4_piece<NT>(acc, w[2], w[3], sc1, x1);
    lm_addr += 32;
    sc_addr += 4;
    sc8_addr += 4;
    xoff += 128;
  }
}

// ---- FP8 stage: pairs of 16 rows x 32 k
template <int NT, bool XS>
__device__ __forceinline__ void stage_fp8(float (&acc)[NT][2][4], uint32_t lm_addr, const uint64_t (&xb)[NT],
                                          int xoff, int npairs) {
#pragma unroll kStageUnroll
  for (int i = 0; i < npairs; ++i) {
    uint32_t w[4];
    ldmatrix_x4(lm_addr, w[0], w[1], w[2], w[3]);
    uint2 x0[NT], x1[NT];
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      x0[n] = ldx8<XS>(xb[n], xoff);
      x1[n] = ldx8<XS>(xb[n], xoff + 32);
    }
    uint32_t a0, a4, a2, a6, c0, c4, c2, c6;
    cvt_e4m3x4(w[0], a0, a4);
    cvt_e4m3x4(w[1], a2, a6);
    cvt_e4m3x4(w[2], c0, c4);
    cvt_e4m3x4(w[3], c2, c6);
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      mma_16816(acc[n][0], a0, a2, a4, a6, x0[n].x, x0[n].y);
      mma_16816(acc[n][1], c0, c2, c4, c6, x1[n].x, x1[n].y);
    }
    lm_addr += 32;
    xoff += 64;
  }
}

// ---- FP16 stage: pairs of 16 rows x 16 k (32 B per row = two 16-byte pieces = one MMA)
template <int NT, bool XS>
__device__ __forceinline__ void stage_fp16(float (&acc)[NT][2][4], uint32_t lm_addr, const uint64_t (&xb)[NT],
                                           int xoff, int npairs) {
  auto one = [&](int c) {
    uint32_t w[4];
    ldmatrix_x4(lm_addr, w[0], w[1], w[2], w[3]);
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      const uint32_t x0 = ldx4<XS>(xb[n], xoff);
      const uint32_t x1 = ldx4<XS>(xb[n], xoff + 16);
      mma_16816(acc[n][c], w[0], w[1], w[2], w[3], x0, x1);
    }
    lm_addr += 32;
    xoff += 32;
  };
  int i = 0;
#pragma unroll 1
  for (; i + 1 < npairs; i += 2) {
    one(0);
    one(1);
  }
  if (i < npairs) one(0);
}

// first image, image count and format of tile gtile
__device__ __forceinline__ void tile_geom(const TSched &sc, int gtile, int &first_img, int &S, int &fmt) {
  if (gtile < sc.t4) {
    fmt = 0; S = sc.S4; first_img = gtile * sc.S4;
  } else if (gtile < sc.t4 + sc.t8) {
    fmt = 1; S = sc.S8; first_img = sc.e4 + (gtile - sc.t4) * sc.S8;
  } else {
    fmt = 2; S = sc.S16; first_img = sc.e8 + (gtile - sc.t4 - sc.t8) * sc.S16;
  }
}

// Split of an activation prologue: a row is cut into `cpr` chunks (a divisor of the twelve warps) of
// `per` 16-byte vectors; a warp takes chunk warp % cpr of the rows warp / cpr, + 12 / cpr, ...  Chunks
// of up to four vectors per lane, and no more rows at a time than there are.
__host__ __device__ inline void prologue_split(int M, int nvec, int &cpr, int &per) {
  cpr = 1;
  per = nvec;
  while (cpr < kMmaWarps && (per > 128 || kMmaWarps / cpr > M)) {
    cpr = cpr == 4 ? 6 : (cpr == 6 ? 12 : cpr + 1);
    per = (nvec + cpr - 1) / cpr;
  }
}
// Up to six rows of 2048 to 3072: a warp takes a twelfth of every row, a vector per lane.  Decode step of four blocks, before and now,
// us: 2560 wide, 3 rows 205.3, 199.0; 4 rows 211.2, 202.1; 6 rows 236.4, 228.2; 3072 wide, 6 rows 272.4, 263.7.  But 8 rows of 2560
// 242.7, 242.9, and 6 rows of 2048 196.8, 200.5.
inline bool norm_by_columns(int M, int K) { return M > 1 && M <= 6 && K > 2048 && (K >> 3) <= kMmaWarps * 32; }
// All rows at once with up to two vectors per lane: they stay in registers between the two passes of a
// norm (2560 wide, one row: 2.0 -> 1.5 us).
inline bool norm_in_registers(int M, int K) {
  int cpr, per;
  prologue_split(M, K >> 3, cpr, per);
  return M <= kMmaWarps / cpr && per <= 64;
}

// NT = number of 8-row activation groups (1: M <= 8, 2: M <= 16)
// EXTRA 1: the launch has an activation prologue or peer destinations (compiled apart so that the
// plain launch carries none of that code).  The usual prologues of up to eight rows are compiled apart
// once more, for the code and registers of the others cost them 1 to 2 %: 2 norm whose rows stay in
// registers (norm_in_registers), 3 silu, 4 bf16, 5 norm of several rows (norm_by_columns).
//
// Warp group g takes the g-th third of the CTA's images, in order, through ring slots g, g + 3, ... of
// its own; epilogue warp g finishes the tiles whose first image (in this CTA) lies in that third.  A
// group therefore hands sums over once per tile -- images dealt out in turn would end every stage of a
// two-image tile with a hand-over, which measured a third of the MMA warps' time -- and everybody
// derives his images from the range alone, without a list.
//
// RUNS: a numbered image is a run of stored ones (TSched), whose pieces the warps of a group share as if they were one.
template <int NT, bool XS, int EXTRA, bool RUNS = false>
__global__ void __launch_bounds__(kThreads, 2) gemv_tiled_kernel(const __grid_constant__ TiledArgs a,
                                                  const __grid_constant__ TSched sc) {
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ __align__(8) uint64_t bar_full[kMaxStages];
  __shared__ __align__(8) uint64_t bar_empty[kMaxStages];
  __shared__ __align__(8) uint64_t fl_full[kGroups][kFlushRing];   // a group's hand-over ring
  __shared__ __align__(8) uint64_t fl_empty[kGroups][kFlushRing];
  __shared__ __align__(8) uint64_t fl_cross[kGroups];  // its sums of a tile that an earlier group started
  __shared__ __align__(8) uint64_t bar_x;
  __shared__ __align__(8) uint64_t bar_never;  // nothing ever arrives here (time-out self-test)
  __shared__ float xred[EXTRA ? RDQ_MAX_GEMV_M : 1][kMmaWarps];  // activation prologue: per-warp sums of squares

  // the prologue: known at compile time but for EXTRA 1
  const int xop = EXTRA == 0 ? 0 : EXTRA == 2 ? 1 : EXTRA == 3 ? 2 : EXTRA == 4 ? 3 : EXTRA == 5 ? 1 : a.xop;
  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  const int K = a.K, M = a.M;
  const int N = a.n4 + a.n8 + a.n16;
  const int nst = a.nstages;
  // hand-over slots of [4 warps][16 rows][mp] partial sums: fdep per group, then one per later group
  // for the tile it shares with an earlier one
  const int mp = (M + 3) & ~3;
  const int fdep = a.fdepth;    // slots per hand-over ring (1 or 2)
  const int gslot_floats = kWarpsPerGroup * kTileRows * mp;
  float *flush = reinterpret_cast<float *>(smem + nst * a.slot_bytes);
  uint8_t *xsm = reinterpret_cast<uint8_t *>(flush + (kGroups * fdep + kGroups - 1) * gslot_floats);
  const int xpitch = 2 * a.K + 16;  // activation row pitch in shared memory: skewed against bank conflicts

  const int s_begin = sc.boundary(blockIdx.x), s_end = sc.boundary(blockIdx.x + 1);
  const int nimg = s_end - s_begin;
  auto third = [&](int g) { return s_begin + nimg * g / kGroups; };
  int32_t *status = a.flags + a.status_idx;
  const int ck = sc.ck;
  const int pitch = (ck >> 1) + 16;

  // In a chain (RDQ_GEMV_PDL) the next kernel may become resident as early as possible: until this grid
  // completes it only fills its own shared-memory ring with weights.  Otherwise it may once this one has
  // waited (the rule at pdl_wait()).
  const bool first = a.early && !a.opens;
  if (first) pdl_launch_dependents();
  if (static_cast<int>(blockIdx.x) >= sc.G) {
    // The grid has a CTA for every SM: one without images holds its place until the kernel before is
    // done, so that the next launch finds one free place per SM, not two on some.
    if (tid == 0) pdl_wait();
    return;
  }

  const uint32_t smem_base = smem_u32(smem);
  if (warp != kMmaWarps) __syncthreads();  // the barriers are set up (the producer warp's part of this is below)

  if (warp == kMmaWarps) {
    // ==================================================================== producer
    const int most = (nimg + kGroups - 1) / kGroups;  // images of the longest third
    auto copy_in = [&](int img, int slot) {
      uint32_t bytes = static_cast<uint32_t>(img < sc.e4 ? sc.img4 : sc.img8);
      long long from;
      if (RUNS) {
        int one;
        bytes = sc.run_at(img, one, from);
        bytes *= one;
      } else {
        from = sc.image_offset(img);
      }
      const uint32_t full = smem_u32(&bar_full[slot]);
      mbar_arrive_expect_tx(full, bytes);
      bulk_g2s(smem_base + slot * a.slot_bytes, a.tiled + from, bytes, full);
    };
    // The ring is filled with weights first (they do not depend on the preceding kernel);
    // only then wait for that kernel and fetch the activations it produced.
    auto fill = [&]() {
      int slot = 0;
      for (int j = 0; j < most && slot < nst; ++j)
        for (int g = 0; g < kGroups && slot < nst; ++g, ++slot)
          if (third(g) + j < third(g + 1)) copy_in(third(g) + j, slot);
    };
    if (lane == 0) {
      for (int i = 0; i < nst; ++i) {
        mbar_init(smem_u32(&bar_full[i]), 1);
        mbar_init(smem_u32(&bar_empty[i]), kWarpsPerGroup);
      }
      for (int g = 0; g < kGroups; ++g) {
        for (int i = 0; i < kFlushRing; ++i) {
          mbar_init(smem_u32(&fl_full[g][i]), kWarpsPerGroup);
          mbar_init(smem_u32(&fl_empty[g][i]), 1);
        }
        mbar_init(smem_u32(&fl_cross[g]), kWarpsPerGroup);
      }
      mbar_init(smem_u32(&bar_x), 1);
      mbar_init(smem_u32(&bar_never), 1);
      mbar_init_fence();
      if (a.early) fill();
    }
    __syncwarp();
    __syncthreads();
    if (lane != 0) return;
    // This thread executes the grid-dependency wait (without the flag the epilogue warps do as well); the
    // other warps sleep on bar_x, which completes after it (and after the activation copies).
    if (!a.beside) pdl_wait();
    if (!first) pdl_launch_dependents();
    const uint32_t bx = smem_u32(&bar_x);
    if (XS && (!EXTRA || xop == 0)) {
      mbar_arrive_expect_tx(bx, static_cast<uint32_t>(M) * 2u * K);
      for (int m = 0; m < M; ++m) bulk_g2s(smem_u32(xsm) + m * xpitch, a.x + 1ll * m * K, 2u * K, bx);
    } else {  // the MMA warps fetch (and transform) the activations themselves
      mbar_arrive(bx);
    }
    if (!a.early) fill();
    // Refills.  Image j of a third sits in the (j mod slots)-th slot of its group; at[g], par: the slot
    // that is next for group g and the parity of the phase in which it was last given back.
    int at[kGroups], par = 0;
#pragma unroll
    for (int g = 0; g < kGroups; ++g) at[g] = g;
#pragma unroll 1
    for (int j = nst / kGroups; j < most; ++j) {
#pragma unroll
      for (int g = 0; g < kGroups; ++g) {
        const int img = third(g) + j;
        if (g + kGroups * j < nst || img >= third(g + 1)) continue;  // in the first fill, or none left
        if (!mbar_wait(smem_u32(&bar_empty[at[g]]), (par >> g) & 1)) {
          atomicExch(status, 1);
          return;
        }
        copy_in(img, at[g]);
        at[g] += kGroups;
        if (at[g] >= nst) {
          at[g] = g;
          par ^= 1 << g;
        }
      }
    }
    if (a.beside) pdl_wait();  // launches that wait for this one rely on the one before as well
    return;
  }

  if (warp > kMmaWarps) {
    // =============================================================== epilogue warps
    const int ej = warp - kMmaWarps - 1;
    const int g_begin = third(ej), g_end = third(ej + 1);
    if (!a.early) {
      // Without leave to read weights early they are asked into L2 ahead of the wait, which is right whatever
      // the kernel before writes: the copies behind the wait read them there.  By these warps, for they have
      // nothing else to do now (the producer, image by image, delayed its own wait by 0.5 us).  In the plain
      // variant, where chains with the flag carry the code as well (host-to-host step 39.4 and 39.3 us without
      // and with it), and in that of bf16 rows; the norm and SiLU variants lost 0.5 % to the code alone.
      if (EXTRA == 0 || EXTRA == 4) {
        long long from = 0, to = 0;
        if (RUNS) {
          int one;
          sc.run_at(g_begin, one, from);
          sc.run_at(g_end, one, to);
        } else {
          from = sc.image_offset(g_begin);
          to = sc.image_offset(g_end);
        }
        to = min(to, from + kAskAhead);
        for (long long at = from + lane * 128; at < to; at += 32 * 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(a.tiled + at));
      }
      pdl_wait();
    }
    // the first tile to finish: the one of the group's first image, unless an earlier group has an image of it
    int gt = 0, f = 0, S = 1, fmt = 0;
    bool mine = g_begin < g_end;
    if (mine) {
      gt = sc.tile_of_image(g_begin);
      tile_geom(sc, gt, f, S, fmt);
      if (f < g_begin && g_begin > s_begin) {
        ++gt;
        mine = f + S < g_end;
        if (mine) tile_geom(sc, gt, f, S, fmt);
      }
    }
    // output column, scale and bias of a tile's rows are constants of the layer: those of the next
    // tile are fetched while this one is computed
    const int row = lane & 15;
    int col = 0;
    float scl = 1.f, bia = 0.f;
    auto fetch = [&](int tile) {
      const int prow = tile * kTileRows + row;
      col = a.perm ? a.perm[prow] : prow;
      scl = (tile < sc.t4) ? a.global4 : (tile < sc.t4 + sc.t8 ? a.s8[prow - a.n4] : 1.f);
      bia = a.bias ? __half2float(a.bias[col]) : 0.f;
    };
    if (mine) fetch(gt);
    // a split tile whose first image this CTA holds (only its last tile can be one): the
    // other parts come from the CTAs bx + 1 .. b_last, in that order
    int b_last = blockIdx.x;
    if (nimg > 0) {
      int fl, Sl, fmtl;
      tile_geom(sc, sc.tile_of_image(s_end - 1), fl, Sl, fmtl);
      const int bnd = sc.boundary(static_cast<int>(blockIdx.x) + lane);  // first image of CTA bx + lane
      b_last += __popc(__ballot_sync(0xffffffffu, lane >= 1 && bnd <= fl + Sl - 1 && bnd < sc.e16));
      if (lane == 0 && b_last >= static_cast<int>(blockIdx.x) + 31) atomicExch(status, 7);
    }
    // y, workspace and flags belong to this launch only once the preceding grid is done
    if (!mbar_wait_launch(smem_u32(&bar_x), 0)) {
      if (lane == 0) atomicExch(status, 6);
      return;
    }
    // work item = (row, quad of four activation rows): lane L takes item L, and item L + 32
    // when M > 8
    constexpr int kItems = NT;
    float *ws_row = a.workspace + 1ll * blockIdx.x * 256 + row * 16;
    int fslot = 0, fpar = 0;
#pragma unroll 1
    while (mine) {
      const int ia = max(f, s_begin), ib = min(f + S, s_end);
      const bool starts = ia == f, ends = ib == f + S;
      const int cur_col = col;
      const float cur_scl = scl, cur_bia = bia;
      // the next tile of this third
      const bool more = f + S < g_end;
      if (more) fetch(gt + 1);
      // Sum first and give the ring slot back at once: the barrier arrival is a release,
      // and behind a global store it would wait for that store to be acknowledged.
      float4 v[kItems];
#pragma unroll
      for (int j = 0; j < kItems; ++j) v[j] = make_float4(0.f, 0.f, 0.f, 0.f);
      auto add = [&](const float *ring) {
#pragma unroll
        for (int j = 0; j < kItems; ++j) {
          const int m0 = ((lane >> 4) + 2 * j) * 4;
          if (m0 >= M) continue;
#pragma unroll
          for (int w = 0; w < kWarpsPerGroup; ++w) {
            const float4 q = *reinterpret_cast<const float4 *>(ring + (w * kTileRows + row) * mp + m0);
            v[j].x += q.x; v[j].y += q.y; v[j].z += q.z; v[j].w += q.w;
          }
        }
      };
      bool ok = mbar_wait(smem_u32(&fl_full[ej][fslot]), fpar);
      if (ok) add(flush + (ej * fdep + fslot) * gslot_floats);
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&fl_empty[ej][fslot]));
      if (++fslot == fdep) {
        fslot = 0;
        fpar ^= 1;
      }
      for (int g = ej + 1; g < kGroups; ++g) {  // groups that continue the tile
        if (third(g) >= ib || third(g) == third(g + 1)) continue;
        ok = ok && mbar_wait(smem_u32(&fl_cross[g]), 0);
        if (ok) add(flush + (kGroups * fdep + g - 1) * gslot_floats);
      }
      if (!ok) {
        if (lane == 0) atomicExch(status, 2);
        return;
      }
      const int b_hi = (starts && !ends) ? b_last : static_cast<int>(blockIdx.x);
#pragma unroll
      for (int j = 0; j < kItems; ++j) {
        const int m0 = ((lane >> 4) + 2 * j) * 4;
        if (m0 >= M) continue;
        const int nm = min(4, M - m0);
        if (!starts) {
          // continuation of a tile another CTA started: store the partial sums into this
          // CTA's workspace slot (idle words read 0xffffffff); the owner polls them
          // strong store: performed at L2 at once (a plain store may linger in this SM while
          // other warps of this CTA poll for another CTA's sums)
          if (nm == 4) {
            asm volatile("st.relaxed.gpu.global.v4.f32 [%0], {%1,%2,%3,%4};" ::"l"(ws_row + m0), "f"(v[j].x), "f"(v[j].y), "f"(v[j].z), "f"(v[j].w) : "memory");
          } else {
            asm volatile("st.relaxed.gpu.global.f32 [%0], %1;" ::"l"(ws_row + m0), "f"(v[j].x) : "memory");
            if (nm > 1) asm volatile("st.relaxed.gpu.global.f32 [%0], %1;" ::"l"(ws_row + m0 + 1), "f"(v[j].y) : "memory");
            if (nm > 2) asm volatile("st.relaxed.gpu.global.f32 [%0], %1;" ::"l"(ws_row + m0 + 2), "f"(v[j].z) : "memory");
          }
          continue;
        }
        // The other CTAs' sums, four activation rows to a load and the next CTA's load in flight
        // behind the present one: each is a round trip to L2, and for M = 8 one row after the other
        // they took 4 us of a 10 us launch.
        const float *pw = a.workspace + 256ll * (blockIdx.x + 1) + row * 16 + m0;
        uint4 nxt = make_uint4(0u, 0u, 0u, 0u);
        if (static_cast<int>(blockIdx.x) < b_hi) nxt = ld_relaxed16(pw);
#pragma unroll 1
        for (int b = blockIdx.x + 1; b <= b_hi; ++b, pw += 256) {
          uint4 w = nxt;
          if (b < b_hi) nxt = ld_relaxed16(pw + 256);
          int spin = 0;
          while (w.x == kIdle || (nm > 1 && w.y == kIdle) || (nm > 2 && w.z == kIdle) || (nm > 3 && w.w == kIdle)) {
            if (++spin > 2000000) {
              ok = false;
              break;
            }
            __nanosleep(100);
            w = ld_relaxed16(pw);
          }
          v[j].x += __uint_as_float(w.x);
          v[j].y += __uint_as_float(w.y);
          v[j].z += __uint_as_float(w.z);
          v[j].w += __uint_as_float(w.w);
          *reinterpret_cast<uint4 *>(const_cast<float *>(pw)) = make_uint4(kIdle, kIdle, kIdle, kIdle);  // slot idle again
        }
        const float o[4] = {fmaf(v[j].x, cur_scl, cur_bia), fmaf(v[j].y, cur_scl, cur_bia), fmaf(v[j].z, cur_scl, cur_bia),
                            fmaf(v[j].w, cur_scl, cur_bia)};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (i >= nm) break;
          const long long at = 1ll * (m0 + i) * N + cur_col;
          if (EXTRA != 1 && EXTRA != 4) {
            static_cast<__half *>(a.y)[at] = __float2half_rn(o[i]);
          } else if (EXTRA == 4 || a.n_dst == 0) {
            store_y(a.y, at, o[i], a.y_bf16);
          } else {
            // the 16 rows of a tile are consecutive columns of the slice: the stores of the lanes
            // of one activation row fall into one 32-byte sector per destination
            for (int d = 0; d < a.n_dst; ++d) a.dst[d][at] = __float2half_rn(o[i]);
          }
        }
      }
      if (__any_sync(0xffffffffu, !ok)) {
        if (lane == 0) atomicExch(status, 3);
        return;
      }
      if (!more) break;
      ++gt;
      tile_geom(sc, gt, f, S, fmt);
    }
    if (EXTRA == 1 && a.n_dst > 0) {
      // This warp's stores to the other GPUs are complete system-wide before it counts itself
      // done; the warp that completes the count publishes the launch number in this rank's flag
      // word on every GPU (release: fence, then the flag stores).
      __threadfence_system();
      __syncwarp();
      if (lane == 0) {
        const int expected = sc.G * kEpiWarps;
        if (atomicAdd(a.peer_state, 1) == expected - 1) {
          __threadfence_system();
          const int launch = a.peer_state[1] + 1;
          a.peer_state[1] = launch;
          a.peer_state[0] = 0;
          for (int d = 0; d < a.n_dst; ++d)
            asm volatile("st.release.sys.global.s32 [%0], %1;" ::"l"(a.peer_flag[d]), "r"(launch) : "memory");
        }
      }
    }
    if (a.test_timeout && blockIdx.x == 0 && ej == 0) {
      // Self-test of the time-out path: all work of this warp is done and nothing of this CTA
      // is in flight; wait (three suspended tries) on a barrier that nothing completes and
      // report the expired wait like any other.
      if (!mbar_wait(smem_u32(&bar_never), 0, 3u) && lane == 0) atomicExch(status, 9);
    }
    return;
  }

  // ==================================================================== MMA warps
  const int g = lane >> 2;  // fragment row / activation row
  const int t = lane & 3;   // fragment k group
  // ldmatrix.x4: lanes 0-7 / 8-15 address rows 0-7 / 8-15 of the first piece of a pair,
  // lanes 16-31 the same rows of the second piece
  const uint32_t lm_lane = ((lane & 7) + ((lane >> 3) & 1) * 8) * pitch + (lane >> 4) * 16;
  const int spitch = scale_pitch(ck);
  const uint32_t sc_lane = kTileRows * pitch + g * spitch;  // block scales of row g
  const uint32_t sel = (t & 2) ? 0x7351u : 0x6240u;          // this lane's 8 codes sit in block t >> 1
  const int npair = ck >> 6;                                 // pairs of 16-byte pieces per row
  const int grp = warp / kWarpsPerGroup, wq = warp % kWarpsPerGroup;

  float acc[NT][2][4];
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[n][c][i] = 0.f;

  const int nvec = K >> 3;
  int cpr = 1, per = nvec;
  if (EXTRA == 5) {
    cpr = kMmaWarps;
    per = (nvec + kMmaWarps - 1) / kMmaWarps;
  } else if (EXTRA && XS && xop != 0) {
    prologue_split(M, nvec, cpr, per);
  }
  const int vlo = (warp % cpr) * per, vhi = min(nvec, vlo + per), rows_at_once = kMmaWarps / cpr;
  uint4 nw[2];  // (EXTRA 2, 5)
  if (EXTRA && XS && xop == 1 && a.early) {
    // the norm's weights are constants: into registers, or L1, while the kernel before this one still runs
    for (int i = vlo + lane, q = 0; i < vhi; i += 32, ++q) {
      const uint4 v = ldg_nc16(a.x_weight + 8 * i);
      if (EXTRA == 5 || (EXTRA == 2 && q == 0)) nw[0] = v;
      else if (EXTRA == 2) nw[1] = v;
      else asm volatile("" ::"r"(v.x));
    }
  }

  // x is produced by the preceding kernel: do not touch it before the producer thread has
  // seen that kernel complete (and, with XS, has copied the rows into shared memory).
  if (!mbar_wait_launch(smem_u32(&bar_x), 0)) {
    if (lane == 0) atomicExch(status, 6);
    return;
  }
  if (EXTRA && XS && xop != 0) {
    // ---- activation prologue: the twelve MMA warps build the CTA's activation rows in shared
    // memory from what the preceding kernels left in global memory (every CTA does the same work:
    // a few KB out of L2).  A row is cut into `cpr` chunks, one warp per chunk, and a lane has
    // four vectors (eight with x_aux) in flight: the cost is a few L2 round trips.
    if (EXTRA == 2) {
      const int m = warp / cpr;
      const __half *xr = a.x + 1ll * m * K;
      uint4 v[2], d[2];
      float ss = 0.f;
      if (m < M) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int i = vlo + lane + 32 * q;
          if (i >= vhi) break;
          v[q] = ldg_cg16(xr + 8 * i);
          if (a.x_aux) d[q] = ldg_cg16(a.x_aux + 1ll * m * K + 8 * i);
          if (!a.early) nw[q] = ldg_nc16(a.x_weight + 8 * i);
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int i = vlo + lane + 32 * q;
          if (i >= vhi) break;
          __half2 *hv = reinterpret_cast<__half2 *>(&v[q]);
          const __half2 *dh = reinterpret_cast<const __half2 *>(&d[q]);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (a.x_aux) hv[j] = __hadd2(hv[j], dh[j]);
            const float2 f = __half22float2(hv[j]);
            ss += f.x * f.x + f.y * f.y;
          }
          if (a.x_out && blockIdx.x == 0) *reinterpret_cast<uint4 *>(a.x_out + 1ll * m * K + 8 * i) = v[q];
        }
        ss = warp_sum(ss);
        if (lane == 0) xred[m][warp % cpr] = ss;
      }
      asm volatile("bar.sync 2, %0;" ::"r"(kMmaWarps * 32) : "memory");
      if (m < M) {
        ss = 0.f;
        for (int w = 0; w < cpr; ++w) ss += xred[m][w];
        const float rs = rsqrtf(ss / K + a.x_eps);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int i = vlo + lane + 32 * q;
          if (i >= vhi) break;
          __half2 *hv = reinterpret_cast<__half2 *>(&v[q]);
          const __half2 *wh = reinterpret_cast<const __half2 *>(&nw[q]);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 f = __half22float2(hv[j]);
            hv[j] = __hmul2(__floats2half2_rn(f.x * rs, f.y * rs), wh[j]);
          }
          *reinterpret_cast<uint4 *>(xsm + m * xpitch + 16 * i) = v[q];
        }
      }
    } else if (EXTRA == 5) {
      // Two rows' loads in flight at a time, the weights there before the wait, and little code: what is run once a launch is
      // fetched while the launch waits (all rows unrolled and kept in registers: slower than the general form).
      constexpr int kRows = 2;
      const int i = vlo + lane;
      const bool in = i < vhi;
      if (!a.early && in) nw[0] = ldg_nc16(a.x_weight + 8 * i);
#pragma unroll 1
      for (int m0 = 0; m0 < M; m0 += kRows) {
        uint4 v[kRows], d[kRows];
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
          v[r] = d[r] = make_uint4(0u, 0u, 0u, 0u);
          if (!in || m0 + r >= M) continue;
          v[r] = ldg_cg16(a.x + 1ll * (m0 + r) * K + 8 * i);
          if (a.x_aux) d[r] = ldg_cg16(a.x_aux + 1ll * (m0 + r) * K + 8 * i);
        }
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
          __half2 *hv = reinterpret_cast<__half2 *>(&v[r]);
          const __half2 *dh = reinterpret_cast<const __half2 *>(&d[r]);
          float ss = 0.f;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (a.x_aux) hv[j] = __hadd2(hv[j], dh[j]);
            const float2 f = __half22float2(hv[j]);
            ss += f.x * f.x + f.y * f.y;
          }
          if (in && m0 + r < M) {
            if (a.x_out && blockIdx.x == 0) *reinterpret_cast<uint4 *>(a.x_out + 1ll * (m0 + r) * K + 8 * i) = v[r];
            *reinterpret_cast<uint4 *>(xsm + (m0 + r) * xpitch + 16 * i) = v[r];
          }
          ss = warp_sum(ss);
          if (lane == 0 && m0 + r < M) xred[m0 + r][warp] = ss;
        }
      }
      asm volatile("bar.sync 2, %0;" ::"r"(kMmaWarps * 32) : "memory");
      float rs = 0.f;  // of row `lane`
      if (lane < M) {
        float sum = 0.f;
#pragma unroll
        for (int w = 0; w < kMmaWarps; ++w) sum += xred[lane][w];
        rs = rsqrtf(sum / K + a.x_eps);
      }
#pragma unroll 1
      for (int m = 0; m < M; ++m) {
        const float rm = __shfl_sync(0xffffffffu, rs, m);
        if (!in) continue;
        uint4 v = *reinterpret_cast<uint4 *>(xsm + m * xpitch + 16 * i);
        __half2 *hv = reinterpret_cast<__half2 *>(&v);
        const __half2 *wh = reinterpret_cast<const __half2 *>(&nw[0]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = __half22float2(hv[j]);
          hv[j] = __hmul2(__floats2half2_rn(f.x * rm, f.y * rm), wh[j]);
        }
        *reinterpret_cast<uint4 *>(xsm + m * xpitch + 16 * i) = v;
      }
    } else if (xop == 1) {
      for (int m = warp / cpr; m < M; m += rows_at_once) {
        const __half *xr = a.x + 1ll * m * K;
        const __half *dr = a.x_aux ? a.x_aux + 1ll * m * K : nullptr;
        __half *orow = (a.x_out && blockIdx.x == 0) ? a.x_out + 1ll * m * K : nullptr;
        float ss = 0.f;
        for (int i0 = vlo + lane; i0 < vhi; i0 += 128) {
          uint4 v[4], d[4];
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (i0 + 32 * q < vhi) v[q] = ldg_cg16(xr + 8 * (i0 + 32 * q));
          if (dr) {
#pragma unroll
            for (int q = 0; q < 4; ++q)
              if (i0 + 32 * q < vhi) d[q] = ldg_cg16(dr + 8 * (i0 + 32 * q));
          }
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int i = i0 + 32 * q;
            if (i >= vhi) break;
            __half2 *hv = reinterpret_cast<__half2 *>(&v[q]);
            if (dr) {
              const __half2 *dh = reinterpret_cast<const __half2 *>(&d[q]);
#pragma unroll
              for (int j = 0; j < 4; ++j) hv[j] = __hadd2(hv[j], dh[j]);
            }
            if (orow) *reinterpret_cast<uint4 *>(orow + 8 * i) = v[q];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float2 f = __half22float2(hv[j]);
              ss += f.x * f.x + f.y * f.y;
            }
            *reinterpret_cast<uint4 *>(xsm + m * xpitch + 16 * i) = v[q];
          }
        }
        ss = warp_sum(ss);
        if (lane == 0) xred[m][warp % cpr] = ss;
      }
      asm volatile("bar.sync 2, %0;" ::"r"(kMmaWarps * 32) : "memory");
      for (int m = warp / cpr; m < M; m += rows_at_once) {
        float ss = 0.f;
        for (int w = 0; w < cpr; ++w) ss += xred[m][w];
        const float rs = rsqrtf(ss / K + a.x_eps);
        for (int i0 = vlo + lane; i0 < vhi; i0 += 128) {
          uint4 v[4], wv[4];
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (i0 + 32 * q < vhi) {
              wv[q] = ldg_nc16(a.x_weight + 8 * (i0 + 32 * q));
              v[q] = *reinterpret_cast<uint4 *>(xsm + m * xpitch + 16 * (i0 + 32 * q));
            }
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int i = i0 + 32 * q;
            if (i >= vhi) break;
            __half2 *hv = reinterpret_cast<__half2 *>(&v[q]);
            const __half2 *wh = reinterpret_cast<const __half2 *>(&wv[q]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float2 f = __half22float2(hv[j]);
              hv[j] = __hmul2(__floats2half2_rn(f.x * rs, f.y * rs), wh[j]);
            }
            *reinterpret_cast<uint4 *>(xsm + m * xpitch + 16 * i) = v[q];
          }
        }
      }
    } else if (xop == 3) {
      for (int m = warp / cpr; m < M; m += rows_at_once) {
        const __half *xr = a.x + 1ll * m * K;
        for (int i0 = vlo + lane; i0 < vhi; i0 += 128) {
          uint4 v[4];
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (i0 + 32 * q < vhi) v[q] = ldg_cg16(xr + 8 * (i0 + 32 * q));
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int i = i0 + 32 * q;
            if (i >= vhi) break;
            *reinterpret_cast<uint4 *>(xsm + m * xpitch + 16 * i) =
                make_uint4(bf16x2_to_f16x2(v[q].x), bf16x2_to_f16x2(v[q].y), bf16x2_to_f16x2(v[q].z), bf16x2_to_f16x2(v[q].w));
          }
        }
      }
    } else {
      for (int m = warp / cpr; m < M; m += rows_at_once) {
        const __half *gr = a.x + 2ll * m * K;
        for (int i0 = vlo + lane; i0 < vhi; i0 += 128) {
          uint4 gv[4], uv[4];
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (i0 + 32 * q < vhi) {
              gv[q] = ldg_cg16(gr + 8 * (i0 + 32 * q));
              uv[q] = ldg_cg16(gr + K + 8 * (i0 + 32 * q));
            }
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int i = i0 + 32 * q;
            if (i >= vhi) break;
            const __half2 *gh = reinterpret_cast<const __half2 *>(&gv[q]);
            const __half2 *uh = reinterpret_cast<const __half2 *>(&uv[q]);
            uint4 o;
            __half2 *oh = reinterpret_cast<__half2 *>(&o);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float2 g2 = __half22float2(gh[j]);
              oh[j] = __hmul2(__floats2half2_rn(silu(g2.x), silu(g2.y)), uh[j]);
            }
            *reinterpret_cast<uint4 *>(xsm + m * xpitch + 16 * i) = o;
          }
        }
      }
    }
    asm volatile("bar.sync 2, %0;" ::"r"(kMmaWarps * 32) : "memory");
  }
  // Lanes of activation rows >= M read row 0 instead: their output columns are never stored.
  uint64_t xb[NT];
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    const int m = n * 8 + g;
    xb[n] = XS ? static_cast<uint64_t>(smem_u32(xsm) + (m < M ? m : 0) * xpitch)
               : reinterpret_cast<uint64_t>(a.x + 1ll * (m < M ? m : 0) * K);
  }

  const int g_begin = third(grp), g_end = third(grp + 1);
  if (g_begin == g_end) return;
  int gt = sc.tile_of_image(g_begin), f, S, fmt;
  tile_geom(sc, gt, f, S, fmt);
  int c = g_begin - f;  // image of its tile
  // sums of a tile that an earlier group started go to that group's epilogue warp
  bool cross = f < g_begin && g_begin > s_begin;
  float *fl_own = flush + grp * fdep * gslot_floats + wq * kTileRows * mp;
  int slot = grp, par = 0;        // ring slot and parity of its phase
  int fslot = 0, fpar = 1;        // hand-over slot and parity of the phase in which it was given back
  int turn = wq;
#pragma unroll 1
  for (int left = g_end - g_begin; left > 0; --left) {
    if (!mbar_wait(smem_u32(&bar_full[slot]), par)) {
      if (lane == 0) atomicExch(status, 4);
      return;
    }
    const uint32_t sbase = smem_base + slot * a.slot_bytes;
    // inside a group the warps take turns on the pair ranges, so uneven splits average out
    const int lw = turn++ & (kWarpsPerGroup - 1);
    const int lo = lw * npair / kWarpsPerGroup, hi = (lw + 1) * npair / kWarpsPerGroup;
    if (RUNS) {
      const int first = c * sc.run, pairs = min(sc.run, (sc.chunks << fmt) - first) * npair;
      const int end = (lw + 1) * pairs / kWarpsPerGroup, img = fmt == 0 ? sc.img4 : sc.img8;
      int p = lw * pairs / kWarpsPerGroup, i = p / npair, q = p - i * npair;
#pragma unroll 1
      while (p < end) {
        const int n = min(npair - q, end - p);
        const uint32_t ibase = sbase + i * img;
        if (fmt == 0) {
          stage_fp4<NT, XS>(acc, ibase + lm_lane + q * 32, ibase + sc_lane + q * 4, ibase + sc_lane + 8 * spitch + q * 4, xb,
                            2 * ((first + i) * ck + q * 64 + t * 8), n, sel);
        } else if (fmt == 1) {
          stage_fp8<NT, XS>(acc, ibase + lm_lane + q * 32, xb, 2 * ((first + i) * (ck >> 1) + q * 32 + t * 4), n);
        } else {
          stage_fp16<NT, XS>(acc, ibase + lm_lane + q * 32, xb, 2 * ((first + i) * (ck >> 2) + q * 16 + t * 2), n);
        }
        p += n;
        ++i;
        q = 0;
      }
    } else if (fmt == 0) {
      stage_fp4<NT, XS>(acc, sbase + lm_lane + lo * 32, sbase + sc_lane + lo * 4, sbase + sc_lane + 8 * spitch + lo * 4,
                        xb, 2 * (c * ck + lo * 64 + t * 8), hi - lo, sel);
    } else if (fmt == 1) {
      stage_fp8<NT, XS>(acc, sbase + lm_lane + lo * 32, xb, 2 * (c * (ck >> 1) + lo * 32 + t * 4), hi - lo);
    } else {
      stage_fp16<NT, XS>(acc, sbase + lm_lane + lo * 32, xb, 2 * (c * (ck >> 2) + lo * 16 + t * 2), hi - lo);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&bar_empty[slot]));
    slot += kGroups;
    if (slot >= nst) {
      slot = grp;
      par ^= 1;
    }
    if (++c < S && left > 1) continue;

    // ---- the group's last image of this tile: hand the partial sums to the epilogue warp
    float *buf = cross ? flush + (kGroups * fdep + grp - 1) * gslot_floats + wq * kTileRows * mp
                       : fl_own + fslot * gslot_floats;
    // (a fresh barrier passes for the parity of the phase before its first)
    if (!cross && !mbar_wait(smem_u32(&fl_empty[grp][fslot]), fpar)) {
      if (lane == 0) atomicExch(status, 5);
      return;
    }
#pragma unroll
    for (int n = 0; n < NT; ++n) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = g + (i >> 1) * 8;
        const int m = n * 8 + 2 * t + (i & 1);
        if (m < M) buf[r * mp + m] = acc[n][0][i] + acc[n][1][i];
        acc[n][0][i] = 0.f;
        acc[n][1][i] = 0.f;
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(cross ? &fl_cross[grp] : &fl_full[grp][fslot]));
    if (!cross && ++fslot == fdep) {
      fslot = 0;
      fpar ^= 1;
    }
    cross = false;
    if (c == S && left > 1) {
      ++gt;
      tile_geom(sc, gt, f, S, fmt);
      c = 0;
    }
  }
}

}  // namespace


void gemv_tiled_scratch(size_t *workspace_bytes, size_t *flag_bytes) {
  const int G = sm_count();
  *workspace_bytes = static_cast<size_t>(G) * 256 * sizeof(float) + 16;  // one partial tile per CTA, from a multiple of 16 on
  *flag_bytes = (static_cast<size_t>(G) + 2) * sizeof(int32_t);     // status word at index G
}

// Stored images per copy: one, unless the chunks are short (K / 64 with a large prime factor: 64 * 2 * 67 has chunks of 128 and
// images of 1.5 KB, eighteen of which were all that an SM had on its way).  As many as leave a slot to every warp group beside the
// most activations that go to shared memory, all runs of a tile about equal: runs of 10, 8 and 5 KB took 8, 17 and 37 % longer over
// fourteen layers.  Calls one after another, image by image and in runs, us, one row / eight: 2368 -> 8192 38.7 / 38.8, 9.5 / 9.6;
// 4736 -> 2048 12.0 / 11.1, 6.4 / 7.8; 11008 -> 4096 25.1 / 22.4, 11.7 / 15.5; 18944 -> 3584 20.5 / 16.0, 15.0 / 15.0, but with leave
// to read weights early 21.1, 21.5 for one.  From chunks of 704 on (26048 -> 1536) runs cost up to 2.5 %.
inline int images_per_run(int K) {
  const int ck = tiled_chunk_k(K), chunks = K / ck, most = kRunBytes / img_bytes(0, ck);
  if (ck > kRunChunk || most < 2) return 1;
  const int runs = (chunks + most - 1) / most;
  return (chunks + runs - 1) / runs;
}

// Shared-memory plan of one launch: weight ring | flush ring | output metadata | activations (if
// they fit).
struct SmemPlan {
  int fdep, nst, smem;
  bool xs;
};
static SmemPlan smem_plan(int M, int K, bool shared) {
  SmemPlan p;
  const int slot_bytes = (images_per_run(K) * img_bytes(0, tiled_chunk_k(K)) + 127) & ~127;
  // hand-over slots of 4 warps x 16 rows x (M rounded up to 4) partial sums (1 - 4 KB): two per group
  // up to eight activation rows, then one, and one for each later group's part of a shared tile
  p.fdep = M <= 8 ? kFlushRing : 1;
  const int fixed = (kGroups * p.fdep + kGroups - 1) * kWarpsPerGroup * kTileRows * ((M + 3) & ~3) * 4;
  // Where weights may be read early, two CTAs (this layer's and the next one's) share an SM's 228 KB:
  // 1 KB each is reserved, static 1.3 KB.  Where they may not, the next one could do nothing before
  // this one ends, and a launch that comes while this one drains would get two places on the SMs
  // that are empty already: seven projections of a block called one by one, 62.0 -> 53.8 us.
  const int total_budget = (shared ? 228 * 1024 / 2 : 228 * 1024) - 1024 - 1408;
  int xbytes = M * (2 * K + 16);
  p.xs = true;
  // Ring depth: slot s belongs to warp group s % 3, so depths 3k and 3k + 2 split the slots
  // 1:1:1 and (k+1):(k+1):k; 3k + 1 would leave one group with half as many more slots as the
  // others and measured slower than 3k.
  auto depth = [&](int xb) {
    int n = (total_budget - fixed - xb) / slot_bytes;
    if (n > kMaxStages) n = kMaxStages;
    return (n % kGroups == 1 && n > kGroups) ? n - 1 : n;
  };
  // activations go to shared memory while that leaves every warp group a ring slot: reading
  // them through L1 costs more than a shallower ring (measured for M = 3 .. 8)
  if (xbytes > 44 * 1024 || depth(xbytes) < min(kGroups, depth(0))) {
    p.xs = false;
    xbytes = 0;
  }
  p.nst = depth(xbytes);
  if (p.nst < kGroups) p.nst = kGroups;  // 3 x 19 KB always fits beside the fixed part
  p.smem = max(p.nst * slot_bytes + fixed + xbytes, shared ? kSlotSmem : kAloneSmem);
  return p;
}
bool tiled_stages_x(int M, int K) { return M >= 1 && M <= RDQ_MAX_GEMV_M && smem_plan(M, K, true).xs; }

// Schedule and shared-memory plan of a (shape, rows) pair.
struct TiledPlan {
  TSched sc;
  SmemPlan pl;
};
static TiledPlan make_tiled_plan(int n4, int n8, int n16, int K, int M, bool shared) {
  TiledPlan p;
  TSched &sc = p.sc;
  p.pl = smem_plan(M, K, shared);
  const int nst = smem_plan(M, K, true).nst;  // in either case: results do not depend on the flag
  const int ck = tiled_chunk_k(K);
  sc.ck = ck;
  sc.chunks = K / ck;
  sc.run = images_per_run(K);
  sc.S4 = (sc.chunks + sc.run - 1) / sc.run;
  sc.S8 = (sc.chunks * 2 + sc.run - 1) / sc.run;
  sc.S16 = (sc.chunks * 4 + sc.run - 1) / sc.run;
  sc.t4 = n4 / kTileRows;
  sc.t8 = n8 / kTileRows;
  const int t16 = n16 / kTileRows;
  sc.e4 = sc.t4 * sc.S4;
  sc.e8 = sc.e4 + sc.t8 * sc.S8;
  sc.e16 = sc.e8 + t16 * sc.S16;
  sc.img4 = img_bytes(0, ck);
  sc.img8 = img_bytes(1, ck);

  // Images are balanced by what they cost a CTA in time, not by their bytes: an NVFP4 image
  // (conversion + block scaling) takes more instructions than an FP8 or FP16 image of the
  // same size, but images beyond the ring's depth mostly cost the wait for their copy.
  int u4, u8, u16;  // scheduling cost of one NVFP4 / FP8 / FP16 image
  {
    // Time model of a CTA that streams n images of one format (cycles, three warp groups):
    // the first nst images are in the ring when the kernel may start and cost their compute
    // time c; each later one costs (landing time + c) / slots per group.  Find the common
    // finishing time T at which the three formats' images fill exactly the grid, and weigh
    // an image by 1 / n(T).
    // Constants measured on B200 with in-kernel clocks (compute) and fitted on the benchmark
    // block (landing time: 2500 .. 7000 give the same step time within 2 %, 1200 is 8 % slower).
    const double kappa[3] = {0.123, 0.0715, 0.038};  // compute cycles per image byte and group
    const double land = 4500.0;                      // cycles from copy issue to landing under load
    const double img[3] = {double(sc.img4) * sc.run, double(sc.img8) * sc.run, double(sc.img8) * sc.run};
    const double cnt[3] = {double(sc.e4), double(sc.e8 - sc.e4), double(sc.e16 - sc.e8)};
    const double spg = double(nst) / kGroups;
    auto n_of = [&](int f, double T) {
      const double c = kappa[f] * img[f], p = (land + c) / spg;
      const double t_ring = nst * c / kGroups;
      return T <= t_ring ? T * kGroups / c : nst + (T - t_ring) * kGroups / p;
    };
    double lo = 1.0, hi = 1e9;
    for (int it = 0; it < 60; ++it) {
      const double T = 0.5 * (lo + hi);
      double ctas = 0;
      for (int f = 0; f < 3; ++f) ctas += cnt[f] / n_of(f, T);
      if (ctas > sm_count()) lo = T; else hi = T;
    }
    const double n4 = n_of(0, hi), n8 = n_of(1, hi), n16 = n_of(2, hi);
    u4 = 1000;
    u8 = max(1, min(1000, static_cast<int>(1000.0 * n4 / n8 + 0.5)));
    u16 = max(1, min(u8, static_cast<int>(1000.0 * n4 / n16 + 0.5)));
  }
  const long long w4 = 1ll * sc.e4 * u4, w8 = w4 + 1ll * (sc.e8 - sc.e4) * u8, W = w8 + 1ll * (sc.e16 - sc.e8) * u16;
  // every CTA must own at least one image: its share may not be shorter than the
  // heaviest image
  int G = min(sm_count(), kMaxCtas);
  // ... and a tile may spread over at most 31 CTAs (the owner finds them with one ballot)
  long long minshare = u4;  // u4 is the largest cost
  const long long tile_cost[3] = {1ll * sc.S4 * u4, 1ll * sc.S8 * u8, 1ll * sc.S16 * u16};
  for (int f = 0; f < 3; ++f)
    if ((tile_cost[f] + 29) / 30 > minshare) minshare = (tile_cost[f] + 29) / 30;
  const long long maxg = W / minshare;
  if (maxg < G) G = static_cast<int>(maxg);
  if (G < 1) G = 1;
  sc.G = G;
  for (int b = 0; b <= G; ++b) {
    const long long pos = W * b / G;
    sc.bound[b] = b == G ? sc.e16
                  : pos < w4 ? static_cast<int>(pos / u4)
                  : pos < w8 ? sc.e4 + static_cast<int>((pos - w4) / u8)
                             : sc.e8 + static_cast<int>((pos - w8) / u16);
  }
  return p;
}
// The plans this thread has used (a decode step calls the same few layers again and again; the time
// model above costs about as much host time as the launch itself).
static const TiledPlan &tiled_plan(int n4, int n8, int n16, int K, int M, bool shared) {
  struct Key {
    int v[7];
    bool operator==(const Key &o) const { return std::equal(v, v + 7, o.v); }
  };
  struct Hash {
    size_t operator()(const Key &k) const {
      size_t h = 1469598103934665603ull;
      for (int x : k.v) h = (h ^ static_cast<size_t>(x)) * 1099511628211ull;
      return h;
    }
  };
  static thread_local std::unordered_map<Key, TiledPlan, Hash> plans;
  const Key key{{n4, n8, n16, K, M, shared, sm_count()}};
  auto it = plans.find(key);
  if (it == plans.end()) {
    if (plans.size() >= 4096) plans.clear();
    it = plans.emplace(key, make_tiled_plan(n4, n8, n16, K, M, shared)).first;
  }
  return it->second;
}

int launch_gemv_tiled(const GemvTiledArgs &h, bool pdl, cudaStream_t stream) {
  const TiledPlan &plan = tiled_plan(h.n4, h.n8, h.n16, h.K, h.M, pdl);
  const TSched &sc = plan.sc;
  const SmemPlan &pl = plan.pl;
  TiledArgs a;
  a.x = static_cast<const __half *>(h.x); a.y_bf16 = h.y_bf16; a.M = h.M; a.tiled = h.tiled; a.s8 = h.s8; a.global4 = h.global4; a.perm = h.perm;
  a.bias = h.bias; a.y = h.y; a.n4 = h.n4; a.n8 = h.n8; a.n16 = h.n16; a.K = h.K;
  // the kernel's loads take four words at a time; a workspace at any word serves, its size leaves room
  a.workspace = reinterpret_cast<float *>((reinterpret_cast<uintptr_t>(h.workspace) + 15) & ~static_cast<uintptr_t>(15));
  a.flags = h.flags;
  a.early = pdl;
  a.opens = h.opens;
  a.beside = h.beside;
  a.test_timeout = h.test_timeout;
  a.n_dst = h.n_dst;
  for (int d = 0; d < kMaxPeers; ++d) {
    a.dst[d] = d < h.n_dst ? h.dst[d] : nullptr;
    a.peer_flag[d] = d < h.n_dst ? h.peer_flag[d] : nullptr;
  }
  a.peer_state = h.peer_state;
  a.xop = h.x_bf16 ? 3 : h.xop; a.x_aux = h.x_aux; a.x_weight = h.x_weight; a.x_out = h.x_out; a.x_eps = h.x_eps;
  a.status_idx = sm_count();
  a.slot_bytes = (sc.run * img_bytes(0, sc.ck) + 127) & ~127;
  const int nt = h.M <= 8 ? 1 : 2;
  a.fdepth = pl.fdep;
  a.nstages = pl.nst;
  const bool xs = pl.xs;
  RDQ_REQUIRE(a.xop == 0 || xs, RDQ_E_UNSUPPORTED,
              "activation prologue needs the activation rows in shared memory (M=%d, K=%d)", h.M, h.K);
  RDQ_REQUIRE(h.xop == 0 || (h.xop == 1 && h.x_weight) || h.xop == 2, RDQ_E_INVALID, "bad activation prologue");
  const int smem = pl.smem;


  static int smem_set[64][20] = {};
  static std::mutex smem_mutex;
  int dev = 0;
  RDQ_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> smem_lock(smem_mutex);
  const bool extra = a.xop != 0 || h.n_dst > 0 || h.y_bf16;
  const bool in_registers = a.xop == 1 && !h.y_bf16 && norm_in_registers(h.M, h.K);
  const bool runs = sc.run > 1;
  const bool own = extra && h.n_dst == 0 && nt == 1 && xs && !runs;  // a variant of its own
  const bool by_columns = a.xop == 1 && !h.y_bf16 && norm_by_columns(h.M, h.K);
  const int variant = own && in_registers                      ? 8
                      : own && by_columns              ? 11
                      : own && a.xop == 2 && !h.y_bf16 ? 9
                      : own && a.xop == 3              ? 10
                                                       : (runs ? 12 : 0) + (extra ? 4 : 0) + (nt - 1) * 2 + (xs ? 1 : 0);
  static const void *const fns[20] = {
      reinterpret_cast<const void *>(gemv_tiled_kernel<1, false, 0>),
      reinterpret_cast<const void *>(gemv_tiled_kernel<1, true, 0>),
      reinterpret_cast<const void *>(gemv_tiled_kernel<2, false, 0>),
      reinterpret_cast<const void *>(gemv_tiled_kernel<2, true, 0>),
      reinterpret_cast<const void *>(gemv_tiled_kernel<1, false, 1>),
      reinterpret_cast<const void *>(gemv_tiled_kernel<1, true, 1>),
      reinterpret_cast<const void *>(gemv_tiled_kernel<2, false, 1>),
      reinterpret_cast<const void *>(gemv_tiled_kernel<2, true, 1>),
      reinterpret_cast<const void *>(gemv_tiled_kernel<1, true, 2>),
      reinterpret_cast<const void *>(gemv_tiled_kernel<1, true, 3>),
      reinterpret_cast<const void *>(gemv_tiled_kernel<1, true, 4>),
      reinterpret_cast<const void *>(gemv_tiled_kernel<1, true, 5>),
      reinterpret_cast<const void *>(gemv_tiled_kernel<1, false, 0, true>),
      reinterpret_cast<const void *>(gemv_tiled_kernel<1, true, 0, true>),
      reinterpret_cast<const void *>(gemv_tiled_kernel<2, false, 0, true>),
      reinterpret_cast<const void *>(gemv_tiled_kernel<2, true, 0, true>),
      reinterpret_cast<const void *>(gemv_tiled_kernel<1, false, 1, true>),
      reinterpret_cast<const void *>(gemv_tiled_kernel<1, true, 1, true>),
      reinterpret_cast<const void *>(gemv_tiled_kernel<2, false, 1, true>),
      reinterpret_cast<const void *>(gemv_tiled_kernel<2, true, 1, true>)};
  const void *fn = fns[variant];
  if (dev < 64 && smem_set[dev][variant] < smem) {
    RDQ_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    // Always the largest shared-memory carve-out: layers of different footprints follow each
    // other, and an SM cannot change its carve-out while a CTA of the previous layer is resident
    // (the next layer's CTA would wait instead of filling its ring alongside).
    RDQ_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
    smem_set[dev][variant] = smem;
  }

  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(sm_count()));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  void *params[2] = {&a, const_cast<TSched *>(&sc)};
  RDQ_CUDA(cudaLaunchKernelExC(&cfg, fn, params));
  return RDQ_OK;
}


// ---------------------------------------------------------------------------------------
// Entry point for callers that cannot allocate device memory (no counterpart in the
// reference).  Its scratch -- the per-CTA partial-tile slots and the status word the
// tiled GEMV needs -- lives in the array below, which every GPU that loads this library
// holds until the process exits.  Sized for GPUs with up to kNoAllocMaxCtas SMs.
// ---------------------------------------------------------------------------------------
namespace {
constexpr int kNoAllocMaxCtas = 160;
constexpr int kNoAllocWsWords = kNoAllocMaxCtas * 256;  // workspace: one 16 x 16 float slot per CTA
constexpr int kNoAllocCntWords = kNoAllocMaxCtas + 32;                  // flags + status word
static __device__ __align__(256) uint32_t g_noalloc_scratch[kNoAllocWsWords + kNoAllocCntWords];

std::mutex g_noalloc_mutex;
void *g_noalloc_ptr[64] = {};

// Device address of the library array on the current device; the first call per device looks
// it up and puts the array into its idle state on `stream`.
int noalloc_array(void **out, cudaStream_t stream) {
  int dev = 0;
  RDQ_CUDA(cudaGetDevice(&dev));
  RDQ_REQUIRE(dev >= 0 && dev < 64, RDQ_E_UNSUPPORTED, "device index %d is beyond the 64 devices this entry point tracks", dev);
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (!g_noalloc_ptr[dev]) {
    // Set-up, once per device, with that device current.  In host code the array's name is
    // only a stand-in; the address a kernel can use has to come from the runtime.
    void *p = nullptr;
    RDQ_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch));
    // idle partial-sum slots read 0xffffffff; flags and status word start at zero
    RDQ_CUDA(cudaMemsetAsync(p, 0xff, sizeof(uint32_t) * kNoAllocWsWords, stream));
    RDQ_CUDA(cudaMemsetAsync(static_cast<uint32_t *>(p) + kNoAllocWsWords, 0, sizeof(uint32_t) * kNoAllocCntWords, stream));
    g_noalloc_ptr[dev] = p;
  }
  *out = g_noalloc_ptr[dev];
  return RDQ_OK;
}

const char *tiled_status_text(int code) {
  switch (code) {
    case 1: return "producer: a ring slot was never released";
    case 2: return "epilogue: a warp group never handed over its partial sums";
    case 3: return "epilogue: another CTA never published its part of a split tile";
    case 4: return "MMA warps: a weight image never landed in the ring";
    case 5: return "MMA warps: a hand-over slot was never released";
    case 6: return "the activations were never staged (wait on the preceding kernel)";
    case 7: return "a tile is spread over more CTAs than the owner can collect";
    case 8: return "more images per CTA than the stage list holds";
    case 9: return "time-out self-test (RDQ_GEMV_TEST_TIMEOUT)";
    default: return "unknown status";
  }
}
}  // namespace

int gemv_tiled_noalloc(const GemvTiledArgs &in, bool pdl, cudaStream_t stream) {
  RDQ_REQUIRE(sm_count() <= kNoAllocMaxCtas, RDQ_E_UNSUPPORTED,
              "built-in scratch holds %d CTA slots but this GPU has %d SMs; use rdq_gemv_tiled with caller scratch",
              kNoAllocMaxCtas, sm_count());
  void *p = nullptr;
  const int rc = noalloc_array(&p, stream);
  if (rc != RDQ_OK) return rc;
  GemvTiledArgs a = in;
  a.workspace = static_cast<float *>(p);
  a.flags = reinterpret_cast<int32_t *>(static_cast<uint32_t *>(p) + kNoAllocWsWords);
  return launch_gemv_tiled(a, pdl, stream);
}

// Status word of the tiled GEMV after everything queued on `stream` has run: the caller's
// scratch pair, or (both null) the library array of the no-allocation entry point.  With
// `reset`, the status word and flags return to zero and every partial-sum slot to its idle
// pattern, so the next launch starts clean even after a launch that gave up a wait.
int gemv_tiled_status(float *workspace, int32_t *flags, bool reset, cudaStream_t stream) {
  size_t ws_bytes = 0, flag_bytes = 0;
  if (!workspace && !flags) {
    void *p = nullptr;
    const int rc = noalloc_array(&p, stream);
    if (rc != RDQ_OK) return rc;
    workspace = static_cast<float *>(p);
    flags = reinterpret_cast<int32_t *>(static_cast<uint32_t *>(p) + kNoAllocWsWords);
    ws_bytes = sizeof(uint32_t) * kNoAllocWsWords;
    flag_bytes = sizeof(uint32_t) * kNoAllocCntWords;
  } else {
    RDQ_REQUIRE(workspace && flags, RDQ_E_INVALID, "workspace and counters must both be given (or both null)");
    gemv_tiled_scratch(&ws_bytes, &flag_bytes);
  }
  int32_t code = 0;
  RDQ_CUDA(cudaMemcpyAsync(&code, flags + sm_count(), sizeof(code), cudaMemcpyDeviceToHost, stream));
  RDQ_CUDA(cudaStreamSynchronize(stream));
  if (reset) {
    RDQ_CUDA(cudaMemsetAsync(workspace, 0xff, ws_bytes, stream));
    RDQ_CUDA(cudaMemsetAsync(flags, 0, flag_bytes, stream));
  }
  RDQ_REQUIRE(code == 0, RDQ_E_DEVICE, "tiled GEMV: a bounded device-side wait ran out (status %d: %s); results of that launch are invalid",
              static_cast<int>(code), tiled_status_text(code));
  return RDQ_OK;
}

// ---------------------------------------------------------------------------------------
// Peer mode, receiving side: wait (bounded) until every rank's flag on this GPU shows the
// launch this call belongs to, then y[i] = buffer[index[i]] (un-permute out of the gather
// buffer).
// ---------------------------------------------------------------------------------------
namespace {
constexpr int kGatherThreads = 256;
__global__ void __launch_bounds__(kGatherThreads) peer_gather_kernel(const __half *buffer, const long long *index, __half *y,
                                                                    long long count, const int32_t *flags, int world,
                                                                    const int32_t *sent_state, int32_t *status, int wait_ms) {
  __shared__ int ok;
  // let the next layer's GEMV become resident now (it only fills its weight rings until this
  // kernel is complete), then wait for this layer's GEMV
  pdl_launch_dependents();
  pdl_wait();
  if (threadIdx.x == 0) ok = 1;
  __syncthreads();
  // the GEMV of this launch has completed on this GPU: its launch number is the one every
  // rank's flag must show
  const int launch = sent_state[1];
  if (threadIdx.x < world) {
    int v = 0;
    // about wait_ms milliseconds of 0.25 us naps
    for (long long spin = 0; spin < 4000ll * wait_ms; ++spin) {
      asm volatile("ld.acquire.sys.global.s32 %0, [%1];" : "=r"(v) : "l"(flags + threadIdx.x) : "memory");
      if (v >= launch) break;
      __nanosleep(250);
    }
    if (v < launch) {
      ok = 0;
      atomicExch(status, 10 + static_cast<int>(threadIdx.x));  // 10 + rank that never arrived
    }
  }
  __syncthreads();
  if (!ok) return;
  const long long stride = 1ll * gridDim.x * blockDim.x;
  long long i = 1ll * blockIdx.x * blockDim.x + threadIdx.x;
  for (; i + 3 * stride < count; i += 4 * stride) {  // four independent index -> value chains in flight
    const long long j0 = index[i], j1 = index[i + stride], j2 = index[i + 2 * stride], j3 = index[i + 3 * stride];
    const __half v0 = buffer[j0], v1 = buffer[j1], v2 = buffer[j2], v3 = buffer[j3];
    y[i] = v0; y[i + stride] = v1; y[i + 2 * stride] = v2; y[i + 3 * stride] = v3;
  }
  for (; i < count; i += stride) y[i] = buffer[index[i]];
}
}  // namespace

int launch_peer_gather(const __half *buffer, const long long *index, __half *y, long long count, const int32_t *flags,
                       int world, const int32_t *sent_state, int32_t *status, int wait_ms, bool pdl, cudaStream_t stream) {
  // one CTA per SM, each with the footprint that keeps a second one off its SM (pin_slot); every
  // CTA waits for the flags, so none leaves before the GEMV after this kernel has its CTAs placed
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(sm_count()));
  cfg.blockDim = dim3(kGatherThreads);
  cfg.dynamicSmemBytes = kSlotSmem;
  cfg.stream = stream;
  RDQ_CUDA(pin_slot(reinterpret_cast<const void *>(peer_gather_kernel), kSlotSmem));
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = pdl ? 1 : 0;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  RDQ_CUDA(cudaLaunchKernelEx(&cfg, peer_gather_kernel, buffer, index, y, count, flags, world, sent_state, status, wait_ms));
  return RDQ_OK;
}

}  // namespace rdq
