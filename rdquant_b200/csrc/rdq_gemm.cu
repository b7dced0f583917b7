// GEMM without scratch memory  y[M, N] = x[M, K] . W[N, K]^T (+ bias)  for the mixed-precision
// layer (callers with a workspace get the faster kernels of rdq_gemm_stream.cu and
// rdq_gemm_dense.cu), sm_100a: dequantise-to-shared-memory producers feeding tcgen05 kind::f16 MMAs with the
// FP32 accumulator in tensor memory.
//
// Tile: 128 or 256 tokens x 128 or 256 output channels per CTA (chosen per launch by a time
// estimate, see gemm_config), k blocks of 64.  The output tile is taken in ORIGINAL channel order:
// channel n0 + j reads permuted row inv_perm[n0 + j], so the permutation costs nothing on the
// store side (rows of all three formats meet in one tile).
//
//   warp 0 (1 thread)   TMA (cp.async.bulk.tensor.2d, 128B swizzle) loads of the 128 x 64
//                       activation blocks into the A stage (one per 128 tokens).
//   warp 1 (1 thread)   issues 4 x tcgen05.mma (M128, N = tile width, K16) per k block and
//                       128-token accumulator, commits the stage back to the producers,
//                       finally commits the accumulators.  The warp also owns the
//                       tensor-memory allocation (up to all 512 columns).
//   warps 2..           12 or 22 dequantisation warps.  The rows of the tile are sorted by
//                       format and padded to groups of four; a warp takes every W-th group,
//                       a quarter warp one row, a lane one 16-byte chunk (8 k) of it: it
//                       loads the next k block's 4 / 8 / 16 packed bytes into registers,
//                       converts the current ones to f16 (NVFP4: hardware E2M1 converter
//                       times the block scale, exact in f16; FP8: E4M3 converter, channel
//                       scale deferred to the epilogue; FP16: copy) and stores its chunk in
//                       the K-major 128B-swizzled layout the MMA descriptor expects -- the
//                       eight lanes of a row write 128 contiguous bytes (no bank conflicts)
//                       and read 32 / 64 / 128 contiguous bytes.
//   epilogue            twelve of those warps: tcgen05.ld of the accumulators (a warp reads
//                       the 32 tensor-memory lanes of its quarter, the warps of a quarter
//                       take pairs of 32-column chunks in turn), channel scale and bias, f16
//                       conversion, transposition through the free stage buffers, stores of
//                       4 rows x 128 contiguous bytes per instruction.
//
// Shared memory: 4 stages x (16 or 32 KB A + 16 KB B), or 3 x (32 KB A + 32 KB B) for the
// 256 x 256 tile.  All mbarrier waits are bounded; a wait that runs out raises an abort flag
// that every role checks, and the kernel drains and frees its tensor memory.
//
// Measured on B200 (in-kernel clocks, 256 x 256 tile): with the weight conversion switched
// off the pipeline runs at the MMA rate (1024 cycles per k block); with it, about 1450 cycles.
// Shared-memory bandwidth is the bound: per k block the MMAs read 96 KB (A and B once per
// M128 instruction), TMA writes 32 KB and the producers 32 KB = 160 KB at 128 B/clk.
//
// FLOPs per launch: 2*M*N*K.  Bound: dense f16 tensor throughput.
//
// Reference behaviour replaced: F.linear over a materialised FP16 weight copy
// (rdquant/inference.py:679-687) and 2 x marlin_gemm + F.linear + cat + index_select
// (rdquant/inference.py:620-677).
#include <cuda.h>

#include "rdq_gemm_common.cuh"
#include "rdq_kernels.cuh"

namespace rdq {

namespace {

constexpr int BM = 128, BK = 64;
constexpr int kStageA = BM * BK * 2;  // 16 KB: one 128-token activation block
constexpr int kMaxBN = 256;

// Tile configurations.  BN = output channels per CTA (= N of one tcgen05.mma), MT = 128-token
// accumulators per CTA.  Producer warps convert groups of four weight rows (a quarter warp per
// row); kTasks = groups a warp handles per k block.
//   <1,128> <2,128>: 12 producer warps, 4 stages         (small problems)
//   <2,256>        : 22 producer warps (768 threads), 3 x 64 KB stages, all 512 tensor-memory columns
template <int MT, int BN>
struct GemmCfg {
  static constexpr int kProducerWarps = (BN == 128) ? 12 : 22;
  static constexpr int kProducers = kProducerWarps * 32;
  static constexpr int kThreads = (2 + kProducerWarps) * 32;
  static constexpr int kStageB = BN * BK * 2;
  static constexpr int kStageAll = kStageA * MT;
  static constexpr int kStages = (BN == 128) ? 4 : 3;
  static constexpr int kTmemCols = BN * MT;  // power of two >= 32
  static constexpr int kSmem = kStages * (kStageAll + kStageB) + 1024;
  static constexpr int kMaxQuads = BN / 4 + 3;  // each format padded to a multiple of four rows
  static constexpr int kTasks = (kMaxQuads + kProducerWarps - 1) / kProducerWarps;
  static constexpr int kPrefetch = 1;  // k blocks of packed weights held in registers ahead of use
};

struct GemmSmem {
  // dynamic part starts 1024-byte aligned: A stages, then B stages
  // static part:
  uint64_t full[4];
  uint64_t empty[4];
  uint64_t accum;
  uint64_t never;  // nothing ever arrives here (time-out self-test)
  uint32_t tmem_base;
  int abort_flag;
  int row_perm[kMaxBN];       // permuted row of tile row j, or -1
  int prow[kMaxBN + 12];      // tile rows sorted by format, each format padded to four (-1)
  int nquad;                  // groups of four rows in prow
  float colscale[kMaxBN];
  float colbias[kMaxBN];
};

__device__ __forceinline__ uint4 ldg_nc16(const void *p) {
  uint4 v;
  asm volatile("ld.global.nc.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ uint32_t ldg_nc4(const void *p) {
  uint32_t v;
  asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

}  // namespace
}  // namespace rdq

#include "rdq_gemm_kernel.inl"
