// Decode GEMV (M <= 16) on the row-major tensors, for layers without a tiled layout (groups that are
// not multiples of 16 rows, awkward K) -- same arithmetic contract as the tiled one.
//
// K % 16 == 0 (gemv_rows_kernel): a block takes 16 rows of one format group, its eight warps every
// eighth step of 64 k.  A lane loads 16 consecutive k of rows g and g + 8 (8 / 16 / 32 packed bytes)
// and the same 16 k of activation row g, several steps ahead; they are the operands of four
// mma.sync m16n8k16 (any assignment of k to lanes is fine as long as both operands use it).  The
// warps' sums meet in shared memory.  Bound: latency (three dependent round trips) below a few MB of
// weights, HBM above.  A warp per row with scalar products and one load in flight took 16.6 us for
// 3001 x 4112 and five activation rows (9 MB), whose activations it read once per row.
//
// Other K (gemv_scalar_kernel): one warp per row, element by element.
//
// Reference behaviour replaced: rdquant/ops.py:55-66 (per-group dequant +
// F.linear + cat + index_select) and kernel K1 rdquant/csrc/fused_gemv.cu:1198-1242.
#include "rdq_kernels.cuh"

namespace rdq {

namespace {

constexpr int kWarps = 8;
// Most bytes of weights that a launch asks into L2 before it may read them.  Calls one after another: 600 x 1040
// at 4 rows 2.8 -> 2.6 us, 3001 x 4112 (9 MB) at 5 rows 7.6 -> 7.3; beyond, the requests are in the way of the kernel before:
// 9000 x 2064 (13 MB) at 3 rows 9.0 -> 9.1, 5000 x 6160 (22 MB) at 8 rows 16.5 -> 18.1.
constexpr double kAskAhead = 10e6;

__device__ __forceinline__ uint4 ldg_stream16(const void *p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ uint2 ldg_stream8(const void *p) {
  uint2 v;
  asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}

// Raw operands of one step: 16 k of two weight rows.
template <int FMT>
struct Raw;
template <>
struct Raw<0> {  // NVFP4: 8 bytes and a block scale per row
  uint2 q[2];
  uint32_t s[2];
  __device__ __forceinline__ void load(const GemvArgs &a, int r, int r8, int k) {
    q[0] = ldg_stream8(a.w4 + 1ll * r * (a.K >> 1) + (k >> 1));
    q[1] = ldg_stream8(a.w4 + 1ll * r8 * (a.K >> 1) + (k >> 1));
    s[0] = __ldg(a.s4 + 1ll * r * (a.K >> 4) + (k >> 4));
    s[1] = __ldg(a.s4 + 1ll * r8 * (a.K >> 4) + (k >> 4));
  }
  __device__ __forceinline__ void halves(int i, uint32_t (&h)[8]) const {
    const uint32_t sc = __byte_perm(cvt_e4m3x2(s[i]), 0u, 0x1010u);
    cvt_e2m1x8(q[i].x, h[0], h[1], h[2], h[3]);
    cvt_e2m1x8(q[i].y, h[4], h[5], h[6], h[7]);
#pragma unroll
    for (int e = 0; e < 8; ++e) h[e] = hmul2_u32(h[e], sc);
  }
};
template <>
struct Raw<1> {  // FP8: 16 bytes per row
  uint4 q[2];
  __device__ __forceinline__ void load(const GemvArgs &a, int r, int r8, int k) {
    q[0] = ldg_stream16(a.w8 + 1ll * r * a.K + k);
    q[1] = ldg_stream16(a.w8 + 1ll * r8 * a.K + k);
  }
  __device__ __forceinline__ void halves(int i, uint32_t (&h)[8]) const {
    cvt_e4m3x4(q[i].x, h[0], h[1]);
    cvt_e4m3x4(q[i].y, h[2], h[3]);
    cvt_e4m3x4(q[i].z, h[4], h[5]);
    cvt_e4m3x4(q[i].w, h[6], h[7]);
  }
};
template <>
struct Raw<2> {  // FP16: 32 bytes per row
  uint4 q[4];
  __device__ __forceinline__ void load(const GemvArgs &a, int r, int r8, int k) {
    const __half *p = a.w16 + 1ll * r * a.K + k, *p8 = a.w16 + 1ll * r8 * a.K + k;
    q[0] = ldg_stream16(p);
    q[1] = ldg_stream16(p + 8);
    q[2] = ldg_stream16(p8);
    q[3] = ldg_stream16(p8 + 8);
  }
  __device__ __forceinline__ void halves(int i, uint32_t (&h)[8]) const {
    const uint4 u = q[2 * i], v = q[2 * i + 1];
    h[0] = u.x; h[1] = u.y; h[2] = u.z; h[3] = u.w;
    h[4] = v.x; h[5] = v.y; h[6] = v.z; h[7] = v.w;
  }
};

// Sums of 16 rows x 8 NT activation rows over this warp's steps.  U: steps in flight.
template <int FMT, int NT, bool XBF16, int U>
__device__ __forceinline__ void run_rows(const GemvArgs &a, int r, int r8, int warp, int t, const __half *const (&xr)[NT],
                                         float (&acc)[NT][4]) {
  const int steps = (a.K + 63) >> 6;
  for (int s0 = warp; s0 < steps; s0 += kWarps * U) {
    Raw<FMT> w[U];
    uint4 x[U][NT][2];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = (s0 + u * kWarps) * 64 + t * 16;
      if (k < a.K) {
        w[u].load(a, r, r8, k);
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          const uint4 *xp = reinterpret_cast<const uint4 *>(xr[n] + k);
          x[u][n][0] = __ldg(xp);
          x[u][n][1] = __ldg(xp + 1);
        }
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = (s0 + u * kWarps) * 64 + t * 16;
      if ((s0 + u * kWarps) * 64 >= a.K) break;  // the whole warp is past the row
      uint32_t h[8], h8[8], xv[NT][8];
      const bool valid = k < a.K;
      if (valid) {
        w[u].halves(0, h);
        w[u].halves(1, h8);
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        h[e] = valid ? h[e] : 0u;
        h8[e] = valid ? h8[e] : 0u;
      }
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        const uint4 p = x[u][n][0], q = x[u][n][1];
        const uint32_t raw[8] = {p.x, p.y, p.z, p.w, q.x, q.y, q.z, q.w};
#pragma unroll
        for (int e = 0; e < 8; ++e) xv[n][e] = valid ? (XBF16 ? bf16x2_to_f16x2(raw[e]) : raw[e]) : 0u;
#pragma unroll
        for (int j = 0; j < 4; ++j)
          mma_16816(acc[n], h[2 * j], h8[2 * j], h[2 * j + 1], h8[2 * j + 1], xv[n][2 * j], xv[n][2 * j + 1]);
      }
    }
  }
}

// NT: blocks of eight activation rows
template <int NT, bool XBF16>
__global__ void __launch_bounds__(kWarps * 32) gemv_rows_kernel(const __grid_constant__ GemvArgs a) {
  __shared__ float sums[kWarps][16][8 * NT + 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int t4 = (a.n4 + 15) >> 4, t8 = (a.n8 + 15) >> 4;
  int tile = blockIdx.x, fmt = 0, rows = a.n4, first = 0;
  if (tile >= t4 + t8) {
    fmt = 2;
    tile -= t4 + t8;
    rows = a.n16;
    first = a.n4 + a.n8;
  } else if (tile >= t4) {
    fmt = 1;
    tile -= t4;
    rows = a.n8;
    first = a.n4;
  }
  if (a.ask_ahead) {
    // The tile's rows follow one another: they are asked into L2 ahead of the wait, which is right whatever the
    // kernel before writes, for the loads behind the wait read them there.
    const long long row = fmt == 0 ? a.K >> 1 : (fmt == 1 ? a.K : 2ll * a.K);
    const uint8_t *w = (fmt == 0 ? a.w4 : (fmt == 1 ? a.w8 : reinterpret_cast<const uint8_t *>(a.w16))) + 16 * tile * row;
    const long long bytes = min(16, rows - tile * 16) * row;
    for (long long at = threadIdx.x * 128; at < bytes; at += kWarps * 32 * 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(w + at));
  }
  pdl_wait();
  pdl_launch_dependents();
  // rows beyond the group repeat its last one; activation rows beyond M repeat row 0: neither is stored
  const int r = min(tile * 16 + g, rows - 1), r8 = min(tile * 16 + g + 8, rows - 1);
  const __half *xr[NT];
#pragma unroll
  for (int n = 0; n < NT; ++n) xr[n] = a.x + (n * 8 + g < a.M ? 1ll * (n * 8 + g) * a.K : 0ll);
  float acc[NT][4];
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[n][i] = 0.f;
  if (fmt == 0) run_rows<0, NT, XBF16, NT == 1 ? 4 : 2>(a, r, r8, warp, t, xr, acc);
  else if (fmt == 1) run_rows<1, NT, XBF16, NT == 1 ? 4 : 2>(a, r, r8, warp, t, xr, acc);
  else run_rows<2, NT, XBF16, 2>(a, r, r8, warp, t, xr, acc);
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    sums[warp][g][n * 8 + 2 * t] = acc[n][0];
    sums[warp][g][n * 8 + 2 * t + 1] = acc[n][1];
    sums[warp][g + 8][n * 8 + 2 * t] = acc[n][2];
    sums[warp][g + 8][n * 8 + 2 * t + 1] = acc[n][3];
  }
  __syncthreads();
  const int N = a.n4 + a.n8 + a.n16;
  for (int i = threadIdx.x; i < 16 * a.M; i += kWarps * 32) {
    const int row = i & 15, m = i >> 4, rr = tile * 16 + row;
    if (rr >= rows) continue;
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) v += sums[w][row][m];
    const int prow = first + rr;
    const int col = a.perm ? a.perm[prow] : prow;
    const float scl = fmt == 0 ? a.global4 : (fmt == 1 ? a.s8[rr] : 1.f);
    const float b = a.bias ? __half2float(a.bias[col]) : 0.f;
    store_y(a.y, 1ll * m * N + col, fmaf(v, scl, b), a.y_bf16);
  }
}

__device__ __forceinline__ float elem(const __half *x, long long i, int bf16) {
  return bf16 ? __half2float(__float2half_rn(__bfloat162float(reinterpret_cast<const __nv_bfloat16 *>(x)[i]))) : __half2float(x[i]);
}
// K not a multiple of 16 (no NVFP4 group then)
__global__ void __launch_bounds__(256) gemv_scalar_kernel(const __grid_constant__ GemvArgs a) {
  pdl_wait();
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int N = a.n4 + a.n8 + a.n16;
  if (row >= N) return;
  const int K = a.K, M = a.M;
  float acc[RDQ_MAX_GEMV_M];
#pragma unroll
  for (int m = 0; m < RDQ_MAX_GEMV_M; ++m) acc[m] = 0.f;
  float out_scale = 1.f;
  const bool is8 = row < a.n4 + a.n8;
  const int rr = is8 ? row - a.n4 : row - a.n4 - a.n8;
  if (is8) out_scale = a.s8[rr];
  for (int k = lane; k < K; k += 32) {
    const float w = is8 ? e4m3_to_float(a.w8[1ll * rr * K + k]) : __half2float(a.w16[1ll * rr * K + k]);
#pragma unroll
    for (int m = 0; m < RDQ_MAX_GEMV_M; ++m)
      if (m < M) acc[m] = fmaf(w, elem(a.x, 1ll * m * K + k, a.x_bf16), acc[m]);
  }
  const int col = a.perm ? a.perm[row] : row;
  const float b = a.bias ? __half2float(a.bias[col]) : 0.f;
#pragma unroll
  for (int m = 0; m < RDQ_MAX_GEMV_M; ++m) {
    const float s = warp_sum(acc[m]);
    if (m < M && lane == 0) store_y(a.y, 1ll * m * N + col, fmaf(s, out_scale, b), a.y_bf16);
  }
}

}  // namespace

int launch_gemv_generic(const GemvArgs &args, cudaStream_t stream) {
  GemvArgs a = args;
  a.ask_ahead = a.K * (0.5 * a.n4 + a.n8 + 2.0 * a.n16) <= kAskAhead;
  const int N = a.n4 + a.n8 + a.n16;
  if (N == 0 || a.M == 0) return RDQ_OK;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(256);
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (a.K % 16 == 0) {
    cfg.gridDim = dim3(static_cast<unsigned>((a.n4 + 15) / 16 + (a.n8 + 15) / 16 + (a.n16 + 15) / 16));
    if (a.M <= 8) {
      RDQ_CUDA(a.x_bf16 ? cudaLaunchKernelEx(&cfg, gemv_rows_kernel<1, true>, a) : cudaLaunchKernelEx(&cfg, gemv_rows_kernel<1, false>, a));
    } else {
      RDQ_CUDA(a.x_bf16 ? cudaLaunchKernelEx(&cfg, gemv_rows_kernel<2, true>, a) : cudaLaunchKernelEx(&cfg, gemv_rows_kernel<2, false>, a));
    }
  } else {
    cfg.gridDim = dim3(static_cast<unsigned>((N + 7) / 8));
    RDQ_CUDA(cudaLaunchKernelEx(&cfg, gemv_scalar_kernel, a));
  }
  return RDQ_OK;
}

}  // namespace rdq
