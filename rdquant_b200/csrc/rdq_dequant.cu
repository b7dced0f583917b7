// Bit-exact dequantisation of a packed mixed-precision layer to FP16 or FP32 [N, K] in original
// channel order.  HBM-bound: reads the packed bytes once, writes 2 (or 4) N K bytes once.
//
// A warp per piece of an output row, a lane per 8 consecutive k: a warp instruction reads 128 / 256 / 512
// contiguous bytes of an NVFP4 / FP8 / FP16 row and stores 512 (f16), up to five of them in flight.
// Pieces, because a warp per row leaves a layer of few long rows with too few warps (3884 rows of
// 13840: 34.4 us, now 25.3) and one whose rows are a few more than the warps of the chip with a second
// round for those (9728 rows of 2560: 15.2, now 13.4).  A piece is one turn without a loop, whose registers would
// leave floats six blocks on an SM instead of eight (64 x 300000 66.4 us, now 52.4).
// (16-element runs per thread, with 32-byte store strides and one run in flight, reached 1.9 TB/s.)
//
// Arithmetic follows the reference oracle exactly:
//   NVFP4  f16( f32(LUT[code]) * f32(e4m3 scale) )        rdquant/core/formats.py:145-159
//          (with a global scale of 1 every product is an f16 value: multiplied in f16)
//   FP8    f16( f32(e4m3 byte) * scale[channel] )          rdquant/inference.py:104-109
//   FP16   bf16 -> f32 -> f16 (or a plain copy of f16)     rdquant/inference.py:111-113
// and the row gather is QuantizedWeight.dequantize's cat()[inv_perm]
// (rdquant/quantize.py:56-69).
#include "rdq_kernels.cuh"

namespace rdq {

namespace {

struct DequantArgs {
  const uint8_t *w4;
  const uint8_t *s4;
  float global4;
  const uint8_t *w8;
  const float *s8;
  const void *w16;
  int w16_is_bf16;
  const int32_t *inv_perm;
  void *out;
  int n4, n8, n16, K;
  int segs, len;  // pieces of a row, vectors of eight in a piece
};

// Most vectors of a lane in a piece.  Floats take twice the bytes: with five 1280 x 8000 FP16 rows take 17.3 us, with
// four 14.4, 2560 x 4096 NVFP4 rows 15.7 and 14.0.  Halves: 1280 x 8000 6.8 us with five, 7.3 with four; longer rows
// are up to 3 % faster with four.
template <typename OutT>
constexpr int kUnroll = sizeof(OutT) == 2 ? 5 : 4;

__device__ __forceinline__ void store8(__half *row, int v, const float (&f)[8]) {
  uint4 o;
  uint32_t *w = reinterpret_cast<uint32_t *>(&o);
#pragma unroll
  for (int i = 0; i < 4; ++i) w[i] = pack_y2(f[2 * i], f[2 * i + 1], 0);
  reinterpret_cast<uint4 *>(row)[v] = o;
}
__device__ __forceinline__ void store8(float *row, int v, const float (&f)[8]) {
  reinterpret_cast<float4 *>(row)[2 * v] = make_float4(f[0], f[1], f[2], f[3]);
  reinterpret_cast<float4 *>(row)[2 * v + 1] = make_float4(f[4], f[5], f[6], f[7]);
}
__device__ __forceinline__ void halves_to_floats(const uint32_t (&h)[4], float (&f)[8]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = h2_to_f2(h[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}

// OutT = __half: the operator's weight (products rounded to f16, round to nearest even).
// OutT = float : the unrounded FP32 product, what formats.dequantize returns.
// VEC: K % 8 == 0, so rows are whole runs of 8 with 16-byte (packed: 4-byte) alignment.
template <typename OutT, bool VEC>
__global__ void __launch_bounds__(256) dequant_kernel(DequantArgs a) {
  constexpr int U = kUnroll<OutT>;
  const int lane = threadIdx.x & 31;
  const int K = a.K, N = a.n4 + a.n8 + a.n16;
  const unsigned task = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), segs = a.segs;
  const int n = static_cast<int>(task / segs), first = static_cast<int>(task - n * segs) * a.len + lane;
  const int nvec = min(K >> 3, first - lane + a.len);  // end of the piece
  if (n < N) {
    const int r = a.inv_perm ? a.inv_perm[n] : n;
    OutT *row = static_cast<OutT *>(a.out) + 1ll * n * K;
    if (r < a.n4) {
      // K % 16 == 0 is a precondition of the NVFP4 layout
      const uint32_t *src = reinterpret_cast<const uint32_t *>(a.w4 + 1ll * r * (K >> 1));
      const uint8_t *ssrc = a.s4 + 1ll * r * (K >> 4);
      const bool plain = sizeof(OutT) == 2 && a.global4 == 1.f;
      uint32_t q[U], s[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (first + 32 * u < nvec) {
          q[u] = __ldg(src + first + 32 * u);
          s[u] = __ldg(ssrc + ((first + 32 * u) >> 1));
        }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (first + 32 * u >= nvec) break;
        uint32_t h[4];
        cvt_e2m1x8(q[u], h[0], h[1], h[2], h[3]);
        if (plain) {
          const uint32_t sc = __byte_perm(cvt_e4m3x2(s[u]), 0u, 0x1010u);
          reinterpret_cast<uint4 *>(row)[first + 32 * u] =
              make_uint4(hmul2_u32(h[0], sc), hmul2_u32(h[1], sc), hmul2_u32(h[2], sc), hmul2_u32(h[3], sc));
        } else {
          const float sc = e4m3_to_float(s[u]) * a.global4;
          float f[8];
          halves_to_floats(h, f);
#pragma unroll
          for (int i = 0; i < 8; ++i) f[i] *= sc;
          store8(row, first + 32 * u, f);
        }
      }
    } else if (r < a.n4 + a.n8) {
      const int rr = r - a.n4;
      const float sc = a.s8[rr];
      const uint8_t *src = a.w8 + 1ll * rr * K;
      if (VEC) {
        uint2 q[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (first + 32 * u < nvec) q[u] = __ldg(reinterpret_cast<const uint2 *>(src) + first + 32 * u);
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (first + 32 * u >= nvec) break;
          uint32_t h[4];
          cvt_e4m3x4(q[u].x, h[0], h[1]);
          cvt_e4m3x4(q[u].y, h[2], h[3]);
          float f[8];
          halves_to_floats(h, f);
#pragma unroll
          for (int i = 0; i < 8; ++i) f[i] *= sc;
          store8(row, first + 32 * u, f);
        }
      } else {
        for (int k = lane; k < K; k += 32) row[k] = static_cast<OutT>(e4m3_to_float(src[k]) * sc);
      }
    } else {
      const long long off = 1ll * (r - a.n4 - a.n8) * K;
      const uint16_t *src = static_cast<const uint16_t *>(a.w16) + off;
      if (VEC) {
        uint4 q[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (first + 32 * u < nvec) q[u] = __ldg(reinterpret_cast<const uint4 *>(src) + first + 32 * u);
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (first + 32 * u >= nvec) break;
          uint32_t h[4] = {q[u].x, q[u].y, q[u].z, q[u].w};
          if (a.w16_is_bf16) {
#pragma unroll
            for (int i = 0; i < 4; ++i) h[i] = bf16x2_to_f16x2(h[i]);
          }
          float f[8];
          halves_to_floats(h, f);
          store8(row, first + 32 * u, f);
        }
      } else {
        for (int k = lane; k < K; k += 32) {
          const __half h = a.w16_is_bf16 ? __float2half_rn(__bfloat162float(__ushort_as_bfloat16(src[k]))) : __ushort_as_half(src[k]);
          row[k] = static_cast<OutT>(__half2float(h));
        }
      }
    }
  }
}

}  // namespace

int launch_dequant(const void *w_fp4, const void *w_fp4_scales, float global4, const void *w_fp8,
                   const float *w_fp8_scales, const void *w_fp16, int fp16_is_bf16,
                   const int32_t *inv_perm, void *w_out, int out_is_f32, int n4, int n8, int n16,
                   int K, cudaStream_t stream) {
  DequantArgs a;
  a.w4 = static_cast<const uint8_t *>(w_fp4);
  a.s4 = static_cast<const uint8_t *>(w_fp4_scales);
  a.global4 = global4;
  a.w8 = static_cast<const uint8_t *>(w_fp8);
  a.s8 = w_fp8_scales;
  a.w16 = w_fp16;
  a.w16_is_bf16 = fp16_is_bf16;
  a.inv_perm = inv_perm;
  a.out = w_out;
  a.n4 = n4;
  a.n8 = n8;
  a.n16 = n16;
  a.K = K;
  const long long rows = 1ll * n4 + n8 + n16;
  if (rows == 0) return RDQ_OK;
  const bool vec = K % 8 == 0;
  const RowPieces cut = vec ? row_pieces(K, out_is_f32 ? kUnroll<float> : kUnroll<__half>) : RowPieces{1, 0};
  a.segs = cut.pieces;
  a.len = 32 * cut.len;
  const unsigned blocks = static_cast<unsigned>((rows * a.segs + 7) / 8);
  if (out_is_f32) {
    if (vec) dequant_kernel<float, true><<<blocks, 256, 0, stream>>>(a);
    else dequant_kernel<float, false><<<blocks, 256, 0, stream>>>(a);
  } else {
    if (vec) dequant_kernel<__half, true><<<blocks, 256, 0, stream>>>(a);
    else dequant_kernel<__half, false><<<blocks, 256, 0, stream>>>(a);
  }
  RDQ_CUDA(cudaGetLastError());
  return RDQ_OK;
}

}  // namespace rdq
