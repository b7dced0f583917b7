// Encoders: a float weight group [n, K] -> the packed checkpoint tensors of the NVFP4 or FP8
// format, bit for bit what the reference's CPU encoders produce
// (rdquant/core/formats.py:84-142 nvfp4_quantize, :166-193 fp8_quantize; byte layout
// rdquant/integrations/hf_export.py:81-102), plus the per-row sum of squared reconstruction
// errors that the per-channel MSE of the format search needs
// (rdquant/core/formats.py:414-436 compute_mse_2d: mean over the row of (w - dequant)^2); and a whole
// layer at once, its rows gathered by the channel permutation on the way in (rdq_quantize_layer).
//
// One warp per row, a lane per 8 consecutive k: loads of 512 (f16) contiguous bytes per warp
// instruction, four in flight; a pair of lanes shares a block of 16 (K % 16 == 0, so the reference's
// blocks over the flattened group coincide with blocks inside rows).
//
// Bound: HBM (reads 2 or 4 bytes per element, writes 0.56 / 1).  The reference divides every element
// by its scale; here
//   NVFP4  no division per element: the code counts the grid midpoints t with fl(v / s) > t, and for a
//          scale s with a 4-bit mantissa that is v > t s (t s is exact; fl(v / s) > t needs v / s to
//          exceed t by half an ulp, and a float v above t s exceeds it by more: the relative step of v
//          is above 2^-24 there, half an ulp of t at most 2^-24).  The sign of a quotient that
//          underflows to zero is the one exception: denormal inputs are compared with s / 2 steps.
//          An f16 v that is not t s itself differs from it by more than 2^-12 of it, so v (1 - 2^-14) / s
//          lies on the right side of every midpoint and below one that v / s hits: the hardware's
//          round-to-nearest E2M1 converter then gives the code (adding +0 turns -0 into +0, whose code
//          is 0).  Counting thresholds instead took 32 us for a 2560 x 9728 layer.
//   FP8    v is multiplied by 1 / scale a little less and a little more; only where the two products
//          round to different E4M3 values does the division decide.
// The E4M3 rounding is the hardware converter's round-to-nearest-even, the same as
// torch.float8_e4m3fn's.
#include <cuda_fp8.h>

#include <algorithm>

#include "rdq_kernels.cuh"

namespace rdq {

namespace {

constexpr int kUnroll = 4;  // vectors of 8 elements in flight per lane

template <typename T>
struct Vec8;
template <>
struct Vec8<__half> {
  uint4 q;
  __device__ __forceinline__ void zero() { q = make_uint4(0u, 0u, 0u, 0u); }
  __device__ __forceinline__ float amax() const {  // (NaN ignored)
    const __half2 a = __hmax2(__habs2(*reinterpret_cast<const __half2 *>(&q.x)), __habs2(*reinterpret_cast<const __half2 *>(&q.y)));
    const __half2 b = __hmax2(__habs2(*reinterpret_cast<const __half2 *>(&q.z)), __habs2(*reinterpret_cast<const __half2 *>(&q.w)));
    const float2 f = __half22float2(__hmax2(a, b));
    return fmaxf(f.x, f.y);
  }
  __device__ __forceinline__ void load(const __half *p) { q = __ldg(reinterpret_cast<const uint4 *>(p)); }
  __device__ __forceinline__ void get(float (&v)[8]) const {
    const uint32_t u[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 f = h2_to_f2(u[e]);
      v[2 * e] = f.x;
      v[2 * e + 1] = f.y;
    }
  }
};
template <>
struct Vec8<float> {
  float4 a, b;
  __device__ __forceinline__ void zero() { a = b = make_float4(0.f, 0.f, 0.f, 0.f); }
  __device__ __forceinline__ float amax() const {
    return fmaxf(fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(a.z), fabsf(a.w))),
                 fmaxf(fmaxf(fabsf(b.x), fabsf(b.y)), fmaxf(fabsf(b.z), fabsf(b.w))));
  }
  __device__ __forceinline__ void load(const float *p) {
    a = __ldg(reinterpret_cast<const float4 *>(p));
    b = __ldg(reinterpret_cast<const float4 *>(p) + 1);
  }
  __device__ __forceinline__ void get(float (&v)[8]) const {
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  }
};

// Largest magnitude of a vector and its neighbour lane's (a block of 16); `finite`: neither infinity nor
// NaN among them (else the magnitude is not to be used).
__device__ __forceinline__ float block_amax(const Vec8<__half> &q, bool &finite) {
  __half2 m = __habs2(*reinterpret_cast<const __half2 *>(&q.q.x));
  m = __hmax2_nan(m, __habs2(*reinterpret_cast<const __half2 *>(&q.q.y)));
  m = __hmax2_nan(m, __habs2(*reinterpret_cast<const __half2 *>(&q.q.z)));
  m = __hmax2_nan(m, __habs2(*reinterpret_cast<const __half2 *>(&q.q.w)));
  const uint32_t other = __shfl_xor_sync(0xffffffffu, *reinterpret_cast<const uint32_t *>(&m), 1);
  m = __hmax2_nan(m, *reinterpret_cast<const __half2 *>(&other));
  const float2 f = __half22float2(m);
  finite = f.x < INFINITY && f.y < INFINITY;
  return fmaxf(f.x, f.y);
}
__device__ __forceinline__ float block_amax(const Vec8<float> &q, bool &finite) {
  float v[8];
  q.get(v);
  // bit patterns order magnitudes and put NaN above infinity
  uint32_t bits = 0;
#pragma unroll
  for (int e = 0; e < 8; ++e) bits = max(bits, __float_as_uint(v[e]) & 0x7fffffffu);
  bits = max(bits, __shfl_xor_sync(0xffffffffu, bits, 1));
  finite = bits < 0x7f800000u;
  return __uint_as_float(bits);
}
// The E4M3 input amax / 6.  An f16 amax gives a quotient that is exact or further than an ulp from every
// rounding boundary (six times a boundary is an f16 value itself): a product with one residual
// correction is as good as the division.
__device__ __forceinline__ float sixth(const Vec8<__half> &, float amax) {
  const float r = 1.f / 6.f, q = amax * r;
  return fmaf(fmaf(-6.f, q, amax), r, q);
}
__device__ __forceinline__ float sixth(const Vec8<float> &, float amax) { return __fdiv_rn(amax, 6.f); }

__device__ __forceinline__ uint8_t to_e4m3(float v) {
  return static_cast<uint8_t>(__nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3));
}
__device__ __forceinline__ float from_e4m3(uint8_t b) {
  const __half_raw h = __nv_cvt_fp8_to_halfraw(static_cast<__nv_fp8_storage_t>(b), __NV_E4M3);
  return __half2float(__half(h));
}
__device__ __forceinline__ float clamp448(float v) { return fminf(fmaxf(v, -448.f), 448.f); }

// deterministic max of non-negative floats through their bit patterns
__device__ __forceinline__ void atomic_max_nonneg(float *addr, float v) {
  atomicMax(reinterpret_cast<unsigned int *>(addr), __float_as_uint(v));
}
__device__ __forceinline__ float max8(const float (&v)[8]) {
  float m = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) m = fmaxf(m, fabsf(v[i]));
  return m;
}

// eight values -> E2M1 codes, a nibble each, the first in the lowest
__device__ __forceinline__ uint32_t cvt_to_e2m1x8(const float (&v)[8]) {
  uint32_t r;
  asm("{\n.reg .b8 b0, b1, b2, b3;\n"
      "cvt.rn.satfinite.e2m1x2.f32 b0, %2, %1;\ncvt.rn.satfinite.e2m1x2.f32 b1, %4, %3;\n"
      "cvt.rn.satfinite.e2m1x2.f32 b2, %6, %5;\ncvt.rn.satfinite.e2m1x2.f32 b3, %8, %7;\n"
      "mov.b32 %0, {b0, b1, b2, b3};\n}\n"
      : "=r"(r)
      : "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]));
  return r;
}
// value of the code in the low four bits: its sign, two exponent bits and a mantissa bit at a float's places
// are the value times 2^-126
__device__ __forceinline__ float grid_value(uint32_t c) {
  return __uint_as_float(((c & 8u) << 28) | ((c & 7u) << 22)) * 8.50705917e37f;
}
// Half a block of 16: codes of eight values (a nibble each, low nibble first), by counting thresholds.
template <bool SQERR>
__device__ __forceinline__ uint32_t encode_fp4(const float (&v)[8], float scale, float &err) {
  const float s = scale == 0.f ? 1.f : scale;
  const float t0 = 0.25f * s, t1 = 0.75f * s, t2 = 1.25f * s, t3 = 1.75f * s, t4 = 2.5f * s, t5 = 3.5f * s, t6 = 5.0f * s;
  // the quotient of a denormal v (its bits count steps of 2^-149) is zero when v is at most s / 2 of them
  const int vanish = static_cast<int>(0.5f * s);
  uint32_t packed = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float mag = fabsf(v[i]);
    const int m = (mag > t0) + (mag > t1) + (mag > t2) + (mag > t3) + (mag > t4) + (mag > t5) + (mag > t6);
    const bool neg = v[i] < 0.f && __float_as_int(mag) > vanish;
    packed |= static_cast<uint32_t>(m + (neg ? 8 : 0)) << (4 * i);
    if (SQERR) {
      const float d = v[i] - __fmul_rn(grid_value(static_cast<uint32_t>(m + (neg ? 8 : 0))), scale);
      err = fmaf(d, d, err);
    }
  }
  return packed;
}

__device__ __noinline__ uint32_t encode_fp4_any(float4 a, float4 b, float scale) {
  const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  float none = 0.f;
  return encode_fp4<false>(v, scale, none);
}
// ... of finite f16 values
__device__ __forceinline__ uint32_t encode_fp4_f16(const float (&v)[8], float scale) {
  const float c = __fdividef(1.f, scale == 0.f ? 1.f : scale) * (1.f - 6.103515625e-5f);
  float p[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) p[i] = fmaf(v[i], c, 0.f);
  return cvt_to_e2m1x8(p);
}

// Vector i of a row (its neighbour lane holds the other half of the block) -> codes u8 [K / 2], scales
// u8 [K / 16]; the block scale joins `top`.  All lanes of the warp take part; live: the vector exists.
template <typename T, bool SQERR>
__device__ __forceinline__ void encode_vec_fp4(Vec8<T> &q, bool live, int i, uint8_t *codes, uint8_t *scales, float &top, float &err) {
  if (!live) q.zero();
  bool finite;
  float amax = block_amax(q, finite);
  float v[8];
  q.get(v);
  float a6 = sixth(q, amax);
  if (__any_sync(0xffffffffu, !finite)) {  // the scale ignores NaN
    amax = max8(v);
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    a6 = __fdiv_rn(amax, 6.f);
  }
  const uint8_t sbits = to_e4m3(a6);  // (saturates at 448)
  const float scale = from_e4m3(sbits);
  top = fmaxf(top, scale);
  if (live) {
    uint32_t code;
    if (sizeof(T) == 4) {
      code = encode_fp4<SQERR>(v, scale, err);
    } else if (finite) {
      code = encode_fp4_f16(v, scale);
      if (SQERR) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float d = v[e] - __fmul_rn(grid_value(code >> (4 * e)), scale);
          err = fmaf(d, d, err);
        }
      }
    } else if (SQERR) {
      code = encode_fp4<SQERR>(v, scale, err);
    } else {
      code = encode_fp4_any(make_float4(v[0], v[1], v[2], v[3]), make_float4(v[4], v[5], v[6], v[7]), scale);
    }
    reinterpret_cast<uint32_t *>(codes)[i] = code;
    if (!(i & 1)) scales[i >> 1] = sbits;
  }
}
// A row of K values
template <typename T, bool SQERR>
__device__ __forceinline__ void encode_row_fp4(const T *w, int K, uint8_t *codes, uint8_t *scales, int lane, float &top, float &err) {
  const int nvec = K >> 3;
  for (int v0 = lane; v0 - lane < nvec; v0 += 32 * kUnroll) {
    Vec8<T> q[kUnroll];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u)
      if (v0 + 32 * u < nvec) q[u].load(w + 8ll * (v0 + 32 * u));
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      if (v0 - lane + 32 * u >= nvec) break;  // the whole warp is past the row
      encode_vec_fp4<T, SQERR>(q[u], v0 + 32 * u < nvec, v0 + 32 * u, codes, scales, top, err);
    }
  }
}

__device__ __forceinline__ uint2 to_e4m3x8(const float (&r)[8]) {
  uint32_t h[4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
    h[i] = __nv_cvt_float2_to_fp8x2(make_float2(r[2 * i], r[2 * i + 1]), __NV_SATFINITE, __NV_E4M3);
  return make_uint2(h[0] | (h[1] << 16), h[2] | (h[3] << 16));
}
// any byte with all of the low seven bits set
__device__ __forceinline__ bool has_nan(uint32_t w) { return (((w & 0x7f7f7f7fu) + 0x01010101u) & 0x80808080u) != 0; }
__device__ __noinline__ uint2 divide_e4m3(float4 a, float4 b, float scale) {
  const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  float r[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) r[i] = clamp448(__fdiv_rn(v[i], scale));
  return to_e4m3x8(r);
}
// fl(v / scale) rounded to E4M3 for eight values; inv = fl(1 / scale) or 0.  The quotient lies between the
// products with inv (1 -+ 2^-21); where both round to the same E4M3 value, so does the quotient.
__device__ __forceinline__ uint2 quotients_e4m3(const float (&v)[8], float scale, float inv) {
  const float lo = inv * (1.f - 4.76837158e-7f), hi = inv * (1.f + 4.76837158e-7f);
  float r[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) r[i] = v[i] * lo;
  const uint2 p = to_e4m3x8(r);
#pragma unroll
  for (int i = 0; i < 8; ++i) r[i] = v[i] * hi;
  const uint2 q = to_e4m3x8(r);
  if (p.x == q.x && p.y == q.y && !has_nan(p.x) && !has_nan(p.y) && inv != 0.f) return p;
  return divide_e4m3(make_float4(v[0], v[1], v[2], v[3]), make_float4(v[4], v[5], v[6], v[7]), scale);
}
// fl(1 / scale), or 0 where a product with it may lose bits that the quotient has
__device__ __forceinline__ float fp8_inverse(float scale) {
  const float inv = __fdiv_rn(1.f, scale);
  return inv > 1e-30f && inv < 1e30f ? inv : 0.f;
}

template <typename T, bool SQERR>
__device__ __forceinline__ void encode_row_fp8(const T *w, int K, float scale, uint8_t *out, int lane, float &err) {
  const float inv = fp8_inverse(scale);
  const int nvec = K >> 3;
  for (int v0 = lane; v0 < nvec; v0 += 32 * kUnroll) {
    Vec8<T> q[kUnroll];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u)
      if (v0 + 32 * u < nvec) q[u].load(w + 8ll * (v0 + 32 * u));
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const int i = v0 + 32 * u;
      if (i >= nvec) break;
      float v[8];
      q[u].get(v);
      const uint2 o = quotients_e4m3(v, scale, inv);
      if (SQERR) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float d = v[e] - __fmul_rn(from_e4m3(static_cast<uint8_t>((e < 4 ? o.x : o.y) >> (8 * (e & 3)))), scale);
          err = fmaf(d, d, err);
        }
      }
      reinterpret_cast<uint2 *>(out)[i] = o;
    }
  }
}

template <typename T>
__device__ __forceinline__ float absmax_row(const T *w, int K, int lane) {
  const int nvec = K >> 3;
  float m = 0.f;
  for (int v0 = lane; v0 < nvec; v0 += 32 * kUnroll) {
    Vec8<T> q[kUnroll];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u)
      if (v0 + 32 * u < nvec) q[u].load(w + 8ll * (v0 + 32 * u));
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      if (v0 + 32 * u >= nvec) break;
      m = fmaxf(m, q[u].amax());
    }
  }
  return m;
}

__device__ __forceinline__ float fp8_scale(float absmax) {
  const float s = __fdiv_rn(absmax, 448.f);
  return s == 0.f ? 1.f : s;
}

template <typename T, bool SQERR>
__global__ void __launch_bounds__(256) quantize_nvfp4_kernel(const T *__restrict__ w, int n, int K, uint8_t *__restrict__ codes,
                                                             uint8_t *__restrict__ scales, float *__restrict__ row_sqerr,
                                                             float *__restrict__ max_scale) {
  const int lane = threadIdx.x & 31;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  float top = 0.f;
  for (int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; row < n; row += warps) {
    float err = 0.f;
    encode_row_fp4<T, SQERR>(w + 1ll * row * K, K, codes + 1ll * row * (K >> 1), scales + 1ll * row * (K >> 4), lane, top, err);
    if (SQERR) {
      err = warp_sum(err);
      if (lane == 0) row_sqerr[row] = err;
    }
  }
  if (max_scale) {
    top = warp_max(top);
    if (lane == 0 && top > 0.f) atomic_max_nonneg(max_scale, top);
  }
}

template <typename T>
__global__ void __launch_bounds__(256) absmax_kernel(const T *__restrict__ w, int n, int K, float *__restrict__ out) {
  const int lane = threadIdx.x & 31;
  float m = 0.f;
  for (int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; row < n; row += (gridDim.x * blockDim.x) >> 5)
    m = fmaxf(m, absmax_row(w + 1ll * row * K, K, lane));
  m = warp_max(m);
  if (lane == 0 && m > 0.f) atomic_max_nonneg(out, m);
}

template <typename T, bool SQERR>
__global__ void __launch_bounds__(256) quantize_fp8_kernel(const T *__restrict__ w, int n, int K, const float *__restrict__ absmax,
                                                           uint8_t *__restrict__ out, float *__restrict__ scale_out,
                                                           float *__restrict__ row_sqerr) {
  const int lane = threadIdx.x & 31;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  const float scale = fp8_scale(*absmax);
  for (int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; row < n; row += warps) {
    float err = 0.f;
    encode_row_fp8<T, SQERR>(w + 1ll * row * K, K, scale, out + 1ll * row * K, lane, err);
    if (lane == 0 && scale_out) scale_out[row] = scale;
    if (SQERR) {
      err = warp_sum(err);
      if (lane == 0) row_sqerr[row] = err;
    }
  }
}

// ---- a whole layer: permuted row r is channel perm[r] of w
struct LayerEncodeArgs {
  const void *w;
  const long long *perm;
  int n4, n8, n16, K;
  uint8_t *codes, *scales, *fp8;
  float *fp8_scale;
  __nv_bfloat16 *fp16;
  float *tops;  // [block of the first pass]: largest NVFP4 block scale, largest magnitude of the FP8 group
  int segs;     // pieces of a row
  int len;      // of 32 vectors each, in a piece
  float *global_scale;
  int32_t *inv_perm;
  int *bad_index;  // pinned host word: 1 once an entry of a permutation was out of range
};
// channel of permuted row r, or -1
__device__ __forceinline__ long long source_row(const LayerEncodeArgs &a, int r) {
  const int n = a.n4 + a.n8 + a.n16;
  long long s = a.perm[r];
  if (s < 0) s += n;  // indices from the end, as in tensor indexing
  return s < 0 || s >= n ? -1 : s;
}

// Pieces of rows as a warp takes them: up to P vectors per lane, those of the next piece loaded before
// the present one is encoded.  A piece costs about 70 instructions besides its vectors (which row it is,
// the channel, addresses); with pieces of five vectors of halves instead of two, and the registers for
// them (three blocks to an SM), a 2560 x 9728 layer takes 23.7 instead of 26.1 us, 13840 x 3884 39.1 instead of
// 47.3.  Six or more, or four with the registers of four blocks, are slower; floats take twice the
// registers.  FULL: pieces have P (a row's last one maybe fewer), else a.len: asking costs 1.5 us of the 39.
constexpr int kShortPiece = 2, kLongPiece = 5;
template <int P>
constexpr int kBlocks = P > kShortPiece ? 3 : 4;
template <typename T, int P, bool FULL>
struct Piece {
  Vec8<T> q[P];
  int r, v0;  // row inside the pass's rows, first vector of this lane
  static __device__ __forceinline__ bool has(const LayerEncodeArgs &a, int u) { return FULL || u < a.len; }
  __device__ __forceinline__ void load(const LayerEncodeArgs &a, int t, int first_row, int lane) {
    r = t / a.segs;
    v0 = (t - r * a.segs) * 32 * a.len + lane;
    const T *row = static_cast<const T *>(a.w) + max(source_row(a, first_row + r), 0ll) * a.K;
#pragma unroll
    for (int u = 0; u < P; ++u)
      if (has(a, u) && v0 + 32 * u < (a.K >> 3)) q[u].load(row + 8ll * (v0 + 32 * u));
  }
};

// First pass over all rows: NVFP4 codes, the FP8 group's magnitude, FP16 rows, inverse permutation.
// Bound by instruction issue for f16 input (88 warp instructions per 256 values with long pieces, 113 with short
// ones; 60 % of the issue slots, 34 % of the DRAM rate): magnitudes and block scales come from packed halves
// and without a division, pieces go round a single wave of blocks.  (A warp per row left the last rows to a wave of their own and
// waited three times per row.)
template <typename T, int P, bool FULL>
__global__ void __launch_bounds__(256, kBlocks<P>) encode_layer_kernel(LayerEncodeArgs a) {
  pdl_launch_dependents();  // (launched in stream order: everything before it is complete)
  __shared__ float red[2][8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int K = a.K, nvec = K >> 3, tasks = (a.n4 + a.n8 + a.n16) * a.segs, stride = (gridDim.x * blockDim.x) >> 5;
  float top = 0.f, amax = 0.f, none = 0.f;
  Piece<T, P, FULL> cur, next;
  int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (t < tasks) cur.load(a, t, 0, lane);
  for (; t < tasks; t += stride) {
    if (t + stride < tasks) next.load(a, t + stride, 0, lane);
    const int r = cur.r, v0 = cur.v0;
    if (v0 == 0) {
      const long long s = source_row(a, r);
      if (s >= 0) a.inv_perm[s] = r;
      else *static_cast<volatile int *>(a.bad_index) = 1;  // (the row has channel 0's values)
    }
#pragma unroll
    for (int u = 0; u < P; ++u) {
      const int i = v0 + 32 * u;
      if (!cur.has(a, u) || i - lane >= nvec) break;  // the whole warp is past the row
      if (r < a.n4) {
        encode_vec_fp4<T, false>(cur.q[u], i < nvec, i, a.codes + 1ll * r * (K >> 1), a.scales + 1ll * r * (K >> 4), top, none);
      } else if (i >= nvec) {
      } else if (r < a.n4 + a.n8) {
        amax = fmaxf(amax, cur.q[u].amax());
      } else {
        // stored as the bf16 rounding of the f16 value
        float v[8];
        cur.q[u].get(v);
        uint4 o;
        uint32_t *ow = reinterpret_cast<uint32_t *>(&o);
#pragma unroll
        for (int e = 0; e < 4; ++e)
          ow[e] = pack_y2(__half2float(__float2half_rn(v[2 * e])), __half2float(__float2half_rn(v[2 * e + 1])), 1);
        reinterpret_cast<uint4 *>(a.fp16 + 1ll * (r - a.n4 - a.n8) * K)[i] = o;
      }
    }
    cur = next;
  }
  top = warp_max(top);
  amax = warp_max(amax);
  if (lane == 0) {
    red[0][warp] = top;
    red[1][warp] = amax;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    float m = 0.f;
    for (int i = 0; i < 8; ++i) m = fmaxf(m, red[threadIdx.x][i]);
    a.tops[2 * blockIdx.x + threadIdx.x] = m;
  }
}

// Second pass: the FP8 rows (their scale is known now; they mostly come out of L2).  Channels that the
// permutation does not name get row 0 as their inverse: whoever reads it finds an index in range.
template <typename T, int P, bool FULL>
__global__ void __launch_bounds__(256, kBlocks<P>) encode_layer_fp8_kernel(LayerEncodeArgs a, int blocks) {
  __shared__ float red[2][8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nvec = a.K >> 3, tasks = a.n8 * a.segs, stride = (gridDim.x * blockDim.x) >> 5;
  Piece<T, P, FULL> cur, next;
  int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (t < tasks) cur.load(a, t, a.n4, lane);  // (inputs of both passes)
  pdl_wait();
  pdl_launch_dependents();
  float m[2] = {0.f, 0.f};
  for (int i = threadIdx.x; i < blocks; i += blockDim.x) {
    const float2 p = __ldcg(reinterpret_cast<const float2 *>(a.tops) + i);
    m[0] = fmaxf(m[0], p.x);
    m[1] = fmaxf(m[1], p.y);
  }
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    m[j] = warp_max(m[j]);
    if (lane == 0) red[j][warp] = m[j];
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 2; ++j)
    for (int i = 0; i < 8; ++i) m[j] = fmaxf(m[j], red[j][i]);
  if (blockIdx.x == 0 && threadIdx.x == 0 && a.n4) a.global_scale[0] = m[0] == 0.f ? 1.f : m[0];
  const float scale = fp8_scale(m[1]), inv = fp8_inverse(scale);
  for (; t < tasks; t += stride) {
    if (t + stride < tasks) next.load(a, t + stride, a.n4, lane);
#pragma unroll
    for (int u = 0; u < P; ++u) {
      const int i = cur.v0 + 32 * u;
      if (!cur.has(a, u) || i >= nvec) break;
      float v[8];
      cur.q[u].get(v);
      reinterpret_cast<uint2 *>(a.fp8 + 1ll * cur.r * a.K)[i] = quotients_e4m3(v, scale, inv);
    }
    if (cur.v0 == 0) a.fp8_scale[cur.r] = scale;
    cur = next;
  }
  const int n = a.n4 + a.n8 + a.n16;
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    const int r = __ldcg(a.inv_perm + j);
    if (r < 0 || r >= n || source_row(a, r) != j) a.inv_perm[j] = 0;
  }
}

int grid_for_rows(int n) {
  const long long want = (1ll * n + 7) / 8;  // 8 warps per block
  const long long cap = 1ll * sm_count() * 8;
  return static_cast<int>(want < cap ? (want > 0 ? want : 1) : cap);
}

// most blocks of 256 threads that run at once
template <typename K>
int one_wave(K kernel) {
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 256, 0) != cudaSuccess || per_sm < 1) per_sm = 1;
  return std::min(sm_count() * per_sm, RDQ_QUANTIZE_LAYER_SCRATCH / 2);
}

// The pinned word of LayerEncodeArgs::bad_index, one per process.
std::atomic<int *> bad_index{nullptr};
int bad_index_word(int **out) {
  static std::mutex mu;
  std::lock_guard<std::mutex> lock(mu);
  int *word = bad_index.load();
  if (word == nullptr) {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;  // the allocation is no part of a capture
    RDQ_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
    void *p = nullptr;
    const cudaError_t e = cudaHostAlloc(&p, sizeof(int), cudaHostAllocPortable | cudaHostAllocMapped);
    cudaThreadExchangeStreamCaptureMode(&mode);
    RDQ_CUDA(e);
    word = static_cast<int *>(p);
    *word = 0;
    bad_index.store(word);
  }
  *out = word;
  return RDQ_OK;
}

template <typename T, int P, bool FULL>
int run_pieces(const LayerEncodeArgs &a, cudaStream_t stream) {
  static const int most1 = one_wave(encode_layer_kernel<T, P, FULL>), most2 = one_wave(encode_layer_fp8_kernel<T, P, FULL>);
  const int blocks = static_cast<int>(std::min<long long>(most1, (1ll * (a.n4 + a.n8 + a.n16) * a.segs + 7) / 8));
  encode_layer_kernel<T, P, FULL><<<blocks, 256, 0, stream>>>(a);
  RDQ_CUDA(cudaGetLastError());
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(std::max(1ll, std::min<long long>(most2, (1ll * a.n8 * a.segs + 7) / 8))));
  cfg.blockDim = dim3(256);
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  RDQ_CUDA(cudaLaunchKernelEx(&cfg, encode_layer_fp8_kernel<T, P, FULL>, a, blocks));
  return RDQ_OK;
}
// Pieces of a row have equal length: the warps take them in turn, so that a short one would always meet the
// same warps.  Long ones where every warp of the chip gets at least ten vectors -- 2560 x 2560 (seven) takes 11.9 us
// with short pieces and 12.3 with long ones, 4096 x 2560 (twelve) 15.0 and 14.3 -- and a row is longer than a
// short piece: otherwise both have the same pieces, and the short kernel has the fourth block on an SM
// (512 x 60000 33.1 us, 38.2 with the long one's three; 64 x 200000 70.3, 82.6; but 768 x 40000 36.0, 31.9).
template <typename T>
int run_layer(LayerEncodeArgs a, cudaStream_t stream) {
  const int chunks = ((a.K >> 3) + 31) / 32;
  const long long vectors = 1ll * (a.n4 + a.n8 + a.n16) * chunks, warps = 8ll * sm_count() * kBlocks<kLongPiece>;
  const bool lengthy = sizeof(T) == 2 && chunks > kShortPiece && vectors >= 10 * warps;
  const RowPieces cut = row_pieces(a.K, lengthy ? kLongPiece : kShortPiece);
  a.segs = cut.pieces;
  a.len = cut.len;
  if (!lengthy) return run_pieces<T, kShortPiece, true>(a, stream);  // (of one vector, if there is but one)
  if constexpr (sizeof(T) == 2)
    return a.len == kLongPiece ? run_pieces<T, kLongPiece, true>(a, stream) : run_pieces<T, kLongPiece, false>(a, stream);
}

template <typename T>
void run_nvfp4(const void *w, int n, int K, uint8_t *codes, uint8_t *scales, float *row_sqerr, float *max_scale, cudaStream_t stream) {
  const T *p = static_cast<const T *>(w);
  const int grid = grid_for_rows(n);
  if (row_sqerr) quantize_nvfp4_kernel<T, true><<<grid, 256, 0, stream>>>(p, n, K, codes, scales, row_sqerr, max_scale);
  else quantize_nvfp4_kernel<T, false><<<grid, 256, 0, stream>>>(p, n, K, codes, scales, nullptr, max_scale);
}
template <typename T>
void run_fp8(const void *w, int n, int K, uint8_t *out, float *scale_out, float *row_sqerr, float *absmax, cudaStream_t stream) {
  const T *p = static_cast<const T *>(w);
  const int grid = grid_for_rows(n);
  absmax_kernel<T><<<grid, 256, 0, stream>>>(p, n, K, absmax);
  if (row_sqerr) quantize_fp8_kernel<T, true><<<grid, 256, 0, stream>>>(p, n, K, absmax, out, scale_out, row_sqerr);
  else quantize_fp8_kernel<T, false><<<grid, 256, 0, stream>>>(p, n, K, absmax, out, scale_out, nullptr);
}

}  // namespace

int launch_quantize_nvfp4(const void *w, bool w_is_f32, int n, int K, uint8_t *codes, uint8_t *scales, float *row_sqerr,
                          float *max_scale, cudaStream_t stream) {
  if (max_scale) RDQ_CUDA(cudaMemsetAsync(max_scale, 0, sizeof(float), stream));
  if (w_is_f32) run_nvfp4<float>(w, n, K, codes, scales, row_sqerr, max_scale, stream);
  else run_nvfp4<__half>(w, n, K, codes, scales, row_sqerr, max_scale, stream);
  RDQ_CUDA(cudaGetLastError());
  return RDQ_OK;
}

int launch_quantize_fp8(const void *w, bool w_is_f32, int n, int K, uint8_t *out, float *scale_out, float *row_sqerr,
                        float *absmax_scratch, cudaStream_t stream) {
  RDQ_CUDA(cudaMemsetAsync(absmax_scratch, 0, sizeof(float), stream));
  if (w_is_f32) run_fp8<float>(w, n, K, out, scale_out, row_sqerr, absmax_scratch, stream);
  else run_fp8<__half>(w, n, K, out, scale_out, row_sqerr, absmax_scratch, stream);
  RDQ_CUDA(cudaGetLastError());
  return RDQ_OK;
}

int quantize_error() {
  volatile int *const word = bad_index.load();
  if (word == nullptr || *word == 0) return RDQ_OK;
  *word = 0;
  RDQ_REQUIRE(false, RDQ_E_INVALID, "rdq_quantize_layer: a permutation given to an earlier call had an entry out of range; "
              "its tensors are invalid");
  return RDQ_OK;
}

}  // namespace rdq

using namespace rdq;

extern "C" int rdq_quantize_layer(const void *w, int w_is_f32, const long long *perm, int n_fp4, int n_fp8, int n_fp16, int K,
                                  void *codes, void *scales, float *global_scale, void *fp8, float *fp8_scale, void *fp16_bf16,
                                  int32_t *inv_perm, float *scratch, void *stream_) {
  RDQ_REQUIRE(n_fp4 >= 0 && n_fp8 >= 0 && n_fp16 >= 0 && K > 0 && K % 16 == 0, RDQ_E_INVALID,
              "rdq_quantize_layer needs K a positive multiple of 16 (n=%d/%d/%d K=%d)", n_fp4, n_fp8, n_fp16, K);
  if (n_fp4 + n_fp8 + n_fp16 == 0) return RDQ_OK;
  RDQ_REQUIRE(w && perm && inv_perm && scratch && (!n_fp4 || (codes && scales && global_scale)) && (!n_fp8 || (fp8 && fp8_scale)) &&
                  (!n_fp16 || fp16_bf16),
              RDQ_E_INVALID, "null pointer");
  RDQ_REQUIRE(aligned16(w) && aligned16(codes) && aligned16(fp8) && aligned16(fp16_bf16), RDQ_E_INVALID,
              "w and the outputs must be 16-byte aligned");
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  LayerEncodeArgs a;
  int rc = bad_index_word(&a.bad_index);
  if (rc == RDQ_OK) rc = quantize_error();
  if (rc != RDQ_OK) return rc;
  a.w = w;
  a.perm = perm;
  a.n4 = n_fp4;
  a.n8 = n_fp8;
  a.n16 = n_fp16;
  a.K = K;
  a.codes = static_cast<uint8_t *>(codes);
  a.scales = static_cast<uint8_t *>(scales);
  a.fp8 = static_cast<uint8_t *>(fp8);
  a.fp8_scale = fp8_scale;
  a.fp16 = static_cast<__nv_bfloat16 *>(fp16_bf16);
  a.tops = scratch;
  a.global_scale = global_scale;
  a.inv_perm = inv_perm;
  return w_is_f32 ? run_layer<float>(a, stream) : run_layer<__half>(a, stream);
}

extern "C" int rdq_quantize_status(void *stream) {
  RDQ_CUDA(cudaStreamSynchronize(static_cast<cudaStream_t>(stream)));
  return quantize_error();
}
