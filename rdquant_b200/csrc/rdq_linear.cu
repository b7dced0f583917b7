// The operator behind one call: picks the kernel by the number of activation rows and by the
// layouts the layer carries, and converts bf16 activations where the kernel does not do it itself.
//
// Reference behaviour replaced: the dispatch of FusedMixedLinear.forward
// (rdquant/inference.py:689-708) with its x.half() / y.to(x.dtype) conversions (:696, :707).
#include "rdq_kernels.cuh"

namespace rdq {

namespace {

// HBM-bound: reads and writes 2 bytes per element.
__global__ void __launch_bounds__(256) cast_rows_kernel(const uint4 *__restrict__ x, uint4 *__restrict__ out, long long nvec) {
  pdl_wait();
  pdl_launch_dependents();
  const long long stride = 1ll * gridDim.x * blockDim.x;
  for (long long i = 1ll * blockIdx.x * blockDim.x + threadIdx.x; i < nvec; i += 4 * stride) {
    uint4 v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (i + q * stride < nvec) v[q] = x[i + q * stride];
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (i + q * stride < nvec)
        out[i + q * stride] =
            make_uint4(bf16x2_to_f16x2(v[q].x), bf16x2_to_f16x2(v[q].y), bf16x2_to_f16x2(v[q].z), bf16x2_to_f16x2(v[q].w));
  }
}
__global__ void __launch_bounds__(256) cast_elems_kernel(const __nv_bfloat16 *__restrict__ x, __half *__restrict__ out,
                                                         long long count) {
  pdl_wait();
  pdl_launch_dependents();
  for (long long i = 1ll * blockIdx.x * blockDim.x + threadIdx.x; i < count; i += 1ll * gridDim.x * blockDim.x)
    out[i] = __float2half_rn(__bfloat162float(x[i]));
}

enum class Path { kGemvTiled, kGemvGeneric, kStream, kGemm, kPanelsTiled, kPanelsGeneric };

bool has_row_major(const rdq_layer &l) {
  return (l.n_fp4 == 0 || l.w_fp4) && (l.n_fp8 == 0 || l.w_fp8) && (l.n_fp16 == 0 || l.w_fp16);
}

// Fewest rows for which the streaming GEMM is taken instead of the decode GEMV.  The GEMV slows with the rows
// (its conversions and activation reads grow with them, above 8 rows it halves its rate), the streaming GEMM hardly
// does.  Calls one after another, GEMV / streaming GEMM in us, without RDQ_GEMV_PDL and with it:
//   36 MB (19456 x 2560)  8 rows 11.1 / 14.5, 14.8 / 13.9     9 rows 24.1 / 14.5, 22.2 / 14.0
//   40 MB (13440 x 4096)  4 rows 10.9 / 14.8, 13.5 / 14.0     8 rows 16.3 / 14.8, 17.4 / 14.2
//   48 MB (8192 x 8192)   2 rows 11.9 / 15.7, 15.8 / 14.8     4 rows 18.3 / 16.0, 19.9 / 15.0
//   97 MB (16384 x 8192)  1 row  19.6 / 22.8, 27.8 / 21.7     4 rows 31.5 / 23.2, 36.5 / 22.1
// The row-major GEMV of layers without a tiled layout starts at 1.9 us where the streaming GEMM takes 6 to 8 (2 MB,
// 3001 x 1024: 2.6 / 6.3 us at one row).  With leave to read weights early or without, f16 rows:
//   12 MB (2001 x 8192)   1 row 10.0 / 10.8    8 rows 10.2 / 10.8    16 rows 11.2 / 10.8
//   15 MB (5001 x 4096)   1 row 10.6 / 10.5    8 rows 11.4 / 10.5    16 rows 12.7 / 10.5
//   19 MB (3072 x 8576)   1 row 11.5 / 12.1    8 rows 12.0 / 12.1    16 rows 13.0 / 12.2
//   22 MB (12001 x 2560)  1 row 11.9 / 10.2    8 rows 12.7 / 10.2    16 rows 14.3 / 10.3
// It keeps up to eight rows up to 22 MB, more of them up to 12.  bf16 rows, which the GEMV rounds itself and the GEMM has
// rounded by a launch before it, stay up to 24 and 18 MB (3341 x 9216, 22 MB, 8 rows 13.2 / 14.5; 5309 x 3520, 14 MB, 9 rows
// 12.1 / 13.1).  The streaming GEMM's narrow copies of block scales (8 bytes where K is no multiple of 256, 4 where it is
// none of 128) keep few rows with the GEMV up to 40 MB, bf16 rows and K of no multiple of 128, unless K is below 2048: time of the GEMM over
// the GEMV's at four rows, f16 and bf16, 26 MB (3659 x 9664) 1.06, 1.40; 40 MB (4677 x 11712) 1.14, 1.50; 26 MB (12227 x 2944) 0.95,
// 1.21; but 30 MB (8613 x 4864) 0.75, 0.97 and 36 MB (33535 x 1472) 0.82, 0.96.  Nor do 9 to 16 f16 rows gain by
// it up to 18 MB where the GEMV's blocks are one wave of two to an SM (4027 x 5504 1.25 at nine, 2813 x 8768 1.06; but with fewer
// or more of them 1671 x 12480 0.89, 5309 x 3520 0.88, 10415 x 2112 0.79).
// Seven and eight rows that the GEMV does not keep in shared memory go to the streaming GEMM from 28 MB on where its
// tiles are whole and its copies wide, or K is below 8000: 37 MB (3584 x 14336) 15.5 / 13.3 us, 38 MB (4096 x 12288) 16.5 / 12.1,
// 30 MB (12672 x 3328) 0.83 of the time, 26 MB (5120 x 7168) 1.1; but 37 MB (3072 x 16000) 14.9 / 16.1, with bf16 rows
// 17.6 / 22.4, and 35 MB (4224 x 11264, cut tiles) with bf16 rows 16.5 / 18.0.  Of 38 layers between 28 and 40 MB 8 % less time,
// at worst 10 % more (bf16 rows, 7040 x 5760); decode steps of eight
// sequences and four blocks, 3328 wide 295 / 272, 3584 wide 313 / 283, but 25 MB (3072 x 11648) cost 2 % there.  Not
// fewer rows: a step whose norms still run inside the GEMV lost 5 % to a streaming down projection in between (3584
// wide, 6 sequences 320 / 337).
int stream_from(const rdq_layer &l, int x_type) {
  const double bytes = l.n_fp4 * (l.K * 0.5625) + l.n_fp8 * (l.K + 4.0) + l.n_fp16 * (l.K * 2.0);
  const bool wide = l.K % 256 == 0;
  if (!l.w_tiled) {
    const bool bf16 = x_type == RDQ_BF16;
    const double few = wide || l.K < 2048 || (!bf16 && l.K % 128 == 0) ? (bf16 ? 24e6 : 22e6) : 40e6;
    if (bytes > few) return 1;
    const int N = l.n_fp4 + l.n_fp8 + l.n_fp16;
    const bool one_wave = N > 16 * 148 && N <= 32 * 148;  // of the GEMV's blocks, two to an SM
    return bytes > (bf16 || (!wide && one_wave) ? 18e6 : 12e6) ? 9 : RDQ_MAX_GEMV_M + 1;
  }
  if (bytes > 40e6) return bytes > 80e6 ? 1 : 3;
  if (bytes <= 28e6 || tiled_stages_x(8, l.K)) return 9;
  if (l.K >= 8000 && (!wide || gemm_stream_uses_words(l.n_fp4, l.n_fp8, l.n_fp16, 8, l.K))) return 9;
  return tiled_stages_x(7, l.K) ? 8 : 7;
}

// Few rows: the decode GEMV (tiled layout, else the any-shape kernel), or the streaming GEMM from
// stream_from() on.  More: the streaming GEMM or the one over decoded weights, which read the
// row-major tensors by TMA (K a multiple of 64 / 16); what they cannot take runs as 16-row panels of
// the decode kernel.
//
// The streaming GEMM converts the weights once more per 128 rows, the other GEMM decodes them once.
// Estimates in microseconds, fitted to both kernels at 16 numbers of rows between 65 and 2048, f16 and
// bf16, on 13 layers (channels x K: 6144, 19456, 4096, 9728 and 1024 x 2560, 2560 x 4096, 2560 x 9728,
// 4096 x 3072, 16384 and 8192 x 8192, 1024 x 16384, 1024 and 11392 x 1024): off by 8 and 7 % on average, by
// up to 40 % on the smallest.  With the present kernels, choosing by them costs 0.3 % on average over the faster
// one on these layers (above 512 rows without 16384 x 8192, where the power cap decides), 31 % at worst (1024 x 16384
// at 2048 f16 rows, 17 % at 1536), elsewhere up to 12 %; on 3584 x 2048, 13824 x 3584, 5120 x 5120, 3072 x 12288
// and 2048 x 6144 0.2 %, 10 % at worst.  (With up to 64 rows the streaming GEMM was always faster.)
// Where the streaming GEMM's tiles are whole, up to 256 rows, its own estimate takes the place of this fit, and the rounding
// launch of bf16 rows counts what 100 layers lost by it (median 3.0 us; with 1.8 1152 -> 9600 at 230 rows, 18.3 us decoded first, took 20.7).
bool stream_beats_dense(const rdq_layer &l, int M, int x_type) {
  if (M <= 64) return true;
  if (M > 2048) return false;
  const int N = l.n_fp4 + l.n_fp8 + l.n_fp16;
  const double weights = 1e-6 * N * l.K;
  const double cast = x_type == RDQ_BF16 ? 1.8 : 0.0;  // the other GEMM's decoding launch rounds bf16 rows along the way
  const double whole = M <= 256 ? gemm_stream_estimate(l.n_fp4, l.n_fp8, l.n_fp16, M, l.K) : 0.0;
  if (whole > 0.0) return (x_type == RDQ_BF16 ? 3.0 : 0.0) + whole < gemm_dense_estimate(M, N, l.K);
  return cast + 15.6 + 1.57e-3 * M * weights < gemm_dense_estimate(M, N, l.K);
}

Path path_of(const rdq_layer &l, int M, int x_type) {
  const bool can_stream = gemm_stream_takes(l.K) && has_row_major(l) && (l.perm || !l.inv_perm);
  if (can_stream && M >= stream_from(l, x_type) && (!gemm_dense_takes(l.K) || stream_beats_dense(l, M, x_type))) return Path::kStream;
  if (M <= RDQ_MAX_GEMV_M) return l.w_tiled ? Path::kGemvTiled : Path::kGemvGeneric;
  if (gemm_dense_takes(l.K) && has_row_major(l)) return Path::kGemm;
  return l.w_tiled ? Path::kPanelsTiled : Path::kPanelsGeneric;
}

// true when the kernel of this path rounds bf16 rows itself
bool takes_bf16(const rdq_layer &l, Path p, int M) {
  return p == Path::kGemvGeneric || p == Path::kPanelsGeneric || (p == Path::kGemvTiled && tiled_stages_x(M, l.K));
}

size_t align256(size_t v) { return (v + 255) & ~static_cast<size_t>(255); }

struct Need {
  size_t cast = 0, gemm = 0;
};
Need need_of(const rdq_layer &l, Path p, int M, int x_type) {
  Need n;
  if (x_type == RDQ_BF16 && !takes_bf16(l, p, M)) n.cast = align256(2ull * M * l.K);
  if (p == Path::kStream) n.gemm = gemm_stream_workspace(l.n_fp4, l.n_fp8, l.n_fp16, M, l.K);
  if (p == Path::kGemm) n.gemm = gemm_workspace_bytes(M, l.n_fp4 + l.n_fp8 + l.n_fp16, l.K);
  return n;
}

bool uses_words(const rdq_layer &l, Path p, int M) {
  return p == Path::kStream && gemm_stream_uses_words(l.n_fp4, l.n_fp8, l.n_fp16, M, l.K);
}

int run_gemv(const rdq_layer &l, bool tiled, const void *x, int x_bf16, int M, const void *bias, void *y, int y_bf16, bool pdl,
             cudaStream_t stream) {
  if (tiled) {
    GemvTiledArgs a;
    a.x = x;
    a.x_bf16 = x_bf16;
    a.y_bf16 = y_bf16;
    a.M = M;
    a.tiled = static_cast<const uint8_t *>(l.w_tiled);
    a.s8 = l.w_fp8_scales;
    a.global4 = l.w_fp4_global_scale;
    a.perm = l.perm;
    a.bias = static_cast<const __half *>(bias);
    a.y = y;
    a.n4 = l.n_fp4;
    a.n8 = l.n_fp8;
    a.n16 = l.n_fp16;
    a.K = l.K;
    a.workspace = static_cast<float *>(l.gemv_ws);
    a.flags = l.gemv_counters;
    return launch_gemv_tiled(a, pdl, stream);
  }
  GemvArgs a;
  a.x = static_cast<const __half *>(x);
  a.M = M;
  a.w4 = static_cast<const uint8_t *>(l.w_fp4);
  a.s4 = static_cast<const uint8_t *>(l.w_fp4_scales);
  a.global4 = l.w_fp4_global_scale;
  a.w8 = static_cast<const uint8_t *>(l.w_fp8);
  a.s8 = l.w_fp8_scales;
  a.w16 = static_cast<const __half *>(l.w_fp16);
  a.perm = l.perm;
  a.bias = static_cast<const __half *>(bias);
  a.y = y;
  a.n4 = l.n_fp4;
  a.n8 = l.n_fp8;
  a.n16 = l.n_fp16;
  a.K = l.K;
  a.x_bf16 = x_bf16;
  a.y_bf16 = y_bf16;
  return launch_gemv_generic(a, stream);
}

// What the kernels rely on, for every layout that the layer carries: the entry points of the single
// kernels check the same.
int check_layouts(const rdq_layer &l) {
  RDQ_REQUIRE(l.n_fp4 >= 0 && l.n_fp8 >= 0 && l.n_fp16 >= 0 && l.K > 0, RDQ_E_INVALID, "bad layer shape");
  RDQ_REQUIRE(l.w_tiled || has_row_major(l), RDQ_E_INVALID, "the layer has neither the tiled nor the row-major tensors");
  if (has_row_major(l)) {
    const int rc = check_layer(l.w_fp4, l.w_fp4_scales, l.w_fp8, l.w_fp8_scales, l.w_fp16, l.n_fp4, l.n_fp8, l.n_fp16, l.K);
    if (rc != RDQ_OK) return rc;
  }
  if (l.w_tiled) {
    RDQ_REQUIRE(l.n_fp4 + l.n_fp8 + l.n_fp16 == 0 || tiled_supported(l.n_fp4, l.n_fp8, l.n_fp16, l.K), RDQ_E_UNSUPPORTED,
                "shape has no tiled layout (K=%d, n=%d/%d/%d)", l.K, l.n_fp4, l.n_fp8, l.n_fp16);
    RDQ_REQUIRE(aligned16(l.w_tiled), RDQ_E_INVALID, "w_tiled must be 16-byte aligned");
    RDQ_REQUIRE(l.n_fp8 == 0 || l.w_fp8_scales, RDQ_E_INVALID, "w_fp8_scales must not be null when n_fp8 > 0");
  }
  return RDQ_OK;
}

}  // namespace

int launch_cast_rows(const void *x_bf16, void *x_f16, long long count, bool pdl, cudaStream_t stream) {
  if (count == 0) return RDQ_OK;
  const bool vec = count % 8 == 0 && aligned16(x_bf16) && aligned16(x_f16);
  const long long per = vec ? 8 * 256 : 256;
  long long blocks = (count + per - 1) / per;
  const long long cap = 8ll * sm_count();
  if (blocks > cap) blocks = cap;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(blocks));
  cfg.blockDim = dim3(256);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = pdl ? 1 : 0;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (vec) {
    RDQ_CUDA(cudaLaunchKernelEx(&cfg, cast_rows_kernel, static_cast<const uint4 *>(x_bf16), static_cast<uint4 *>(x_f16),
                                count / 8));
  } else {
    RDQ_CUDA(cudaLaunchKernelEx(&cfg, cast_elems_kernel, static_cast<const __nv_bfloat16 *>(x_bf16),
                                static_cast<__half *>(x_f16), count));
  }
  return RDQ_OK;
}

}  // namespace rdq

using namespace rdq;

extern "C" {

int rdq_linear_workspace_size(const rdq_layer *layer, int M, int x_type, size_t *bytes) {
  RDQ_REQUIRE(layer && bytes && M >= 0 && (x_type == RDQ_F16 || x_type == RDQ_BF16), RDQ_E_INVALID,
              "bad arguments to rdq_linear_workspace_size");
  const int rc = check_layouts(*layer);
  if (rc != RDQ_OK) return rc;
  *bytes = 0;
  if (M == 0 || layer->n_fp4 + layer->n_fp8 + layer->n_fp16 == 0) return RDQ_OK;
  const Need n = need_of(*layer, path_of(*layer, M, x_type), M, x_type);
  *bytes = n.cast + n.gemm;
  return RDQ_OK;
}

int rdq_linear_uses_words(const rdq_layer *layer, int M, int x_type) {
  if (!layer || M <= 0 || (x_type != RDQ_F16 && x_type != RDQ_BF16) || check_layouts(*layer) != RDQ_OK ||
      layer->n_fp4 + layer->n_fp8 + layer->n_fp16 == 0)
    return 0;
  return uses_words(*layer, path_of(*layer, M, x_type), M) ? 1 : 0;
}

int rdq_linear(const rdq_layer *layer, const void *x, int x_type, int M, const void *bias, void *y, void *workspace,
               size_t workspace_bytes, int flags, void *stream) {
  return rdq_linear_words(layer, x, x_type, M, bias, y, workspace, workspace_bytes, layer ? layer->gemv_counters : nullptr,
                          flags & ~RDQ_LINEAR_FRESH, stream);
}

int rdq_linear_words(const rdq_layer *layer, const void *x, int x_type, int M, const void *bias, void *y, void *workspace,
                     size_t workspace_bytes, int32_t *words, int flags, void *stream_) {
  RDQ_REQUIRE(layer != nullptr && M >= 0 && (x_type == RDQ_F16 || x_type == RDQ_BF16), RDQ_E_INVALID, "bad arguments to rdq_linear");
  const rdq_layer &l = *layer;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  int rc = quantize_error();
  if (rc == RDQ_OK) rc = check_layouts(l);
  if (rc != RDQ_OK) return rc;
  const int N = l.n_fp4 + l.n_fp8 + l.n_fp16;
  if (M == 0 || N == 0) return RDQ_OK;
  const Path p = path_of(l, M, x_type);
  RDQ_REQUIRE(x && y, RDQ_E_INVALID, "x and y must not be null");
  const Need need = need_of(l, p, M, x_type);
  RDQ_REQUIRE(need.cast + need.gemm <= workspace_bytes && (need.cast + need.gemm == 0 || (workspace && aligned16(workspace))),
              RDQ_E_INVALID, "rdq_linear needs %zu bytes of 16-byte aligned workspace for this shape", need.cast + need.gemm);
  const int bf16 = x_type == RDQ_BF16 ? 1 : 0;
  bool pdl = (flags & RDQ_GEMV_PDL) != 0;
  if (words && (flags & RDQ_LINEAR_FRESH)) RDQ_CUDA(cudaMemsetAsync(words, 0, RDQ_LINEAR_WORDS * sizeof(int32_t), stream));
  RDQ_REQUIRE(words || !uses_words(l, p, M), RDQ_E_INVALID, "words must not be null");
  const void *xh = x;
  int x_bf16 = bf16;
  // (the decoded-once GEMM's first launch rounds the rows itself)
  const bool cast_inside = need.cast && p == Path::kGemm && aligned16(x);
  if (cast_inside) {
    xh = workspace;
  } else if (need.cast) {
    rc = launch_cast_rows(x, workspace, 1ll * M * l.K, pdl, stream);
    if (rc != RDQ_OK) return rc;
    xh = workspace;
    x_bf16 = 0;
    pdl = true;  // the kernel before is ours and waits for its own predecessor
  }
  void *rest = static_cast<char *>(workspace) + need.cast;
  switch (p) {
    case Path::kGemvTiled:
    case Path::kGemvGeneric:
    case Path::kPanelsTiled:
    case Path::kPanelsGeneric: {
      const bool tiled = p == Path::kGemvTiled || p == Path::kPanelsTiled;
      RDQ_REQUIRE(!tiled || (l.gemv_ws && l.gemv_counters), RDQ_E_INVALID, "the tiled GEMV needs its scratch pair");
      RDQ_REQUIRE(aligned16(xh) || (!tiled && l.K % 16 != 0), RDQ_E_INVALID, "x must be 16-byte aligned");
      for (int r0 = 0; r0 < M; r0 += RDQ_MAX_GEMV_M) {
        const int m = M - r0 < RDQ_MAX_GEMV_M ? M - r0 : RDQ_MAX_GEMV_M;
        rc = run_gemv(l, tiled, static_cast<const char *>(xh) + 2ll * r0 * l.K, x_bf16, m, bias,
                                static_cast<char *>(y) + 2ll * r0 * N, bf16, pdl, stream);
        if (rc != RDQ_OK) return rc;
      }
      return RDQ_OK;
    }
    case Path::kStream:
    case Path::kGemm:
      break;
  }
  RDQ_REQUIRE(aligned16(xh) && aligned16(y), RDQ_E_INVALID, "x and y must be 16-byte aligned");
  GemmArgs a;
  a.x = static_cast<const __half *>(xh);
  a.M = M;
  a.w4 = static_cast<const uint8_t *>(l.w_fp4);
  a.s4 = static_cast<const uint8_t *>(l.w_fp4_scales);
  a.global4 = l.w_fp4_global_scale;
  a.w8 = static_cast<const uint8_t *>(l.w_fp8);
  a.s8 = l.w_fp8_scales;
  a.w16 = static_cast<const __half *>(l.w_fp16);
  a.inv_perm = l.inv_perm;
  a.perm = l.perm;
  a.counters = words;
  a.bias = static_cast<const __half *>(bias);
  a.y = y;
  a.n4 = l.n_fp4;
  a.n8 = l.n_fp8;
  a.n16 = l.n_fp16;
  a.K = l.K;
  a.y_bf16 = bf16;
  if (cast_inside) a.x_bf16 = x;
  if (p == Path::kStream) return launch_gemm_stream(a, rest, need.gemm, pdl, stream);
  return launch_gemm(a, rest, need.gemm, stream);
}

}  // extern "C"
