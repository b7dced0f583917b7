// Internal launch interfaces shared by the C-ABI translation unit and the
// kernel translation units.
#pragma once

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <mutex>

#include "rdq_common.cuh"

namespace rdq {

constexpr int kMaxPeers = 8;  // GPUs of one node a peer-mode launch can write to

// Arguments of the decode GEMV kernels (permuted-row tensors, see rdq_b200.h).
struct GemvArgs {
  const __half *x;
  int M;
  const uint8_t *w4;
  const uint8_t *s4;
  float global4;
  const uint8_t *w8;
  const float *s8;
  const __half *w16;
  const int32_t *perm;
  const __half *bias;
  void *y;
  int n4, n8, n16, K;
  int x_bf16 = 0;  // x is bf16: rounded to f16 as it is read
  int y_bf16 = 0;  // y is bf16 instead of f16
  int ask_ahead = 0;  // (set by the launcher) ask the weights into L2 ahead of the grid-dependency wait
};

struct GemmArgs {
  const void *x_bf16 = nullptr;  // bf16 rows to be rounded into x first (launch_gemm with a workspace)
  const __half *x;
  int M;
  const uint8_t *w4;
  const uint8_t *s4;
  float global4;
  const uint8_t *w8;
  const float *s8;
  const __half *w16;
  const int32_t *inv_perm;
  const int32_t *perm = nullptr;  // inverse of inv_perm
  int32_t *counters = nullptr;    // one zero word per SM, zero again when the launch ends
  const __half *bias;
  void *y;
  int n4, n8, n16, K;
  int y_bf16 = 0;  // y is bf16 instead of f16
  int test_timeout = 0;  // self-test: CTA (0,0,0) ends with a wait that runs out
};

// RDQ_OK, or an error when sizes, pointers or alignments are not what the row-major kernels rely on (rdq_api.cu)
int check_layer(const void *w_fp4, const void *w_fp4_scales, const void *w_fp8, const float *w_fp8_scales, const void *w_fp16,
                int n4, int n8, int n16, int K);

int launch_dequant(const void *w_fp4, const void *w_fp4_scales, float global4, const void *w_fp8,
                   const float *w_fp8_scales, const void *w_fp16, int fp16_is_bf16,
                   const int32_t *inv_perm, void *w_out, int out_is_f32, int n4, int n8, int n16,
                   int K, cudaStream_t stream);

// bf16 -> f16, count % 8 == 0, both 16-byte aligned
int launch_cast_rows(const void *x_bf16, void *x_f16, long long count, bool pdl, cudaStream_t stream);

int launch_gemv_generic(const GemvArgs &a, cudaStream_t stream);

// ---- tiled layout (rdq_gemv_tiled.cu)
struct GemvTiledArgs {
  const void *x;
  int x_bf16 = 0;  // x is bf16: the kernel rounds the rows to f16 as it stages them in shared memory
  int y_bf16 = 0;  // y is bf16 instead of f16
  int M;
  const uint8_t *tiled;
  const float *s8;
  float global4;
  const int32_t *perm;
  const __half *bias;
  void *y;
  int n4, n8, n16, K;
  float *workspace;
  int32_t *flags;
  int test_timeout = 0;  // RDQ_GEMV_TEST_TIMEOUT
  int opens = 0, beside = 0;  // RDQ_GEMV_OPENS, RDQ_GEMV_BESIDE
  // peer mode (see TiledArgs): destinations, this rank's flag word on every GPU, local state
  int n_dst = 0;
  __half *dst[kMaxPeers] = {};
  int32_t *peer_flag[kMaxPeers] = {};
  int32_t *peer_state = nullptr;
  // activation prologue (see TiledArgs)
  int xop = 0;
  const __half *x_aux = nullptr;
  const __half *x_weight = nullptr;
  __half *x_out = nullptr;
  float x_eps = 0.f;
};
int tiled_chunk_k(int K);
// true when the launcher keeps the activation rows of this shape in shared memory (a requirement
// of the activation prologue)
bool tiled_stages_x(int M, int K);
bool tiled_supported(int n4, int n8, int n16, int K);
size_t tiled_bytes(int n4, int n8, int n16, int K);
int launch_repack(const void *w_fp4, const void *w_fp4_scales, const void *w_fp8, const void *w_fp16,
                  void *tiled_out, int n4, int n8, int n16, int K, cudaStream_t stream);
void gemv_tiled_scratch(size_t *workspace_bytes, size_t *flag_bytes);
int launch_gemv_tiled(const GemvTiledArgs &a, bool pdl, cudaStream_t stream);
// same kernel with the scratch in a library-owned device array (no allocation anywhere)
int gemv_tiled_noalloc(const GemvTiledArgs &a, bool pdl, cudaStream_t stream);
// synchronise `stream`, report (and optionally clear) the kernel's status word; null scratch
// pointers select the library array of the no-allocation entry point
int gemv_tiled_status(float *workspace, int32_t *flags, bool reset, cudaStream_t stream);
int launch_peer_gather(const __half *buffer, const long long *index, __half *y, long long count, const int32_t *flags,
                       int world, const int32_t *sent_state, int32_t *status, int wait_ms, bool pdl, cudaStream_t stream);

int launch_gemm(const GemmArgs &a, void *workspace, size_t workspace_bytes, cudaStream_t stream);
// synchronise `stream`, report (and optionally clear) the GEMM's per-device status word
int gemm_status(bool reset, cudaStream_t stream);
int gemm_status_ptr(int **out);
int gemm_test_timeout();
// self-test switch: 1: launches made while it is on end with a wait that runs out, 2: CTAs that share a
// tile leave at once when they would have to wait
void gemm_set_test_timeout(int mode);
size_t gemm_workspace_bytes(int M, int N, int K);
bool gemm_better_without_scratch(int M, int N, int K);
// weight-streaming GEMM (rdq_gemm_stream.cu)
bool gemm_stream_takes(int K);
size_t gemm_stream_workspace(int n4, int n8, int n16, int M, int K);
double gemm_stream_estimate(int n4, int n8, int n16, int M, int K);  // microseconds where its tiles are whole, else 0
bool gemm_stream_uses_words(int n4, int n8, int n16, int M, int K);  // GemmArgs::counters
int launch_gemm_stream(const GemmArgs &a, void *workspace, size_t workspace_bytes, bool pdl, cudaStream_t stream);
// GEMM over weights decoded once per call (rdq_gemm_dense.cu)
bool gemm_dense_takes(int K);
size_t gemm_dense_workspace(int M, int N, int K);
double gemm_dense_estimate(int M, int N, int K);  // microseconds, decoding and product
int launch_gemm_dense(const GemmArgs &a, void *workspace, size_t workspace_bytes, cudaStream_t stream);

// staging copy by kernel (rdq_stage.cu)
int launch_stage_copy(void *dst, const void *src, size_t bytes, int *state, int *flag, cudaStream_t stream);

// decode-step glue (rdq_glue.cu)
int launch_add_rmsnorm(__half *x, const __half *delta, const __half *w, __half *out, int B, int H, float eps, bool pdl,
                       cudaStream_t stream);
int launch_qk_rope_cache(const __half *qkv, const __half *qn, const __half *kn, const __half *cos_t, const __half *sin_t,
                         const long long *pos, __half *q_out, __half *k_cache, __half *v_cache, int B, int nq, int nkv,
                         int dh, int S, float eps, bool pdl, cudaStream_t stream);
// The GEMVs of a decode step and the kernels between them are launched with one CTA per SM and at
// least this much dynamic shared memory, so that an SM has room for two of their CTAs whichever they
// are.  With a third place on some SMs (kernels of 60 KB, GEMVs of 93 KB) two CTAs of a launch landed
// there, a later GEMV found 107 of 148 SMs and its doubled CTAs took 6 us longer than the others.
constexpr int kSlotSmem = 100 * 1024;
cudaError_t pin_slot(const void *fn, int smem);
int attn_chunk();
// q/k norm + rotary + cache write + attention + merge of the splits in one launch
int rope_attn_splits(int B, int nkv, int S);
size_t rope_attn_scratch_bytes(int B, int nq, int nkv, int dh, int S);
int launch_rope_attn(const __half *qkv, const __half *qn, const __half *kn, const __half *cos_t, const __half *sin_t,
                     const long long *pos, __half *k_cache, __half *v_cache, void *scratch, __half *out, int B, int nq,
                     int nkv, int dh, int S, float scale, float eps, bool pdl, cudaStream_t stream);
int launch_attn_decode(const __half *q, const __half *k_cache, const __half *v_cache, const long long *pos, float *scratch,
                       __half *out, int B, int nq, int nkv, int dh, int S, float scale, bool pdl, cudaStream_t stream);
int launch_silu_mul(const __half *gu, __half *out, int B, int F, bool pdl, cudaStream_t stream);

// A row of K values cut into `pieces` of equal length -- `len` turns of a warp whose lanes hold eight values each,
// at most `most` -- of which only the last can be shorter.
struct RowPieces {
  int pieces, len;
};
inline RowPieces row_pieces(int K, int most) {
  const int turns = (K / 8 + 31) / 32, pieces = turns > most ? (turns + most - 1) / most : 1;
  return {pieces, (turns + pieces - 1) / pieces};
}

// encoders (rdq_quantize.cu)
int launch_quantize_nvfp4(const void *w, bool w_is_f32, int n, int K, uint8_t *codes, uint8_t *scales, float *row_sqerr,
                          float *max_scale, cudaStream_t stream);
// RDQ_OK, or the error of an encoder launch that found a permutation entry out of range (reported once; looks at
// a word of host memory)
int quantize_error();
int launch_quantize_fp8(const void *w, bool w_is_f32, int n, int K, uint8_t *out, float *scale_out, float *row_sqerr,
                        float *absmax_scratch, cudaStream_t stream);

}  // namespace rdq
