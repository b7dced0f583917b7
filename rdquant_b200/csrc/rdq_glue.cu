// Decode-step glue between the mixed-precision linears of a transformer block: residual add +
// RMSNorm, per-head q/k RMSNorm + rotary embedding + KV-cache write, single-token attention over
// the cache, SiLU x mul.  The reference leaves these to the HuggingFace model code around its
// linear modules (rdquant/inference.py:689-708 is the module boundary; its end-to-end harness
// benchmarks/bench_e2e.py:103-155 captures that code in a CUDA graph); here they are small
// HBM/latency-bound kernels of their own because, at one token per step, each of the ~20 framework
// kernels between two linears costs more than the linear itself.
//
// Every kernel takes part in programmatic dependent launch the way the decode GEMV does: it reads its
// inputs only after griddepcontrol.wait, and those that keep the one-CTA-per-SM shape (`first`, see
// pdl_wait()) let their successor become resident at once, so that the next GEMV fills its weight rings
// while they run.  All arithmetic is FP32 with one rounding to FP16 per stored value.
#include "rdq_kernels.cuh"

#include <utility>
#include <vector>

namespace rdq {

namespace {

__device__ __forceinline__ float block_sum(float v, float *smem) {
  v = warp_sum(v);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = (blockDim.x + 31) >> 5;
  __syncthreads();  // smem may still be read from a previous call
  if (lane == 0) smem[warp] = v;
  __syncthreads();
  float t = (lane < nw) ? smem[lane] : 0.f;
  return warp_sum(t);
}

// A hint; it takes whole runs of 16 bytes at addresses that are multiples of 16, others go without.
__device__ __forceinline__ void prefetch_l2(const void *p, int bytes) {
  if ((reinterpret_cast<uintptr_t>(p) | static_cast<uintptr_t>(bytes)) & 15) return;
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// ---- x (+= delta); out = rmsnorm(x) * w.  One CTA per row.
// Bound: latency.  The first kNormVecs vectors of a thread (8192 values of a row: more than the models
// this serves have) stay in registers between the sum and the product, and their norm weights are
// loaded beside them: one round trip to memory per row instead of one per vector and pass.  With the
// loads of silu_mul_kernel ahead likewise: 4 blocks of 32 rows x 2560 323.7 -> 318.8 us.
constexpr int kNormVecs = 4;

__global__ void __launch_bounds__(256) add_rmsnorm_kernel(__half *x, const __half *delta, const __half *w, __half *out,
                                                         int B, int H, float eps, bool first) {
  __shared__ float red[32];
  if (first) pdl_launch_dependents();
  if (blockIdx.x == 0 && threadIdx.x == 0) prefetch_l2(w, H * 2);  // a hint while the kernel before runs
  pdl_wait();
  if (!first) pdl_launch_dependents();
  if (static_cast<int>(blockIdx.x) >= B) {  // the grid has a CTA per SM (see linger())
    linger(1500);
    return;
  }
  const int n8 = H / 8, tail = kNormVecs * static_cast<int>(blockDim.x);
  uint4 *xr = reinterpret_cast<uint4 *>(x + 1ll * blockIdx.x * H);
  const uint4 *dr = reinterpret_cast<const uint4 *>(delta ? delta + 1ll * blockIdx.x * H : nullptr);
  const uint4 *w8 = reinterpret_cast<const uint4 *>(w);
  float ss = 0.f;
  auto add_and_sum = [&](uint4 &v, const uint4 &d, int i) {
    __half2 *h = reinterpret_cast<__half2 *>(&v);
    if (dr) {
      const __half2 *dh = reinterpret_cast<const __half2 *>(&d);
#pragma unroll
      for (int j = 0; j < 4; ++j) h[j] = __hadd2(h[j], dh[j]);
      xr[i] = v;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = __half22float2(h[j]);
      ss += f.x * f.x + f.y * f.y;
    }
  };
  uint4 v[kNormVecs], d[kNormVecs], wv[kNormVecs];
#pragma unroll
  for (int u = 0; u < kNormVecs; ++u) {
    const int i = u * blockDim.x + threadIdx.x;
    if (i < n8) {
      v[u] = xr[i];
      if (dr) d[u] = dr[i];
      wv[u] = w8[i];
    }
  }
#pragma unroll
  for (int u = 0; u < kNormVecs; ++u) {
    const int i = u * blockDim.x + threadIdx.x;
    if (i < n8) add_and_sum(v[u], d[u], i);
  }
  for (int i = tail + threadIdx.x; i < n8; i += blockDim.x) {
    uint4 vt = xr[i], dt = make_uint4(0, 0, 0, 0);
    if (dr) dt = dr[i];
    add_and_sum(vt, dt, i);
  }
  ss = block_sum(ss, red);
  const float rs = rsqrtf(ss / H + eps);
  uint4 *orow = reinterpret_cast<uint4 *>(out + 1ll * blockIdx.x * H);
  auto scaled = [&](const uint4 &vv, const uint4 &ww) {
    const __half2 *h = reinterpret_cast<const __half2 *>(&vv);
    const __half2 *wh = reinterpret_cast<const __half2 *>(&ww);
    uint4 o;
    __half2 *oh = reinterpret_cast<__half2 *>(&o);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = __half22float2(h[j]);
      oh[j] = __hmul2(__floats2half2_rn(f.x * rs, f.y * rs), wh[j]);
    }
    return o;
  };
#pragma unroll
  for (int u = 0; u < kNormVecs; ++u) {
    const int i = u * blockDim.x + threadIdx.x;
    if (i < n8) orow[i] = scaled(v[u], wv[u]);
  }
  for (int i = tail + threadIdx.x; i < n8; i += blockDim.x) orow[i] = scaled(xr[i], w8[i]);
}

// ---- per head: (q, k) RMSNorm over head_dim (optional), rotary embedding, q -> q_out, k / v -> cache
// at position *pos.  grid = (nq + 2 nkv, B); one thread per rotary pair (i, i + dh / 2).
__global__ void __launch_bounds__(128) qk_rope_cache_kernel(const __half *qkv, const __half *qn, const __half *kn,
                                                           const __half *cos_t, const __half *sin_t, const long long *pos,
                                                           __half *q_out, __half *k_cache, __half *v_cache, int nq, int nkv,
                                                           int dh, int S, float eps) {
  __shared__ float red[32];
  pdl_wait();
  pdl_launch_dependents();
  const int head = blockIdx.x, b = blockIdx.y, i = threadIdx.x, half = dh >> 1;
  const long long p = *pos;
  const __half *src = qkv + (1ll * b * (nq + 2 * nkv) + head) * dh;
  const float x0 = __half2float(src[i]), x1 = __half2float(src[i + half]);
  if (head >= nq + nkv) {  // v: copy
    __half *dst = v_cache + ((1ll * b * nkv + (head - nq - nkv)) * S + p) * dh;
    dst[i] = src[i];
    dst[i + half] = src[i + half];
    return;
  }
  const bool is_q = head < nq;
  const __half *nw = is_q ? qn : kn;
  float y0 = x0, y1 = x1;
  if (nw) {
    const float ss = block_sum(x0 * x0 + x1 * x1, red);
    const float rs = rsqrtf(ss / dh + eps);
    y0 = __half2float(__hmul(__float2half_rn(x0 * rs), nw[i]));
    y1 = __half2float(__hmul(__float2half_rn(x1 * rs), nw[i + half]));
  }
  const float c0 = __half2float(cos_t[p * dh + i]), s0 = __half2float(sin_t[p * dh + i]);
  const float c1 = __half2float(cos_t[p * dh + i + half]), s1 = __half2float(sin_t[p * dh + i + half]);
  const __half o0 = __float2half_rn(y0 * c0 - y1 * s0), o1 = __float2half_rn(y1 * c1 + y0 * s1);
  __half *dst = is_q ? q_out + (1ll * b * nq + head) * dh : k_cache + ((1ll * b * nkv + (head - nq)) * S + p) * dh;
  dst[i] = o0;
  dst[i + half] = o1;
}

// ---- attention of one new token over the cache, positions 0 .. *pos, split over blockIdx.x.
// grid = (nsplit, nkv, B); warp w serves the query heads kvh * group + w, w + 4, ... of its KV head;
// a lane owns dh / 32 consecutive dimensions.  Partial (max, sum, weighted values) per split go to
// scratch; attn_combine_kernel merges them.
constexpr int kAttnWarps = 4;
constexpr int kMaxDimsPerLane = 8;  // head_dim <= 256

__global__ void __launch_bounds__(kAttnWarps * 32) attn_split_kernel(const __half *q, const __half *k_cache,
                                                                    const __half *v_cache, const long long *pos,
                                                                    float *part, int nq, int nkv, int dh, int S, int chunk,
                                                                    float scale) {
  pdl_wait();
  pdl_launch_dependents();
  const int split = blockIdx.x, kvh = blockIdx.y, b = blockIdx.z;
  const int nsplit = gridDim.x, group = nq / nkv;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int dpl = dh >> 5;  // dims per lane
  const int n = static_cast<int>(*pos) + 1;
  const int p0 = split * chunk, p1 = min(n, p0 + chunk);
  const __half *kb = k_cache + (1ll * b * nkv + kvh) * S * dh + lane * dpl;
  const __half *vb = v_cache + (1ll * b * nkv + kvh) * S * dh + lane * dpl;
  for (int hq = warp; hq < group; hq += kAttnWarps) {
    const int head = kvh * group + hq;
    float qv[kMaxDimsPerLane], acc[kMaxDimsPerLane];
    const __half *qp = q + (1ll * b * nq + head) * dh + lane * dpl;
#pragma unroll
    for (int j = 0; j < kMaxDimsPerLane; ++j) {
      qv[j] = j < dpl ? __half2float(qp[j]) * scale : 0.f;
      acc[j] = 0.f;
    }
    float m = -INFINITY, l = 0.f;
    for (int p = p0; p < p1; ++p) {
      float kf[kMaxDimsPerLane], vf[kMaxDimsPerLane];
      if (dpl == 4) {  // head_dim 128: one 8-byte load per lane and tensor
        const uint2 kr = *reinterpret_cast<const uint2 *>(kb + 1ll * p * dh);
        const uint2 vr = *reinterpret_cast<const uint2 *>(vb + 1ll * p * dh);
        const float2 k01 = __half22float2(*reinterpret_cast<const __half2 *>(&kr.x));
        const float2 k23 = __half22float2(*reinterpret_cast<const __half2 *>(&kr.y));
        const float2 v01 = __half22float2(*reinterpret_cast<const __half2 *>(&vr.x));
        const float2 v23 = __half22float2(*reinterpret_cast<const __half2 *>(&vr.y));
        kf[0] = k01.x; kf[1] = k01.y; kf[2] = k23.x; kf[3] = k23.y;
        vf[0] = v01.x; vf[1] = v01.y; vf[2] = v23.x; vf[3] = v23.y;
      } else {
#pragma unroll
        for (int j = 0; j < kMaxDimsPerLane; ++j) {
          kf[j] = j < dpl ? __half2float(kb[1ll * p * dh + j]) : 0.f;
          vf[j] = j < dpl ? __half2float(vb[1ll * p * dh + j]) : 0.f;
        }
      }
      float s = 0.f;
#pragma unroll
      for (int j = 0; j < kMaxDimsPerLane; ++j)
        if (j < dpl) s += qv[j] * kf[j];
      s = warp_sum(s);
      const float mn = fmaxf(m, s);
      const float corr = __expf(m - mn), w = __expf(s - mn);
      l = l * corr + w;
#pragma unroll
      for (int j = 0; j < kMaxDimsPerLane; ++j)
        if (j < dpl) acc[j] = acc[j] * corr + w * vf[j];
      m = mn;
    }
    float *dst = part + ((1ll * b * nq + head) * nsplit + split) * (dh + 2);
    if (lane == 0) {
      dst[0] = m;
      dst[1] = l;
    }
#pragma unroll
    for (int j = 0; j < kMaxDimsPerLane; ++j)
      if (j < dpl) dst[2 + lane * dpl + j] = acc[j];
  }
}

// grid = (nq, B), one thread per dimension
__global__ void __launch_bounds__(256) attn_combine_kernel(const float *part, __half *out, int nq, int dh, int nsplit) {
  pdl_wait();
  pdl_launch_dependents();
  const int head = blockIdx.x, b = blockIdx.y, d = threadIdx.x;
  const float *src = part + (1ll * b * nq + head) * nsplit * (dh + 2);
  float m = -INFINITY;
  for (int s = 0; s < nsplit; ++s) m = fmaxf(m, src[s * (dh + 2)]);
  float l = 0.f, a = 0.f;
  for (int s = 0; s < nsplit; ++s) {
    const float ms = src[s * (dh + 2)];
    if (ms == -INFINITY) continue;
    const float w = __expf(ms - m);
    l += src[s * (dh + 2) + 1] * w;
    a += src[s * (dh + 2) + 2 + d] * w;
  }
  out[(1ll * b * nq + head) * dh + d] = __float2half_rn(a / l);
}

// ---- out[b, f] = silu(gu[b, f]) * gu[b, F + f]
__global__ void __launch_bounds__(256) silu_mul_kernel(const __half *gu, __half *out, int B, int F, bool first) {
  if (first) pdl_launch_dependents();
  pdl_wait();
  if (!first) pdl_launch_dependents();
  // every CTA takes an equal, contiguous share of the 16-byte vectors, so that (nearly) all SMs
  // work and leave together
  const long long total = 1ll * B * (F / 8);
  const long long per = (total + gridDim.x - 1) / gridDim.x;
  const long long lo = per * blockIdx.x, hi = lo + per < total ? lo + per : total;
  if (lo >= total) {  // the grid has a CTA per SM (see linger())
    linger(1500);
    return;
  }
  // Two vectors per turn, their loads ahead of the arithmetic: at 32 rows of 9728 a share is 263
  // vectors for 256 threads.  Rows by a 32-bit division of the distance from the share's first row.
  const unsigned f8 = static_cast<unsigned>(F / 8), n = static_cast<unsigned>(hi - lo);
  const long long row0 = lo / f8;
  const unsigned off0 = static_cast<unsigned>(lo - row0 * f8);
  for (unsigned i = threadIdx.x; i < n; i += 2 * blockDim.x) {
    uint4 gv[2], uv[2], *dst[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const unsigned e = i + k * blockDim.x;
      if (e < n) {
        const unsigned r = (off0 + e) / f8, j = off0 + e - r * f8;
        const long long b = row0 + r;
        gv[k] = reinterpret_cast<const uint4 *>(gu + 2 * b * F)[j];
        uv[k] = reinterpret_cast<const uint4 *>(gu + 2 * b * F + F)[j];
        dst[k] = reinterpret_cast<uint4 *>(out + b * F) + j;
      }
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      if (i + k * blockDim.x >= n) break;
      const __half2 *gh = reinterpret_cast<const __half2 *>(&gv[k]);
      const __half2 *uh = reinterpret_cast<const __half2 *>(&uv[k]);
      uint4 o;
      __half2 *oh = reinterpret_cast<__half2 *>(&o);
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const float2 a = __half22float2(gh[t]), c = __half22float2(uh[t]);
        // silu in FP32, rounded to FP16 before the product like the framework's two kernels
        const __half2 s = __floats2half2_rn(silu(a.x), silu(a.y));
        oh[t] = __hmul2(s, __floats2half2_rn(c.x, c.y));
      }
      *dst[k] = o;
    }
  }
}

// ---- q/k RMSNorm + rotary embedding + KV-cache write + attention of the new token over the
// cache + merge of the splits, in one launch.
// CTA c is (sequence, KV head) c / nsplit and split c % nsplit, with nsplit = SMs / (sequences x KV
// heads) (at most 16, at least 1); it serves the `group` query heads of its KV head over the cache
// rows [split * chunk, (split + 1) * chunk), chunk = the n = *pos + 1 rows divided by nsplit.
//   1. the four warps normalise and rotate the query heads into shared memory (FP16-rounded, like the
//      stored q of the separate kernel); the warp whose rows include *pos does the same for the new
//      key, takes the new value, and writes both to the cache.
//   2. every warp takes every fourth block of 16 rows through a ring of two blocks of its own
//      (cp.async, rows outside the split zero-filled), so that warps do not wait for one another and
//      a CTA keeps up to eight blocks (70 KB at head_dim 128) in flight.
//   3. tensor-core products (mma.sync m16n8k16, FP32 sums) with cache rows as the row operand and up to
//      eight query heads as columns: S^T = K Q^T, online softmax per block, O^T += V^T P^T.  P, at
//      most 1, goes in as the sum of two FP16 values of 2^15 P: its rounding is 2^-22 of it down to
//      P = 2^-28 and 2^-40 below, less than FP32 sums lose of terms that small next to 1.  (Without the
//      factor weights below 2^-25 were lost: 4 % of the result for 4096 rows of weight 2^-26 whose values
//      are 750 times the others'.)
//   4. the warps' (max, sum, values) are merged in shared memory; with one split that is the result.
//      Else every CTA stores its partial sums in scratch and counts itself, and the CTA that counts last
//      merges the heads of its (sequence, KV head), a warp per head, the loads of all splits in flight, in
//      split order.  Nobody waits, so nothing relies on the CTAs of a launch running at the same time.
//      The words it read and the count go back to zero.
// Under programmatic launch the norm weights, the rotary rows and the cache rows are asked into L2 while
// the kernel before this one runs (a position that is out of date costs no more than the hint).
// Bound: HBM (K and V rows once) for many sequences, latency for one.  The scalar kernel before (a
// lane per row, every query head converting the K rows again) took 44 us for 32 sequences of 700 rows
// (92 MB).
constexpr int kFusedAttnWarps = 4;
constexpr int kFusedAttnThreads = kFusedAttnWarps * 32;
constexpr float kProbScale = 32768.f;
constexpr int kFusedAttnMaxSplit = 16;  // vectors a lane of the merge has in flight

// 16 bytes, or zeros
__device__ __forceinline__ void cp_async16_if(uint32_t dst, const void *src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t &r0, uint32_t &r1, uint32_t &r2, uint32_t &r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t v) {
  uint32_t r;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
  return r;
}

// N consecutive floats (2, 4 or 8, aligned to 8 or 16 bytes) past L1
template <int N>
__device__ __forceinline__ void ldcg_floats(const float *p, float (&v)[N]) {
  if (N == 2) {
    const float2 t = __ldcg(reinterpret_cast<const float2 *>(p));
    v[0] = t.x;
    v[1] = t.y;
  } else {
#pragma unroll
    for (int i = 0; i < N / 4; ++i) {
      const float4 t = __ldcg(reinterpret_cast<const float4 *>(p) + i);
      v[4 * i] = t.x;
      v[4 * i + 1] = t.y;
      v[4 * i + 2] = t.z;
      v[4 * i + 3] = t.w;
    }
  }
}
template <int N>
__device__ __forceinline__ void stcg_floats(float *p, const float (&v)[N]) {
  if (N == 2) {
    __stcg(reinterpret_cast<float2 *>(p), make_float2(v[0], v[1]));
  } else {
#pragma unroll
    for (int i = 0; i < N / 4; ++i)
      __stcg(reinterpret_cast<float4 *>(p) + i, make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]));
  }
}

// NB: blocks of eight query heads per KV head
template <int DH, int NB>
__global__ void __launch_bounds__(kFusedAttnThreads, 2) rope_attn_kernel(
    const __half *qkv, const __half *qn, const __half *kn, const __half *cos_t, const __half *sin_t, const long long *pos,
    __half *k_cache, __half *v_cache, float *part, int *counters, __half *out, int nq, int nkv, int S, float scale, float eps,
    int nsplit, int npair, bool first) {
  constexpr int W = kFusedAttnWarps;
  constexpr int PITCH = 2 * DH + 16;   // row pitch in shared memory (bytes): an odd multiple of 16
  constexpr int BLK = 16 * PITCH;      // 16 rows of K or of V
  constexpr int QP = DH + 8;           // query row pitch (halves)
  constexpr int HALF = DH / 2;
  constexpr int DPL = DH / 32;         // dimensions per lane in the merge of the warps
  constexpr int VPR = DH / 8;          // 16-byte vectors per row
  constexpr int KS = DH / 16;          // k steps of S, row blocks of O
  constexpr int PR = DH + 4;  // a partial: max, sum, two unused, then the DH weighted values (16-byte aligned)
  extern __shared__ __align__(16) uint8_t smem[];
  __half *qs = reinterpret_cast<__half *>(smem + W * 4 * BLK);  // [8 NB][QP]
  float *mrg = reinterpret_cast<float *>(smem);                 // [W][8 NB][PR], over the rings once they are done

  if (first) pdl_launch_dependents();
  // The grid has one CTA per SM (or one per (sequence, KV head) when those outnumber the SMs); CTAs
  // beyond the work linger.
  const int pair = static_cast<int>(blockIdx.x) / nsplit, split = static_cast<int>(blockIdx.x) - pair * nsplit;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3;
  if (tid == 0 && pair < npair) {
    const long long p = *static_cast<const volatile long long *>(pos);
    // (more rows than a quarter of L2 would only displace one another and the next layers' weights)
    if (p >= 0 && p < S && 4ll * npair * p * DH <= (32ll << 20)) {
      const int rows = static_cast<int>(p) / nsplit + 1, r0 = split * rows, r1 = min(static_cast<int>(p), r0 + rows);
      const long long off = (1ll * pair * S + r0) * DH;  // pair = sequence x KV heads + KV head
      if (r0 < r1) {
        prefetch_l2(k_cache + off, (r1 - r0) * DH * 2);
        prefetch_l2(v_cache + off, (r1 - r0) * DH * 2);
      }
      prefetch_l2(cos_t + p * DH, DH * 2);
      prefetch_l2(sin_t + p * DH, DH * 2);
    }
    if (qn) prefetch_l2(qn, DH * 2);
    if (kn) prefetch_l2(kn, DH * 2);
  }
  pdl_wait();
  if (!first) pdl_launch_dependents();
  if (pair >= npair) {
    linger(4000);
    return;
  }
  const int kvh = pair % nkv, b = pair / nkv;
  const int group = nq / nkv;
  // Loads that do not depend on the position go first, so that they share a round trip with it: the
  // raw values of this warp's first query head and the norm weights.
  const __half *row = qkv + 1ll * b * (nq + 2 * nkv) * DH;
  float qx0[HALF / 32], qx1[HALF / 32], qw0[HALF / 32], qw1[HALF / 32];
  auto load_row = [&](const __half *src, float (&x0)[HALF / 32], float (&x1)[HALF / 32]) {
#pragma unroll
    for (int u = 0; u < HALF / 32; ++u) {
      x0[u] = __half2float(src[lane + 32 * u]);
      x1[u] = __half2float(src[lane + 32 * u + HALF]);
    }
  };
  if (warp < group) load_row(row + 1ll * (kvh * group + warp) * DH, qx0, qx1);
  if (qn) load_row(qn, qw0, qw1);
  const long long p_new = *pos;
  const int n = static_cast<int>(p_new) + 1;
  const int chunk = (n + nsplit - 1) / nsplit;
  const int used = (n + chunk - 1) / chunk;
  if (split >= used) {
    linger(4000);
    return;
  }
  const int p0 = split * chunk, p1 = min(n, p0 + chunk);
  const int nblk = (p1 - p0 + 15) >> 4;
  const __half *kb = k_cache + (1ll * b * nkv + kvh) * S * DH;
  const __half *vb = v_cache + (1ll * b * nkv + kvh) * S * DH;
  const uint32_t ring = smem_u32(smem) + warp * 4 * BLK;  // [2 stages][K, V][16][PITCH]

  auto load_block = [&](int i, int st) {
    const int r0 = p0 + 16 * i;
    const uint32_t dst = ring + st * 2 * BLK;
#pragma unroll
    for (int u = 0; u < 16 * VPR / 32; ++u) {
      const int e = u * 32 + lane, r = e / VPR, c = e - r * VPR;
      const bool valid = r0 + r < p1 && r0 + r != p_new;  // the new row is not in the cache yet
      const long long off = valid ? 1ll * (r0 + r) * DH + 8 * c : 0;
      cp_async16_if(dst + r * PITCH + 16 * c, kb + off, valid);
      cp_async16_if(dst + BLK + r * PITCH + 16 * c, vb + off, valid);
    }
  };
  // Small loads first: behind 64 KB of cache rows they would wait for those.
  const __half *cs = cos_t + p_new * DH, *sn = sin_t + p_new * DH;
  float c0[HALF / 32], s0[HALF / 32], c1[HALF / 32], s1[HALF / 32];
  load_row(cs, c0, c1);
  load_row(sn, s0, s1);
  // the warp whose block holds the new row: key and value to the cache now, into the block when it is current
  const int new_blk = p_new >= p0 && p_new < p1 ? static_cast<int>(p_new - p0) >> 4 : -1;
  const bool owns_new = new_blk >= 0 && new_blk % W == warp;
  __half knew0[HALF / 32], knew1[HALF / 32], vnew[DPL];
  float kx0[HALF / 32], kx1[HALF / 32], kw0[HALF / 32], kw1[HALF / 32];
  if (owns_new) {
    const __half *vsrc = row + 1ll * (nq + nkv + kvh) * DH;
    load_row(row + 1ll * (nq + kvh) * DH, kx0, kx1);
    if (kn) load_row(kn, kw0, kw1);
#pragma unroll
    for (int j = 0; j < DPL; ++j) vnew[j] = vsrc[lane + 32 * j];
  }
  if (warp < nblk) load_block(warp, 0);
  cp_async_commit();
  if (warp + W < nblk) load_block(warp + W, 1);
  cp_async_commit();

  // ---- 1. query heads, new key and value
  // RMSNorm over the head (when nw), rotary embedding
  auto norm_rope = [&](const float (&x0)[HALF / 32], const float (&x1)[HALF / 32], bool nw, const float (&w0)[HALF / 32],
                       const float (&w1)[HALF / 32], __half (&o0)[HALF / 32], __half (&o1)[HALF / 32]) {
    float ss = 0.f;
#pragma unroll
    for (int u = 0; u < HALF / 32; ++u) ss += x0[u] * x0[u] + x1[u] * x1[u];
    float rs = 1.f;
    if (nw) rs = rsqrtf(warp_sum(ss) / DH + eps);
#pragma unroll
    for (int u = 0; u < HALF / 32; ++u) {
      float y0 = x0[u], y1 = x1[u];
      if (nw) {
        y0 = __half2float(__hmul(__float2half_rn(x0[u] * rs), __float2half_rn(w0[u])));
        y1 = __half2float(__hmul(__float2half_rn(x1[u] * rs), __float2half_rn(w1[u])));
      }
      o0[u] = __float2half_rn(y0 * c0[u] - y1 * s0[u]);
      o1[u] = __float2half_rn(y1 * c1[u] + y0 * s1[u]);
    }
  };
  for (int hq = warp; hq < 8 * NB; hq += W) {
    __half o0[HALF / 32], o1[HALF / 32];
    if (hq < group) {
      if (hq != warp) load_row(row + 1ll * (kvh * group + hq) * DH, qx0, qx1);
      norm_rope(qx0, qx1, qn != nullptr, qw0, qw1, o0, o1);
    } else {
#pragma unroll
      for (int u = 0; u < HALF / 32; ++u) o0[u] = o1[u] = __float2half_rn(0.f);
    }
#pragma unroll
    for (int u = 0; u < HALF / 32; ++u) {
      qs[hq * QP + lane + 32 * u] = o0[u];
      qs[hq * QP + lane + 32 * u + HALF] = o1[u];
    }
  }
  if (owns_new) {
    norm_rope(kx0, kx1, kn != nullptr, kw0, kw1, knew0, knew1);
    __half *kd = k_cache + ((1ll * b * nkv + kvh) * S + p_new) * DH;
    __half *vd = v_cache + ((1ll * b * nkv + kvh) * S + p_new) * DH;
#pragma unroll
    for (int u = 0; u < HALF / 32; ++u) {
      kd[lane + 32 * u] = knew0[u];
      kd[lane + 32 * u + HALF] = knew1[u];
    }
#pragma unroll
    for (int j = 0; j < DPL; ++j) vd[lane + 32 * j] = vnew[j];
  }
  __syncthreads();  // qs complete

  // ---- 2./3. blocks of 16 rows
  uint32_t qf[NB][KS][2];  // query fragments: head g of the block, dimensions 16 k + 2 t (+ 8)
#pragma unroll
  for (int nb = 0; nb < NB; ++nb)
#pragma unroll
    for (int k = 0; k < KS; ++k) {
      const __half *src = qs + (nb * 8 + g) * QP + 16 * k + 2 * t;
      qf[nb][k][0] = *reinterpret_cast<const uint32_t *>(src);
      qf[nb][k][1] = *reinterpret_cast<const uint32_t *>(src + 8);
    }
  float m_run[NB][2], l_run[NB][2], acc[NB][KS][4];  // heads 2 t, 2 t + 1; acc: dimensions 16 k + g, + 8
#pragma unroll
  for (int nb = 0; nb < NB; ++nb) {
    m_run[nb][0] = m_run[nb][1] = -INFINITY;
    l_run[nb][0] = l_run[nb][1] = 0.f;
#pragma unroll
    for (int k = 0; k < KS; ++k)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[nb][k][j] = 0.f;
  }
  const uint32_t k_lane = ((lane & 7) + ((lane >> 3) & 1) * 8) * PITCH + (lane >> 4) * 16;
  const uint32_t v_lane = BLK + ((lane & 7) + (lane >> 4) * 8) * PITCH + ((lane >> 3) & 1) * 16;
  int st = 0;
  for (int i = warp; i < nblk; i += W, st ^= 1) {
    cp_async_wait<1>();
    const uint32_t blk = ring + st * 2 * BLK;
    if (owns_new && i == new_blk) {
      const int rr = static_cast<int>(p_new - p0) & 15;
      __half *sk = reinterpret_cast<__half *>(smem + warp * 4 * BLK + st * 2 * BLK + rr * PITCH);
      __half *sv = reinterpret_cast<__half *>(smem + warp * 4 * BLK + st * 2 * BLK + BLK + rr * PITCH);
      __syncwarp();  // other lanes' zero fill of this row has landed
#pragma unroll
      for (int u = 0; u < HALF / 32; ++u) {
        sk[lane + 32 * u] = knew0[u];
        sk[lane + 32 * u + HALF] = knew1[u];
      }
#pragma unroll
      for (int j = 0; j < DPL; ++j) sv[lane + 32 * j] = vnew[j];
    }
    __syncwarp();
    float s[NB][4], s_odd[NB][4];  // two chains: a product waits for the one before the last
#pragma unroll
    for (int nb = 0; nb < NB; ++nb)
#pragma unroll
      for (int j = 0; j < 4; ++j) s[nb][j] = s_odd[nb][j] = 0.f;
#pragma unroll
    for (int k = 0; k < KS; ++k) {
      uint32_t a0, a1, a2, a3;
      ldmatrix_x4(blk + k_lane + 32 * k, a0, a1, a2, a3);
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) mma_16816(k & 1 ? s_odd[nb] : s[nb], a0, a1, a2, a3, qf[nb][k][0], qf[nb][k][1]);
    }
#pragma unroll
    for (int nb = 0; nb < NB; ++nb)
#pragma unroll
      for (int j = 0; j < 4; ++j) s[nb][j] += s_odd[nb][j];
    const int rows = p1 - p0 - 16 * i;  // valid rows of the block
    uint32_t ph[NB][2], pl[NB][2];
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      float corr[2], p[4];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float x0 = g < rows ? s[nb][h] * scale : -INFINITY, x1 = g + 8 < rows ? s[nb][2 + h] * scale : -INFINITY;
        float mx = fmaxf(x0, x1);
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float mn = fmaxf(m_run[nb][h], mx);
        corr[h] = __expf(m_run[nb][h] - mn);  // 0 the first time (m_run = -inf, mn finite)
        m_run[nb][h] = mn;
        p[h] = __expf(x0 - mn);
        p[2 + h] = __expf(x1 - mn);
        l_run[nb][h] = l_run[nb][h] * corr[h] + p[h] + p[2 + h];  // per-lane partial sum, reduced at the end
      }
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const float p0 = p[2 * half] * kProbScale, p1 = p[2 * half + 1] * kProbScale;
        const __half2 hi = __floats2half2_rn(p0, p1);
        const float2 hf = __half22float2(hi);
        const __half2 lo = __floats2half2_rn(p0 - hf.x, p1 - hf.y);
        ph[nb][half] = movmatrix_trans(*reinterpret_cast<const uint32_t *>(&hi));
        pl[nb][half] = movmatrix_trans(*reinterpret_cast<const uint32_t *>(&lo));
      }
#pragma unroll
      for (int k = 0; k < KS; ++k) {
        acc[nb][k][0] *= corr[0];
        acc[nb][k][1] *= corr[1];
        acc[nb][k][2] *= corr[0];
        acc[nb][k][3] *= corr[1];
      }
    }
#pragma unroll
    for (int k = 0; k < KS; ++k) {
      uint32_t a0, a1, a2, a3;
      ldmatrix_x4_trans(blk + v_lane + 32 * k, a0, a1, a2, a3);
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) {
        mma_16816(acc[nb][k], a0, a1, a2, a3, pl[nb][0], pl[nb][1]);
        mma_16816(acc[nb][k], a0, a1, a2, a3, ph[nb][0], ph[nb][1]);
      }
    }
    __syncwarp();  // every lane is done with the block before it is refilled
    if (i + 2 * W < nblk) load_block(i + 2 * W, st);
    cp_async_commit();
  }
  cp_async_wait<0>();

  // ---- 4. merge of the warps
  __syncthreads();
#pragma unroll
  for (int nb = 0; nb < NB; ++nb)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float l = l_run[nb][h];
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
      float *dst = mrg + (warp * 8 * NB + nb * 8 + 2 * t + h) * PR;
      if (g == 0) {
        dst[0] = m_run[nb][h];
        dst[1] = l;
      }
#pragma unroll
      for (int k = 0; k < KS; ++k) {
        dst[4 + 16 * k + g] = acc[nb][k][h] * (1.f / kProbScale);
        dst[4 + 16 * k + g + 8] = acc[nb][k][2 + h] * (1.f / kProbScale);
      }
    }
  __syncthreads();
  for (int hq = warp; hq < group; hq += W) {
    float m = -INFINITY, l = 0.f, a[DPL];
#pragma unroll
    for (int w = 0; w < W; ++w) m = fmaxf(m, mrg[(w * 8 * NB + hq) * PR]);
#pragma unroll
    for (int j = 0; j < DPL; ++j) a[j] = 0.f;
#pragma unroll
    for (int w = 0; w < W; ++w) {  // (a warp without rows has max -inf and weight 0; warp 0 always has rows)
      const float *src = mrg + (w * 8 * NB + hq) * PR;
      const float ws = __expf(src[0] - m);
      l += src[1] * ws;
#pragma unroll
      for (int j = 0; j < DPL; ++j) a[j] += ws * src[4 + lane * DPL + j];
    }
    const int head = kvh * group + hq;
    if (used == 1) {
      __half *o = out + (1ll * b * nq + head) * DH + lane * DPL;
      const float inv = 1.f / l;
#pragma unroll
      for (int j = 0; j < DPL; ++j) o[j] = __float2half_rn(a[j] * inv);
    } else {
      float *dst = part + ((1ll * b * nq + head) * nsplit + split) * PR;
      if (lane == 0) __stcg(reinterpret_cast<float2 *>(dst), make_float2(m, l));
      stcg_floats(dst + 4 + lane * DPL, a);
    }
  }
  if (used == 1) return;
  __shared__ int last;
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    last = atomicAdd(&counters[pair], 1) == used - 1;
    __threadfence();
  }
  __syncthreads();
  if (!last) return;
  if (tid == 0) counters[pair] = 0;
  for (int hq = warp; hq < group; hq += W) {
    const int head = kvh * group + hq;
    float *src = part + (1ll * b * nq + head) * nsplit * PR;
    // lane s: the (max, sum) of split s; every lane: its dimensions of all splits
    float2 ml = make_float2(-INFINITY, 0.f);
    if (lane < used) ml = __ldcg(reinterpret_cast<const float2 *>(src + lane * PR));
    float v[kFusedAttnMaxSplit][DPL];
#pragma unroll
    for (int q = 0; q < kFusedAttnMaxSplit; ++q)
      if (q < used) ldcg_floats(src + q * PR + 4 + lane * DPL, v[q]);
    const float m = warp_max(ml.x);
    const float w = lane < used ? __expf(ml.x - m) : 0.f;
    const float inv = 1.f / warp_sum(ml.y * w);
    const float zeros[DPL] = {};
    float a[DPL];
#pragma unroll
    for (int j = 0; j < DPL; ++j) a[j] = 0.f;
#pragma unroll
    for (int q = 0; q < kFusedAttnMaxSplit; ++q) {
      const float ws = __shfl_sync(0xffffffffu, w, q);
      if (q < used) {
#pragma unroll
        for (int j = 0; j < DPL; ++j) a[j] += ws * v[q][j];
        stcg_floats(src + q * PR + 4 + lane * DPL, zeros);
      }
    }
    if (lane < used) *reinterpret_cast<float2 *>(src + lane * PR) = make_float2(0.f, 0.f);
    __half *o = out + (1ll * b * nq + head) * DH + lane * DPL;
#pragma unroll
    for (int j = 0; j < DPL; ++j) o[j] = __float2half_rn(a[j] * inv);
  }
}

// `slot`: the kernel sits between two GEMVs of a decode step: it reserves kSlotSmem of (unused)
// shared memory so that no SM takes two of its CTAs (see pin_slot).
template <typename... Args>
int launch_pdl(void (*kernel)(Args...), dim3 grid, dim3 block, bool slot, bool pdl, cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = slot ? kSlotSmem : 0;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = pdl ? 1 : 0;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (slot) RDQ_CUDA(pin_slot(reinterpret_cast<const void *>(kernel), kSlotSmem));
  RDQ_CUDA(cudaLaunchKernelEx(&cfg, kernel, args...));
  return RDQ_OK;
}

}  // namespace

// An SM cannot change its shared-memory carve-out while a CTA is resident, and the kernels of a
// decode step overlap on every SM: all of them ask for the largest carve-out, like the GEMV.
// `smem` is the dynamic shared memory the kernel will be launched with.  Once per kernel, device
// and size.
cudaError_t pin_slot(const void *fn, int smem) {
  static std::mutex mu;
  static std::vector<std::pair<std::pair<const void *, int>, int>> done;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lock(mu);
  for (const auto &d : done)
    if (d.first.first == fn && d.first.second == dev && d.second >= smem) return cudaSuccess;
  e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
  if (e == cudaSuccess && smem > 48 * 1024) e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e == cudaSuccess) done.push_back({{fn, dev}, smem});
  return e;
}

// Up to eight rows the linears around these kernels are GEMVs, which share an SM by halves (kSlotSmem).
// Above they are streaming GEMMs, which need most of an SM's shared memory: their CTAs load weights
// while a kernel without any runs beside them.
static bool takes_slot(int B) { return B <= 8; }

int launch_add_rmsnorm(__half *x, const __half *delta, const __half *w, __half *out, int B, int H, float eps, bool pdl,
                       cudaStream_t stream) {
  return launch_pdl(add_rmsnorm_kernel, dim3(std::max(B, sm_count())), dim3(256), takes_slot(B), pdl, stream, x, delta, w, out, B, H,
                    eps, takes_slot(B));
}

int launch_qk_rope_cache(const __half *qkv, const __half *qn, const __half *kn, const __half *cos_t, const __half *sin_t,
                         const long long *pos, __half *q_out, __half *k_cache, __half *v_cache, int B, int nq, int nkv,
                         int dh, int S, float eps, bool pdl, cudaStream_t stream) {
  return launch_pdl(qk_rope_cache_kernel, dim3(nq + 2 * nkv, B), dim3(dh / 2), false, pdl, stream, qkv, qn, kn, cos_t, sin_t, pos,
                    q_out, k_cache, v_cache, nq, nkv, dh, S, eps);
}

int attn_chunk() { return 32; }

int launch_attn_decode(const __half *q, const __half *k_cache, const __half *v_cache, const long long *pos, float *scratch,
                       __half *out, int B, int nq, int nkv, int dh, int S, float scale, bool pdl, cudaStream_t stream) {
  const int chunk = attn_chunk();
  const int nsplit = (S + chunk - 1) / chunk;
  int rc = launch_pdl(attn_split_kernel, dim3(nsplit, nkv, B), dim3(kAttnWarps * 32), false, pdl, stream, q, k_cache, v_cache, pos,
                      scratch, nq, nkv, dh, S, chunk, scale);
  if (rc != RDQ_OK) return rc;
  return launch_pdl(attn_combine_kernel, dim3(nq, B), dim3(dh), false, pdl, stream, static_cast<const float *>(scratch), out, nq, dh,
                    nsplit);
}

// Splits of the cache rows per (sequence, KV head): as many as give every SM one CTA.
int rope_attn_splits(int B, int nkv, int S) {
  (void)S;
  return std::min(kFusedAttnMaxSplit, std::max(1, sm_count() / std::max(1, B * nkv)));
}

// The count of each (sequence, KV head) comes first, then the partial sums.
static size_t rope_attn_counter_bytes(int B, int nkv) { return (sizeof(int) * static_cast<size_t>(B) * nkv + 255) / 256 * 256; }

size_t rope_attn_scratch_bytes(int B, int nq, int nkv, int dh, int S) {
  // Sized for every batch up to B (fewer sequences get more splits each), so one buffer serves smaller
  // batches: all of it is zero between calls.
  size_t rows = 0;
  for (int b = 1; b <= B; ++b) rows = std::max(rows, static_cast<size_t>(b) * rope_attn_splits(b, nkv, S));
  return rope_attn_counter_bytes(B, nkv) + sizeof(float) * rows * nq * (dh + 4);
}

int launch_rope_attn(const __half *qkv, const __half *qn, const __half *kn, const __half *cos_t, const __half *sin_t,
                     const long long *pos, __half *k_cache, __half *v_cache, void *scratch, __half *out, int B, int nq,
                     int nkv, int dh, int S, float scale, float eps, bool pdl, cudaStream_t stream) {
  const int nsplit = rope_attn_splits(B, nkv, S);
  int *counters = static_cast<int *>(scratch);
  float *part = reinterpret_cast<float *>(static_cast<char *>(scratch) + rope_attn_counter_bytes(B, nkv));
  const int group = nq / nkv;
  const int nb = group <= 8 ? 1 : 2;
  int smem = kFusedAttnWarps * 4 * 16 * (2 * dh + 16) + 8 * nb * (dh + 8) * 2;
  // two CTAs per SM while that is enough for the grid: with three, 256 CTAs were placed on 86 SMs
  const bool slot = nsplit * nkv * B <= 2 * sm_count();
  if (slot) smem = std::max(smem, kSlotSmem);
  auto launch = [&](auto kernel) -> int {
    cudaLaunchConfig_t cfg = {};
    // one CTA per SM while the (sequence, KV head) pairs fit: like the GEMVs around it
    cfg.gridDim = dim3(std::max(sm_count(), nsplit * nkv * B));
    cfg.blockDim = dim3(kFusedAttnThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = pdl ? 1 : 0;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    RDQ_CUDA(pin_slot(reinterpret_cast<const void *>(kernel), smem));
    RDQ_CUDA(cudaLaunchKernelEx(&cfg, kernel, qkv, qn, kn, cos_t, sin_t, pos, k_cache, v_cache, part, counters, out, nq, nkv, S, scale,
                                eps, nsplit, nkv * B, slot));
    return RDQ_OK;
  };
  switch (dh) {
    case 64: return nb == 1 ? launch(rope_attn_kernel<64, 1>) : launch(rope_attn_kernel<64, 2>);
    case 128: return nb == 1 ? launch(rope_attn_kernel<128, 1>) : launch(rope_attn_kernel<128, 2>);
    case 256: return nb == 1 ? launch(rope_attn_kernel<256, 1>) : launch(rope_attn_kernel<256, 2>);
  }
  RDQ_REQUIRE(false, RDQ_E_UNSUPPORTED, "head_dim must be 64, 128 or 256, got %d", dh);
  return RDQ_OK;
}

int launch_silu_mul(const __half *gu, __half *out, int B, int F, bool pdl, cudaStream_t stream) {
  const long long total = 1ll * B * (F / 8);
  (void)total;
  return launch_pdl(silu_mul_kernel, dim3(sm_count()), dim3(256), takes_slot(B), pdl, stream, gu, out, B, F, takes_slot(B));
}

}  // namespace rdq
