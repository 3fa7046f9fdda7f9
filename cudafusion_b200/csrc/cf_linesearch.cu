// cf_linesearch.cu — the GN step's acceptance on the device: the increment's
// validation statistics, the scaled and clamped trial increment and the
// correspondence RMSE.
//
// DynamicFusionPipeline runs these on the host after downloading the
// increment (include/fusion_app.h:409-490) and, for each of the line
// search's ten trials, every correspondence record (correspondence_rmse,
// :1331-1350; 23 MB at 640x480).  Here they are reductions over device
// arrays that stay on the stream, so the whole line search is enqueued
// without a host round trip (cf_line_search in cf_api.cu drives it).
#include <cmath>

#include "cf_device.cuh"
#include "cf_internal.h"

namespace cf {

namespace {

constexpr int kLsThreads = 256;

__device__ __forceinline__ float ls_norm3(float a, float b, float c) {
  return __fsqrt_rn(fmaf(c, c, fmaf(b, b, __fmul_rn(a, a))));
}

// Per node rn = |dx[0:3]|, tn = |dx[3:6]|; sums in FP64 and maxima of the raw
// and of the scaled-and-clamped values (fusion_app.h:434-458); a non-finite
// rn or tn clears out->finite.  Block partials then atomics: maxima of
// non-negative floats compare as their bit patterns.
__global__ void __launch_bounds__(kLsThreads) update_stats_kernel(const float* dx, int N,
                                                                   float update_scale, float max_rot,
                                                                   float max_trans, double* __restrict__ sums,
                                                                   unsigned* __restrict__ maxima,
                                                                   int* __restrict__ finite) {
  after_previous();
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  float m[4] = {0.f, 0.f, 0.f, 0.f};
  bool fin = true;
  for (int i = blockIdx.x * kLsThreads + threadIdx.x; i < N; i += gridDim.x * kLsThreads) {
    const float* d = dx + 6 * (size_t)i;
    const float rn = ls_norm3(d[0], d[1], d[2]), tn = ls_norm3(d[3], d[4], d[5]);
    fin = fin && isfinite(rn) && isfinite(tn);
    float er = __fmul_rn(update_scale, rn), et = __fmul_rn(update_scale, tn);
    if (max_rot > 0.f) er = fminf(er, max_rot);
    if (max_trans > 0.f) et = fminf(et, max_trans);
    s[0] += rn;
    s[1] += tn;
    s[2] += er;
    s[3] += et;
    m[0] = fmaxf(m[0], rn);
    m[1] = fmaxf(m[1], tn);
    m[2] = fmaxf(m[2], er);
    m[3] = fmaxf(m[3], et);
  }
  __shared__ double rs[4][kLsThreads / 32];
  __shared__ float rm[4][kLsThreads / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    double v = s[c];
    float mv = m[c];
    for (int o = 16; o; o >>= 1) {
      v += __shfl_xor_sync(0xffffffffu, v, o);
      mv = fmaxf(mv, __shfl_xor_sync(0xffffffffu, mv, o));
    }
    if (lane == 0) {
      rs[c][w] = v;
      rm[c][w] = mv;
    }
  }
  if (!__all_sync(0xffffffffu, fin) && lane == 0) atomicExch(finite, 0);
  __syncthreads();
  if (threadIdx.x < 4) {
    double v = 0.0;
    float mv = 0.f;
    for (int j = 0; j < kLsThreads / 32; ++j) {
      v += rs[threadIdx.x][j];
      mv = fmaxf(mv, rm[threadIdx.x][j]);
    }
    atomicAdd(sums + threadIdx.x, v);
    atomicMax(maxima + threadIdx.x, __float_as_uint(mv));
  }
}

// upload_scaled_delta_x (fusion_app.h:1352-1375): per node rs = max_rot / rn
// when rn exceeds a positive max_rot (else 1), ts likewise, then
// dx[k] * (rs * scale) and dx[k] * (ts * scale).
__device__ __forceinline__ void ls_scale(const float* d, float max_rot, float max_trans, float scale,
                                         float (&o)[6]) {
  const float rn = ls_norm3(d[0], d[1], d[2]), tn = ls_norm3(d[3], d[4], d[5]);
  float rs = 1.f, ts = 1.f;
  if (max_rot > 0.f && rn > max_rot) rs = __fdiv_rn(max_rot, rn);
  if (max_trans > 0.f && tn > max_trans) ts = __fdiv_rn(max_trans, tn);
  const float fr = __fmul_rn(rs, scale), ft = __fmul_rn(ts, scale);
#pragma unroll
  for (int k = 0; k < 3; ++k) o[k] = __fmul_rn(d[k], fr);
#pragma unroll
  for (int k = 3; k < 6; ++k) o[k] = __fmul_rn(d[k], ft);
}
__global__ void scale_delta_kernel(const float* dx, int N, float max_rot, float max_trans, float scale,
                                   float* __restrict__ out) {
  after_previous();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  float o[6];
  ls_scale(dx + 6 * (size_t)i, max_rot, max_trans, scale, o);
#pragma unroll
  for (int k = 0; k < 6; ++k) out[6 * (size_t)i + k] = o[k];
}

// A trial's transforms: the saved ones with the scaled increment applied (the
// restore, scale_delta and apply_twist of the host flow, in one launch: the
// copy and two launches took 8 us a trial, this 3).
__global__ void trial_transforms_kernel(const cf_dual_quat* saved, const float* dx, int N,
                                        float max_rot, float max_trans, float scale, float* __restrict__ delta,
                                        cf_dual_quat* __restrict__ T) {
  after_previous();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  float o[6];
  ls_scale(dx + 6 * (size_t)i, max_rot, max_trans, scale, o);
#pragma unroll
  for (int k = 0; k < 6; ++k) delta[6 * (size_t)i + k] = o[k];
  const float* q = reinterpret_cast<const float*>(saved + i);  // (the caller's scratch: whole floats)
  DQ t;
  t.r = make_float4(q[0], q[1], q[2], q[3]);
  t.d = make_float4(q[4], q[5], q[6], q[7]);
  store_dq(T + i, twist_update(t, o, max_rot, max_trans, 1.f));
}

// v[0] + v[1] + ... in order, by one thread, the reads ahead of the adds.
__device__ __forceinline__ double ls_sum(const double* v, int n) {
  double s = 0.0;
  int j = 0;
  for (; j + 16 <= n; j += 16) {
    double x[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) x[k] = v[j + k];
#pragma unroll
    for (int k = 0; k < 16; ++k) s += x[k];
  }
  for (; j < n; ++j) s += v[j];
  return s;
}

// correspondence_rmse's sums (fusion_app.h:1336-1347): block b sums the
// records of its fixed slice in index order per thread and then in thread
// order; rmse_final_kernel adds the blocks in block order.  Deterministic.
__global__ void __launch_bounds__(kLsThreads) rmse_partial_kernel(const cf_correspondence* corrs, int M,
                                                                   double* __restrict__ part) {
  after_previous();
  const int per = (M + gridDim.x - 1) / gridDim.x;
  const int lo = blockIdx.x * per, hi = min(M, lo + per);
  double s = 0.0, ws = 0.0;
  for (int c = lo + threadIdx.x; c < hi; c += kLsThreads) {
    const cf_correspondence& r = corrs[c];
    if (!r.valid || !(r.weight > 0.f)) continue;
    const float dx = __fsub_rn(r.src.x, r.dst.x), dy = __fsub_rn(r.src.y, r.dst.y), dz = __fsub_rn(r.src.z, r.dst.z);
    const double e = fma((double)r.normal.z, (double)dz, fma((double)r.normal.y, (double)dy,
                                                              (double)r.normal.x * (double)dx));
    const double w = (double)fmaxf(0.f, r.weight);
    s = fma(w * e, e, s);
    ws += w;
  }
  __shared__ double sh[2][kLsThreads];
  sh[0][threadIdx.x] = s;
  sh[1][threadIdx.x] = ws;
  __syncthreads();
  if (threadIdx.x < 2) part[2 * blockIdx.x + threadIdx.x] = ls_sum(sh[threadIdx.x], kLsThreads);
}

// The block sums in block order, for the whole CTA (256 threads).
__device__ __forceinline__ void ls_total(const double* part, double (&out)[2]) {
  __shared__ double sh[2][CF_RMSE_BLOCKS];
  __shared__ double tot[2];
  for (int b = threadIdx.x; b < 2 * CF_RMSE_BLOCKS; b += blockDim.x) sh[b & 1][b >> 1] = part[b];
  __syncthreads();
  if (threadIdx.x < 2) tot[threadIdx.x] = ls_sum(sh[threadIdx.x], CF_RMSE_BLOCKS);
  __syncthreads();
  out[0] = tot[0];
  out[1] = tot[1];
}
__global__ void __launch_bounds__(256) rmse_final_kernel(const double* part, double* __restrict__ out) {
  after_previous();
  double t[2];
  ls_total(part, t);
  if (threadIdx.x < 2) out[threadIdx.x] = t[threadIdx.x];
}

// After a trial's records: its sums (every CTA adds the block sums itself;
// slot: sum, wsum and valid count) and whether the trial is the best so far
// under the line search's acceptance rule (fusion_app.h:575-582, the host's
// arithmetic: IEEE double quotient and square root), chaining the best RMSE from
// best_in (or best0) to best_out; a kept trial's index goes to *kept and its
// outputs (4-byte words) are copied aside, so that the accepted trial need not
// be predicted and searched again.
__global__ void __launch_bounds__(256) ls_keep_kernel(LsKeepArgs a) {
  after_previous();
  double t[2];
  ls_total(a.part, t);
  const int valid = *a.valid;
  const double rmse = t[1] > 0.0 ? sqrt(t[0] / t[1]) : (double)INFINITY;
  const double best = a.best_in ? *a.best_in : a.best0;
  const bool take = valid >= a.min_valid && valid >= a.need && isfinite(rmse) && rmse < best;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.slot[0] = t[0];
    a.slot[1] = t[1];
    a.slot[2] = (double)valid;
    *a.best_out = take ? rmse : best;
    if (take) *a.kept = a.trial;
  }
  if (!take) return;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (int b = 0; b < a.nbuf; ++b) {
    const int* src = a.src[b];
    int* dst = a.dst[b];
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < a.words[b]; i += stride) dst[i] = src[i];
  }
}

}  // namespace

cudaError_t launch_ls_keep(const LsKeepArgs& a, cudaStream_t s) {
  launch_next(ls_keep_kernel, 296, 256, 0, s, a);
  return cudaGetLastError();
}

cudaError_t launch_update_stats(const float* dx, int N, float update_scale, float max_rot, float max_trans,
                                double* sums, unsigned* maxima, int* finite, cudaStream_t s) {
  if (N <= 0) return cudaSuccess;
  int blocks = (N + kLsThreads - 1) / kLsThreads;
  if (blocks > 148) blocks = 148;
  launch_next(update_stats_kernel, blocks, kLsThreads, 0, s, dx, N, update_scale, max_rot, max_trans, sums, maxima,
              finite);
  return cudaGetLastError();
}

cudaError_t launch_scale_delta(const float* dx, int N, float max_rot, float max_trans, float scale, float* out,
                               cudaStream_t s) {
  if (N <= 0) return cudaSuccess;
  launch_next(scale_delta_kernel, (N + 255) / 256, 256, 0, s, dx, N, max_rot, max_trans, scale, out);
  return cudaGetLastError();
}

cudaError_t launch_trial_transforms(const cf_dual_quat* saved, const float* dx, int N, float max_rot, float max_trans,
                                    float scale, float* delta, cf_dual_quat* T, cudaStream_t s) {
  if (N <= 0) return cudaSuccess;
  launch_next(trial_transforms_kernel, (N + 63) / 64, 64, 0, s, saved, dx, N, max_rot, max_trans, scale, delta, T);
  return cudaGetLastError();
}

cudaError_t launch_corr_rmse(const cf_correspondence* corrs, int M, double* partials, double* out, cudaStream_t s) {
  launch_next(rmse_partial_kernel, CF_RMSE_BLOCKS, kLsThreads, 0, s, corrs, M, partials);
  if (out) launch_next(rmse_final_kernel, 1, 256, 0, s, partials, out);
  return cudaGetLastError();
}

}  // namespace cf
