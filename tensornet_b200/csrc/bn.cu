// Global batch-norm statistics on the GPU.
//
// The reference keeps, per feature and in double precision, the running sum, squared sum and
// count with Kahan-compensated adds and a moving-window decay once `max_count` records have been
// seen (core/ps/table/bn_table.cc:65-121); the layer pushes one batch's sums per step and
// normalises with the table's moments (tensornet/layers/normalization_layer.py:129-177), and the
// ranks exchange their increments by RPC (core/kernels/bn_table_ops.cc:86-159,233-299).
//
// Here the table lives in device memory and a training step of the layer is three small kernels
// with no host round trip, so it can sit inside a captured CUDA graph:
//   bn_batch_stats   per-feature sum and squared sum (optionally around a centre) in fp64
//   bn_table_append  fold the batch into the totals, refresh the fp32 moments, re-zero the scratch
//   bn_apply_fwd/bwd normalise with the moments (moments are constants for the backward pass)
//   bn_join_fwd/bwd  the same for [h | x], where h is a tower's padded bf16 output and x fp32, straight into the padded bf16
//                    operand of the next layer and back (the ReLU mask of the tower's output included)
//   bn_join_train    bn_batch_stats, bn_table_append and bn_join_fwd of up to kTrainRows examples in one launch
// and, when the layer is synchronised, every `sync_freq` steps
//   bn_table_sync    cross-GPU exchange of the pending increments by peer loads, bracketed by
//                    bounded flag handshakes.
#include <cuda_bf16.h>
#include "tn_device.cuh"
#include "tn_ops.h"

namespace tn {

namespace {

constexpr int kBnCols = 32;    // columns per CTA
constexpr int kBnRows = 8;     // row lanes per CTA (256 threads)
constexpr int kBnMinRows = 64; // rows per CTA at least

__device__ __forceinline__ float bn_at(const BnInput& in, int r, int c) {
  if (c < in.nh) return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(in.h)[(size_t)r * in.ldh + c]);
  return in.x[(size_t)r * in.ldx + (c - in.nh)];
}

__global__ void __launch_bounds__(kBnCols * kBnRows) bn_batch_stats_kernel(const BnInput in, int B, int C, const float* __restrict__ center,
                                                                          double* batch, int rows_per_cta) {
  pdl_sync();
  __shared__ double s_sum[kBnRows][kBnCols], s_sq[kBnRows][kBnCols];
  const int cl = threadIdx.x % kBnCols, rl = threadIdx.x / kBnCols;
  const int c = blockIdx.x * kBnCols + cl;
  const int r0 = blockIdx.y * rows_per_cta;
  const int r1 = min(B, r0 + rows_per_cta);
  double s = 0.0, q = 0.0;
  if (c < C) {
    const float ctr = center ? center[c] : 0.f;
    for (int r = r0 + rl; r < r1; r += kBnRows) {
      const double v = (double)bn_at(in, r, c);
      const double d = v - (double)ctr;
      s += v;
      q += d * d;
    }
  }
  s_sum[rl][cl] = s;
  s_sq[rl][cl] = q;
  __syncthreads();
  if (rl == 0 && c < C) {
#pragma unroll
    for (int k = 1; k < kBnRows; ++k) { s += s_sum[k][cl]; q += s_sq[k][cl]; }
    atomicAdd(&batch[c], s);
    atomicAdd(&batch[C + c], q);
    if (blockIdx.y == 0) batch[2 * C + c] = (double)B;     // every feature saw B records
  }
}

__device__ __forceinline__ double block_max(double v) {
  __shared__ double s_w[32];
  __shared__ double s_out;
  for (int off = 16; off > 0; off >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, off));
  if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    double w = threadIdx.x < (blockDim.x + 31) / 32 ? s_w[threadIdx.x] : -1.0;
    for (int off = 16; off > 0; off >>= 1) w = fmax(w, __shfl_xor_sync(0xffffffffu, w, off));
    if (threadIdx.x == 0) s_out = w;
  }
  __syncthreads();
  const double r = s_out;
  __syncthreads();
  return r;
}

struct BnTotals { double sum, sum_err, sq, sq_err, count; };
__device__ __forceinline__ BnTotals bn_totals(const BnTableView& t, int c) {
  return {t.total_sum[c], t.total_sum_err[c], t.total_sq[c], t.total_sq_err[c], t.total_count[c]};
}
__device__ __forceinline__ void bn_keep_sums(const BnTableView& t, int c, const BnTotals& a) {
  t.total_sum[c] = a.sum; t.total_sum_err[c] = a.sum_err; t.total_sq[c] = a.sq; t.total_sq_err[c] = a.sq_err;
}

// One Kahan-compensated update of a feature's totals with (as, aq, ac); `decay_k` < 0 selects the plain path.
__device__ __forceinline__ void bn_fold(BnTotals& a, double as, double aq, double ac, double decay_k) {
  if (decay_k >= 0.0) {
    a.sum *= (1.0 - decay_k); as *= decay_k;
    a.sq *= (1.0 - decay_k); aq *= decay_k;
  } else {
    a.count += ac;
  }
  double y = as - a.sum_err, u = a.sum + y;
  a.sum_err = (u - a.sum) - y; a.sum = u;
  y = aq - a.sq_err; u = a.sq + y;
  a.sq_err = (u - a.sq) - y; a.sq = u;
}

__device__ __forceinline__ void bn_moments(const BnTableView& t, const BnTotals& a, float* mean_out, float* var_out) {
  const double n = a.count;
  const bool ok = n != 0.0 && n == n;
  const double mean = ok ? a.sum / n : 0.0;
  *mean_out = (float)mean;
  if (t.pctr) {
    *var_out = (float)a.sq;
  } else {
    const float m = (float)mean, sm = ok ? (float)(a.sq / n) : 0.f;
    *var_out = ok ? fmaxf(sm - m * m, 0.f) : 1.f;     // no record yet: identity scale, the layer's initial moving variance
  }
}

// `acc` = [3][C] sums to fold in.  Decides between plain accumulation and the moving window exactly as the
// host table does: window mode once max(total_count) exceeds max_count, with ratio = max(acc_count) / max(total_count).
// `drop_inc`: nobody is waiting for the pending increments, which go to zero instead.
__device__ void bn_append_block(const BnTableView& t, const double* acc, bool is_local, bool zero_acc, bool drop_inc = false) {
  const int C = t.C;
  double cur = 0.0, am = 0.0;
  for (int c = threadIdx.x; c < C; c += blockDim.x) { cur = fmax(cur, t.total_count[c]); am = fmax(am, acc[2 * C + c]); }
  cur = floor(block_max(cur));
  am = floor(block_max(am));
  const bool window = t.max_count > 0 && cur > (double)t.max_count;
  const double k = window ? (1.0 - t.moment) * (am / cur) : -1.0;
  for (int c = threadIdx.x; c < C; c += blockDim.x) {
    const double as = acc[c], aq = acc[C + c], ac = acc[2 * C + c];
    if (drop_inc) { t.inc[c] = 0.0; t.inc[C + c] = 0.0; t.inc[2 * C + c] = 0.0; }
    else if (is_local) { t.inc[c] += as; t.inc[C + c] += aq; t.inc[2 * C + c] += ac; }
    BnTotals a = bn_totals(t, c);
    bn_fold(a, as, aq, ac, k);
    bn_keep_sums(t, c, a);
    if (!window) t.total_count[c] = a.count;
    bn_moments(t, a, t.mean + c, t.var + c);
    if (zero_acc) { const_cast<double*>(acc)[c] = 0.0; const_cast<double*>(acc)[C + c] = 0.0; const_cast<double*>(acc)[2 * C + c] = 0.0; }
  }
}

__global__ void __launch_bounds__(1024) bn_table_append_kernel(const BnTableView t, double* batch, int drop_inc) {
  pdl_sync();
  bn_append_block(t, batch, true, true, drop_inc != 0);
}

__global__ void __launch_bounds__(1024) bn_table_refresh_moments_kernel(const BnTableView t) {
  for (int c = threadIdx.x; c < t.C; c += blockDim.x) bn_moments(t, bn_totals(t, c), t.mean + c, t.var + c);
}

// Cross-GPU exchange.  One CTA per GPU: (1) tell every peer "my increments are final" and wait for theirs,
// (2) sum the peers' increments with peer loads into `scratch` and fold them in as one non-local append,
// (3) tell every peer "I have read yours" and wait for the same, (4) clear the own increments.
__global__ void __launch_bounds__(1024) bn_table_sync_kernel(const BnTableView t, const BnSyncView s, double* scratch) {
  __shared__ int s_fail;
  const int C = t.C, W = s.world, R = s.rank;
  const unsigned long long epoch = __ldcg(s.epoch) + 1ull;
  if (threadIdx.x == 0) s_fail = 0;
  __syncthreads();
  if (threadIdx.x < W && threadIdx.x != R) {
    const int p = threadIdx.x;
    __threadfence_system();
    st_release_sys_u64(s.sig[p] + R, epoch << 32);
    unsigned long long v;
    if (!wait_flag_ge(s.sig[R] + p, epoch, &v, s.wait_ns, s.status, 61, p)) s_fail = 1;
  }
  __syncthreads();
  if (s_fail) return;
  for (int i = threadIdx.x; i < 3 * C; i += blockDim.x) {
    double a = 0.0;
    for (int k = 1; k < W; ++k) {
      const double* pi = s.inc[(R + k) % W];
      a += __ldcg(&pi[i]);
    }
    scratch[i] = a;
  }
  __syncthreads();
  bn_append_block(t, scratch, false, true);
  __syncthreads();
  if (threadIdx.x < W && threadIdx.x != R) {
    const int p = threadIdx.x;
    st_release_sys_u64(s.sig[p] + kMaxWorld + R, epoch << 32);
    unsigned long long v;
    if (!wait_flag_ge(s.sig[R] + kMaxWorld + p, epoch, &v, s.wait_ns, s.status, 62, p)) s_fail = 1;
  }
  __syncthreads();
  if (s_fail) return;
  for (int i = threadIdx.x; i < 3 * C; i += blockDim.x) t.inc[i] = 0.0;
  if (threadIdx.x == 0) *s.epoch = epoch;
}

__global__ void bn_apply_fwd_kernel(const float* __restrict__ x, int ldx, int B, int C, const float* __restrict__ mean,
                                    const float* __restrict__ var, const float* __restrict__ gamma, const float* __restrict__ beta,
                                    float eps, float* __restrict__ y, int ldy) {
  pdl_sync();
  const long long n = (long long)B * C;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int r = (int)(i / C), c = (int)(i - (long long)r * C);
    float v = (x[(size_t)r * ldx + c] - mean[c]) * rsqrtf(var[c] + eps);
    if (gamma) v *= gamma[c];
    if (beta) v += beta[c];
    y[(size_t)r * ldy + c] = v;
  }
}

// dx = dy * gamma * rsqrt(var + eps); dgamma = sum dy * xhat; dbeta = sum dy (accumulated into gg / gb).
__global__ void __launch_bounds__(kBnCols * kBnRows) bn_apply_bwd_kernel(const float* __restrict__ dy, int ldd, const float* __restrict__ x,
                                                                        int ldx, int B, int C, const float* __restrict__ mean,
                                                                        const float* __restrict__ var, const float* __restrict__ gamma,
                                                                        float eps, float* __restrict__ dx, int ldo, float* gg, float* gb,
                                                                        int rows_per_cta) {
  pdl_sync();
  __shared__ float s_g[kBnRows][kBnCols], s_b[kBnRows][kBnCols];
  const int cl = threadIdx.x % kBnCols, rl = threadIdx.x / kBnCols;
  const int c = blockIdx.x * kBnCols + cl;
  const int r0 = blockIdx.y * rows_per_cta, r1 = min(B, r0 + rows_per_cta);
  float ag = 0.f, ab = 0.f;
  if (c < C) {
    const float rs = rsqrtf(var[c] + eps), m = mean[c], gm = gamma ? gamma[c] : 1.f;
    for (int r = r0 + rl; r < r1; r += kBnRows) {
      const float d = dy[(size_t)r * ldd + c];
      ag += d * (x[(size_t)r * ldx + c] - m) * rs;
      ab += d;
      if (dx) dx[(size_t)r * ldo + c] = d * gm * rs;
    }
  }
  s_g[rl][cl] = ag;
  s_b[rl][cl] = ab;
  __syncthreads();
  if (rl == 0 && c < C) {
#pragma unroll
    for (int k = 1; k < kBnRows; ++k) { ag += s_g[k][cl]; ab += s_b[k][cl]; }
    if (gg) atomicAdd(&gg[c], ag);
    if (gb) atomicAdd(&gb[c], ab);
  }
}

// z = bf16([bn([h | x]) | 1 | 0]); one thread per pair of columns.  `mean_out` / `var_out` keep the moments it used for the
// backward pass.  As separate kernels (h to fp32, concatenation, two copies of the moments, normalisation, operand assembly)
// this took six launches of 1 to 4 us at 32 x 260, and their gradients nine: from the tower to the loss 24 us and back 28.  A
// Wide&Deep step of 1024 examples and 42 columns went from 133 to 108 us with these.
__global__ void __launch_bounds__(256) bn_join_fwd_kernel(const BnInput in, int B, int C, const float* __restrict__ mean,
                                                          const float* __restrict__ var, const float* __restrict__ gamma,
                                                          const float* __restrict__ beta, float eps, __nv_bfloat16* __restrict__ z, int ldz,
                                                          float* __restrict__ mean_out, float* __restrict__ var_out) {
  pdl_sync();
  const int half = ldz >> 1;
  const long long n = (long long)B * half, first = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  for (long long i = first; i < C; i += (long long)gridDim.x * blockDim.x) { mean_out[i] = mean[i]; var_out[i] = var[i]; }
  for (long long i = first; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int r = (int)(i / half), c0 = 2 * (int)(i - (long long)r * half);
    float v[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int c = c0 + k;
      v[k] = c == C ? 1.f : 0.f;
      if (c < C) {
        v[k] = (bn_at(in, r, c) - mean[c]) * rsqrtf(var[c] + eps);
        if (gamma) v[k] *= gamma[c];
        if (beta) v[k] += beta[c];
      }
    }
    *reinterpret_cast<__nv_bfloat162*>(z + (size_t)r * ldz + c0) = __floats2bfloat162_rn(v[0], v[1]);
  }
}

// A training step's forward pass over the layer: sums of the batch, table and normalised operand.  A block has all rows of eight
// columns, of which a thread holds a pair in kR rows in registers, so the batch is read once and no block waits for another: each
// works its columns' moments out of the table and its own sums.  What they share is the count that decides between accumulation
// and window, taken over all columns; every block reads it before it draws a ticket, and the last to draw writes the counts back.
// `ticket` is a word of the batch scratch, which is zero between launches.
// A chain of loads, barriers and 64-bit arithmetic: 32 x 260 4.2 us where the three launches take 8.1, 1024 x 42 6.3 for 9; in a
// captured step, where launches overlap, 4.0 us for 6.5 from the tower's end to the head's start.  (With the totals read after
// the barrier and a last block found out in front of the arithmetic, 4.9.)  Beyond kTrainRows a thread's registers would not
// hold its rows.
constexpr int kTrainPairs = 4;
constexpr int kTrainMaxLanes = 256;                       // of rows, in a block
constexpr int kTrainMaxFlight = 8;
constexpr int kTrainRows = kTrainMaxLanes * kTrainMaxFlight;

template <int kR>
__global__ void __launch_bounds__(kTrainPairs * kTrainMaxLanes) bn_join_train_kernel(const BnTableView t, const BnInput in, int B,
                                                                                     const float* __restrict__ gamma,
                                                                                     const float* __restrict__ beta, float eps, int drop_inc,
                                                                                     __nv_bfloat16* __restrict__ z, int ldz,
                                                                                     float* __restrict__ mean_out,
                                                                                     float* __restrict__ var_out, unsigned* ticket) {
  constexpr int kCols = 2 * kTrainPairs;
  __shared__ double s_part[kTrainPairs * kTrainMaxLanes / 32][kCols][2];
  __shared__ double s_count[32];
  __shared__ float s_mean[kCols], s_rs[kCols];
  pdl_sync();
  const int C = t.C, lanes = blockDim.x / kTrainPairs, pair = threadIdx.x % kTrainPairs, rl = threadIdx.x / kTrainPairs;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const int c0 = 2 * (blockIdx.x * kTrainPairs + pair);
  float v[kR][2];
#pragma unroll
  for (int i = 0; i < kR; ++i) {
    const int r = rl + i * lanes;
#pragma unroll
    for (int k = 0; k < 2; ++k) v[i][k] = r < B && c0 + k < C ? bn_at(in, r, c0 + k) : 0.f;
  }
  double cur = 0.0;
  for (int c = threadIdx.x; c < C; c += blockDim.x) cur = fmax(cur, t.total_count[c]);
  // the first warp's lanes take a column each, four lanes to a column, of which the first keeps the table
  const int own = blockIdx.x * kCols + lane % kCols;
  const bool owner = warp == 0 && lane < kCols && own < C;
  BnTotals total = {};
  if (owner) total = bn_totals(t, own);
  float g[2] = {1.f, 1.f}, b[2] = {0.f, 0.f};
#pragma unroll
  for (int k = 0; k < 2; ++k)
    if (c0 + k < C) {
      if (gamma) g[k] = gamma[c0 + k];
      if (beta) b[k] = beta[c0 + k];
    }
  double s[2] = {0.0, 0.0}, q[2] = {0.0, 0.0};
#pragma unroll
  for (int i = 0; i < kR; ++i)
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const double d = (double)v[i][k];
      s[k] += d;
      q[k] += d * d;
    }
#pragma unroll
  for (int k = 0; k < 2; ++k)
    for (int off = kTrainPairs; off < 32; off <<= 1) {
      s[k] += __shfl_xor_sync(0xffffffffu, s[k], off);
      q[k] += __shfl_xor_sync(0xffffffffu, q[k], off);
    }
  for (int off = 16; off > 0; off >>= 1) cur = fmax(cur, __shfl_xor_sync(0xffffffffu, cur, off));
  if (lane < kTrainPairs) {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      s_part[warp][2 * pair + k][0] = s[k];
      s_part[warp][2 * pair + k][1] = q[k];
    }
  }
  if (lane == 0) s_count[warp] = cur;
  __syncthreads();
  bool window = false, last = false;
  if (warp == 0 || warp == warps - 1) {
    cur = lane < warps ? s_count[lane] : 0.0;
    for (int off = 16; off > 0; off >>= 1) cur = fmax(cur, __shfl_xor_sync(0xffffffffu, cur, off));
    cur = floor(cur);
    window = t.max_count > 0 && cur > (double)t.max_count;
  }
  if (warp == warps - 1 && lane == 0) {                   // (never the first warp: a block has at least four)
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  if (warp == 0) {
    double as = 0.0, aq = 0.0;
    for (int w = lane / kCols; w < warps; w += 32 / kCols) { as += s_part[w][lane % kCols][0]; aq += s_part[w][lane % kCols][1]; }
    for (int off = kCols; off < 32; off <<= 1) {
      as += __shfl_xor_sync(0xffffffffu, as, off);
      aq += __shfl_xor_sync(0xffffffffu, aq, off);
    }
    if (owner) {
      bn_fold(total, as, aq, (double)B, window ? (1.0 - t.moment) * ((double)B / cur) : -1.0);
      float mean, var;
      bn_moments(t, total, &mean, &var);
      s_mean[lane] = mean;
      s_rs[lane] = rsqrtf(var + eps);
      t.mean[own] = mean_out[own] = mean;
      t.var[own] = var_out[own] = var;
      if (drop_inc) { t.inc[own] = 0.0; t.inc[C + own] = 0.0; t.inc[2 * C + own] = 0.0; }
      else { t.inc[own] += as; t.inc[C + own] += aq; t.inc[2 * C + own] += (double)B; }
      bn_keep_sums(t, own, total);
    }
  }
  __syncthreads();
  float m[2], rs[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    m[k] = c0 + k < C ? s_mean[2 * pair + k] : 0.f;
    rs[k] = c0 + k < C ? s_rs[2 * pair + k] : 0.f;
  }
#pragma unroll
  for (int i = 0; i < kR; ++i) {
    const int r = rl + i * lanes;
    if (r >= B) break;
    float o[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      o[k] = c0 + k == C ? 1.f : 0.f;
      if (c0 + k < C) {
        o[k] = (v[i][k] - m[k]) * rs[k];
        if (gamma || beta) o[k] = __fmaf_rn(o[k], g[k], b[k]);
      }
    }
    *reinterpret_cast<__nv_bfloat162*>(z + (size_t)r * ldz + c0) = __floats2bfloat162_rn(o[0], o[1]);
  }
  if (warp == warps - 1 && __shfl_sync(0xffffffffu, (int)last, 0)) {
    if (!window)
      for (int c = lane; c < C; c += 32) t.total_count[c] += (double)B;
    if (lane == 0) *ticket = 0u;
  }
}

// Gradients of the same: gh (bf16, zero beyond its columns, and with `mask` where h is not above zero), gx (fp32), gamma, beta.
__global__ void __launch_bounds__(kBnCols * kBnRows) bn_join_bwd_kernel(const __nv_bfloat16* __restrict__ dz, int ldz, const BnInput in, int B,
                                                                        int C, const float* __restrict__ mean, const float* __restrict__ var,
                                                                        const float* __restrict__ gamma, float eps, int mask,
                                                                        __nv_bfloat16* __restrict__ gh, float* __restrict__ gx, int ldg,
                                                                        float* gg, float* gb, int rows_per_cta) {
  pdl_sync();
  __shared__ float s_g[kBnRows][kBnCols], s_b[kBnRows][kBnCols];
  const int cl = threadIdx.x % kBnCols, rl = threadIdx.x / kBnCols;
  const int c = blockIdx.x * kBnCols + cl;
  const int r0 = blockIdx.y * rows_per_cta, r1 = min(B, r0 + rows_per_cta);
  float ag = 0.f, ab = 0.f;
  if (c < C) {
    const float rs = rsqrtf(var[c] + eps), m = mean[c], gm = gamma ? gamma[c] : 1.f;
    for (int r = r0 + rl; r < r1; r += kBnRows) {
      const float d = __bfloat162float(dz[(size_t)r * ldz + c]), x = bn_at(in, r, c);
      ag += d * (x - m) * rs;
      ab += d;
      const float dx = d * gm * rs;
      if (c < in.nh) {
        if (gh) gh[(size_t)r * in.ldh + c] = __float2bfloat16(mask && !(x > 0.f) ? 0.f : dx);
      } else if (gx) {
        gx[(size_t)r * ldg + (c - in.nh)] = dx;
      }
    }
  } else if (gh && c - C < in.ldh - in.nh) {               // the columns behind h's
    for (int r = r0 + rl; r < r1; r += kBnRows) gh[(size_t)r * in.ldh + in.nh + (c - C)] = __float2bfloat16(0.f);
  }
  s_g[rl][cl] = ag;
  s_b[rl][cl] = ab;
  __syncthreads();
  if (rl == 0 && c < C) {
#pragma unroll
    for (int k = 1; k < kBnRows; ++k) { ag += s_g[k][cl]; ab += s_b[k][cl]; }
    if (gg) atomicAdd(&gg[c], ag);
    if (gb) atomicAdd(&gb[c], ab);
  }
}

inline int rows_per_cta_for(int B, int C) {
  const int col_tiles = (C + kBnCols - 1) / kBnCols;
  int want_y = (148 * 4 + col_tiles - 1) / col_tiles;       // enough CTAs to fill the GPU
  if (want_y < 1) want_y = 1;
  int rows = (B + want_y - 1) / want_y;
  if (rows < kBnMinRows) rows = kBnMinRows;
  return rows;
}

}  // namespace

void launch_bn_batch_stats(const BnInput& in, int B, int C, const float* center, double* batch, cudaStream_t st) {
  const int rows = rows_per_cta_for(B, C);
  dim3 grid((C + kBnCols - 1) / kBnCols, (B + rows - 1) / rows);
  launch_pdl(bn_batch_stats_kernel, grid, dim3(kBnCols * kBnRows), 0, st, in, B, C, center, batch, rows);
}
void launch_bn_table_append(const BnTableView& t, double* batch, bool drop_inc, cudaStream_t st) {
  launch_pdl(bn_table_append_kernel, dim3(1), dim3(1024), 0, st, t, batch, drop_inc ? 1 : 0);
}
void launch_bn_join_fwd(const BnInput& in, int B, int C, const float* mean, const float* var, const float* gamma, const float* beta, float eps,
                        void* z, int ldz, float* mean_out, float* var_out, cudaStream_t st) {
  long long blocks = ((long long)B * (ldz >> 1) + 255) / 256;
  if (blocks > 148 * 8) blocks = 148 * 8;
  launch_pdl(bn_join_fwd_kernel, dim3(blocks < 1 ? 1 : (int)blocks), dim3(256), 0, st, in, B, C, mean, var, gamma, beta, eps,
             reinterpret_cast<__nv_bfloat16*>(z), ldz, mean_out, var_out);
}
bool bn_join_train_fits(int B, int C, int ldz) { return B >= 1 && B <= kTrainRows && C >= 1 && ldz % (2 * kTrainPairs) == 0; }
void launch_bn_join_train(const BnTableView& t, const BnInput& in, int B, const float* gamma, const float* beta, float eps, bool drop_inc,
                          void* z, int ldz, float* mean_out, float* var_out, double* batch, cudaStream_t st) {
  int lanes = 32;
  while (lanes < B && lanes < kTrainMaxLanes) lanes <<= 1;
  const dim3 grid(ldz / (2 * kTrainPairs)), block(kTrainPairs * lanes);
  auto go = [&](auto kernel) {
    launch_pdl(kernel, grid, block, 0, st, t, in, B, gamma, beta, eps, drop_inc ? 1 : 0, reinterpret_cast<__nv_bfloat16*>(z), ldz, mean_out,
               var_out, reinterpret_cast<unsigned*>(batch));
  };
  const int rows = (B + lanes - 1) / lanes;
  if (rows <= 1) go(bn_join_train_kernel<1>);
  else if (rows <= 2) go(bn_join_train_kernel<2>);
  else if (rows <= 4) go(bn_join_train_kernel<4>);
  else go(bn_join_train_kernel<kTrainMaxFlight>);
}
void launch_bn_join_bwd(const void* dz, int ldz, const BnInput& in, int B, int C, const float* mean, const float* var, const float* gamma,
                        float eps, int mask, void* gh, float* gx, int ldg, float* gg, float* gb, cudaStream_t st) {
  const int cols = C + (in.ldh - in.nh), rows = rows_per_cta_for(B, cols);
  dim3 grid((cols + kBnCols - 1) / kBnCols, (B + rows - 1) / rows);
  launch_pdl(bn_join_bwd_kernel, grid, dim3(kBnCols * kBnRows), 0, st, reinterpret_cast<const __nv_bfloat16*>(dz), ldz, in, B, C, mean, var,
             gamma, eps, mask, reinterpret_cast<__nv_bfloat16*>(gh), gx, ldg, gg, gb, rows);
}
void launch_bn_table_refresh(const BnTableView& t, cudaStream_t st) { bn_table_refresh_moments_kernel<<<1, 1024, 0, st>>>(t); }
void launch_bn_table_sync(const BnTableView& t, const BnSyncView& s, double* scratch, cudaStream_t st) {
  bn_table_sync_kernel<<<1, 1024, 0, st>>>(t, s, scratch);
}
void launch_bn_apply_fwd(const float* x, int ldx, int B, int C, const float* mean, const float* var, const float* gamma,
                         const float* beta, float eps, float* y, int ldy, cudaStream_t st) {
  long long n = (long long)B * C;
  int blocks = (int)((n + 255) / 256);
  if (blocks > 148 * 8) blocks = 148 * 8;
  if (blocks < 1) blocks = 1;
  launch_pdl(bn_apply_fwd_kernel, dim3(blocks), dim3(256), 0, st, x, ldx, B, C, mean, var, gamma, beta, eps, y, ldy);
}
void launch_bn_apply_bwd(const float* dy, int ldd, const float* x, int ldx, int B, int C, const float* mean, const float* var,
                         const float* gamma, float eps, float* dx, int ldo, float* gg, float* gb, cudaStream_t st) {
  const int rows = rows_per_cta_for(B, C);
  dim3 grid((C + kBnCols - 1) / kBnCols, (B + rows - 1) / rows);
  launch_pdl(bn_apply_bwd_kernel, grid, dim3(kBnCols * kBnRows), 0, st, dy, ldd, x, ldx, B, C, mean, var, gamma, eps, dx, ldo, gg, gb, rows);
}

}  // namespace tn
