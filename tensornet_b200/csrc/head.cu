// The Dense(1) head of every model over the pieces its operand is made of (a tower's output, cross columns, linear weights,
// an FM term; examples/models/{wide_deep,deepfm,deep_cross}.py in the reference):
//
//   head_loss  : logit, sigmoid cross-entropy, CTR / PCTR sums and the complete backward pass of the head (gradient of every
//                piece with the tower's ReLU mask applied, gradient of the weights) in one kernel - the logit's gradient
//                depends on nothing but the logit and the label, so forward and backward of the head are one pass
//   head_score : the logits alone
#include <cuda_bf16.h>
#include "tn_device.cuh"
#include "tn_ops.h"

namespace tn {

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ void unpack8(const uint4& x, float* v) {
  const uint32_t u[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u[k]));
    v[2 * k] = f.x; v[2 * k + 1] = f.y;
  }
}

// Bits of the pair of bf16 columns of which the first `n` count.  What lies behind a piece's columns is left out, not multiplied by
// a zero weight: it need not be a number.
__device__ __forceinline__ uint32_t pair_mask(int n) { return n >= 2 ? 0xffffffffu : n == 1 ? 0x0000ffffu : 0u; }

// The loss is summed in a word of the scratch that is zero between launches; the last block to finish moves it into
// `loss_out` and re-arms the scratch, so the caller never has to clear anything.  One thread per block, after its own add.
__device__ __forceinline__ bool publish_loss(const HeadArgs& a) {
  __threadfence();
  const bool last = atomicAdd(reinterpret_cast<unsigned*>(a.scratch) + 1, 1u) == gridDim.x - 1;
  if (last) {
    __threadfence();
    *a.loss_out = atomicExch(&a.scratch[0], 0.f);
    reinterpret_cast<unsigned*>(a.scratch)[1] = 0u;
  }
  return last;
}

// The weights in shared memory, every piece's on a boundary of eight floats with zeros behind its last one.
__device__ __forceinline__ void load_weights(const HeadArgs& a, float* s_w) {
  for (int k = threadIdx.x; k < a.span; k += blockDim.x) {
    float v = 0.f;
#pragma unroll
    for (int p = 0; p < kMaxHeadPieces; ++p)
      if (p < a.n && k >= a.at[p] && k < a.at[p] + a.width[p]) v = __ldg(a.w + a.first[p] + (k - a.at[p]));
    s_w[k] = v;
  }
}

// kRows dot products of a warp side by side: rows b0, b0 + stride, ... (those below B).
template <int kRows>
__device__ __forceinline__ void row_dots(const HeadArgs& a, const float* s_w, int b0, int stride, int lane, float* dot) {
#pragma unroll
  for (int q = 0; q < kRows; ++q) dot[q] = 0.f;
  for (int p = 0; p < a.n; ++p) {
    const float* sw = s_w + a.at[p];
    const int width = a.width[p];
    if (a.kind[p] == kHeadBf16) {
      for (int c = 8 * lane; c < width; c += 256) {
        uint4 z[kRows];
#pragma unroll
        for (int q = 0; q < kRows; ++q) {
          const int b = b0 + q * stride;
          z[q] = b < a.B ? *reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(a.src[p]) + (size_t)b * a.ld[p] + c)
                         : make_uint4(0u, 0u, 0u, 0u);
        }
        const float4 w0 = *reinterpret_cast<const float4*>(sw + c), w1 = *reinterpret_cast<const float4*>(sw + c + 4);
        const int n = width - c;
        const uint32_t m0 = pair_mask(n), m1 = pair_mask(n - 2), m2 = pair_mask(n - 4), m3 = pair_mask(n - 6);
#pragma unroll
        for (int q = 0; q < kRows; ++q) {
          float v[8];
          z[q].x &= m0; z[q].y &= m1; z[q].z &= m2; z[q].w &= m3;
          unpack8(z[q], v);
          dot[q] += v[0] * w0.x + v[1] * w0.y + v[2] * w0.z + v[3] * w0.w + v[4] * w1.x + v[5] * w1.y + v[6] * w1.z + v[7] * w1.w;
        }
      }
    } else if (a.kind[p] == kHeadF32x4) {
      for (int c = 4 * lane; c < width; c += 128) {
        float4 z[kRows];
#pragma unroll
        for (int q = 0; q < kRows; ++q) {
          const int b = b0 + q * stride;
          z[q] = b < a.B ? *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(a.src[p]) + (size_t)b * a.ld[p] + c)
                         : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        const float4 w = *reinterpret_cast<const float4*>(sw + c);
#pragma unroll
        for (int q = 0; q < kRows; ++q) dot[q] += z[q].x * w.x + z[q].y * w.y + z[q].z * w.z + z[q].w * w.w;
      }
    } else {
      for (int c = lane; c < width; c += 32) {
        const float w = sw[c];
#pragma unroll
        for (int q = 0; q < kRows; ++q) {
          const int b = b0 + q * stride;
          if (b < a.B) dot[q] += reinterpret_cast<const float*>(a.src[p])[(size_t)b * a.ld[p] + c] * w;
        }
      }
    }
  }
#pragma unroll
  for (int q = 0; q < kRows; ++q) dot[q] = warp_sum(dot[q]);
}

// A block takes kWarps * kRows rows at a time.  First a warp per kRows rows: dot products, loss and the logits' gradients,
// which meet in shared memory.  Then a thread per 16-byte unit of a row (eight bf16 or four fp32 columns; one where rows are
// not on such boundaries): it reads its columns of the block's rows once more (from L1), writes their gradients and sums
// dlogit * z in registers, so the gradient of the weights needs no atomics below the block.  Narrow heads leave threads over:
// they take every second, fourth, ... row of the same unit.
// The blocks' weight gradients meet in kHeadCopies partial copies in `scratch` (hundreds of blocks that add to the same few
// hundred words at once queue up in L2), and the last block to finish folds the copies into gw, writes the loss and leaves the
// scratch at zero; a single block adds to gw directly.
// Scratch: [0] loss, [1] finished blocks, [2] gradient of the bias, from [4] on the copies.
template <int kRows>
__global__ void __launch_bounds__(kThreads, 4) head_loss_kernel(const __grid_constant__ HeadArgs a) {
  pdl_sync();
  extern __shared__ __align__(16) float s_mem[];
  constexpr int kBlockRows = kWarps * kRows;
  float* s_w = s_mem;
  float* s_gw = s_mem + a.span;                // [row groups][span]
  __shared__ float s_dl[kBlockRows];
  __shared__ float s_sum[4][kWarps];
  __shared__ int s_last;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  load_weights(a, s_w);
  for (int k = threadIdx.x; k < a.span * a.groups; k += kThreads) s_gw[k] = 0.f;
  const float bias = __ldg(a.w + a.K);
  const float invB = 1.f / (float)a.B;
  const int slots = kThreads / a.groups, slot = threadIdx.x % slots, group = threadIdx.x / slots;
  float ls = 0.f, ys = 0.f, ps = 0.f, gb = 0.f;
  __syncthreads();
  for (int r0 = blockIdx.x * kBlockRows; r0 < a.B; r0 += gridDim.x * kBlockRows) {
    {
      const int b0 = r0 + wib, mine = b0 + lane * kWarps;          // lane q looks after row q of the warp's
      const bool own = lane < kRows && mine < a.B;
      const float y = own ? __ldg(a.label + mine) : 0.f;
      float dot[kRows], sum = 0.f;
      row_dots<kRows>(a, s_w, b0, kWarps, lane, dot);
#pragma unroll
      for (int q = 0; q < kRows; ++q) if (lane == q) sum = dot[q];
      const float logit = sum + bias;
      const float p = 1.f / (1.f + expf(-logit));
      if (own) {
        const float dl = (p - y) * invB;
        ls += fmaxf(logit, 0.f) + log1pf(expf(-fabsf(logit))) - y * logit;
        ys += y; ps += p; gb += dl;
        if (a.pred) a.pred[mine] = p;
        if (a.nbins > 0)
          atomicAdd(reinterpret_cast<unsigned*>(a.sums + 4) + (y > 0.5f ? 0 : a.nbins) + min(a.nbins - 1, (int)(p * (float)a.nbins)), 1u);
        s_dl[wib + lane * kWarps] = dl;
      }
    }
    __syncthreads();
    const int rows = min(kBlockRows, a.B - r0);
    int u0 = 0;                                                     // first unit of the piece
    for (int p = 0; p < a.n; ++p) {
      const int units = a.units[p];
      int u = slot - u0 % slots;
      if (u < 0) u += slots;
      u0 += units;
      for (; u < units; u += slots) {
        if (a.kind[p] == kHeadBf16) {
          const int c = 8 * u;
          float w[8], acc[8];
          bool on[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            on[k] = c + k < a.width[p];
            w[k] = on[k] ? s_w[a.at[p] + c + k] : 0.f;
            acc[k] = 0.f;
          }
          const __nv_bfloat16* z = reinterpret_cast<const __nv_bfloat16*>(a.src[p]) + (size_t)r0 * a.ld[p] + c;
          __nv_bfloat16* g = a.grad[p] ? reinterpret_cast<__nv_bfloat16*>(a.grad[p]) + (size_t)r0 * a.gld[p] + c : nullptr;
          const bool mask = p == 0 && a.relu_first;
#pragma unroll 2
          for (int r = group; r < rows; r += a.groups) {
            float v[8];
            unpack8(*reinterpret_cast<const uint4*>(z + (size_t)r * a.ld[p]), v);
            const float dl = s_dl[r];
            uint32_t o[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const float gx = !mask || v[2 * k] > 0.f ? dl * w[2 * k] : 0.f, gy = !mask || v[2 * k + 1] > 0.f ? dl * w[2 * k + 1] : 0.f;
              const __nv_bfloat162 h = __floats2bfloat162_rn(gx, gy);
              o[k] = *reinterpret_cast<const uint32_t*>(&h);
            }
            if (g) *reinterpret_cast<uint4*>(g + (size_t)r * a.gld[p]) = make_uint4(o[0], o[1], o[2], o[3]);
#pragma unroll
            for (int k = 0; k < 8; ++k) acc[k] += dl * v[k];
          }
          float* gw = s_gw + group * a.span + a.at[p] + c;
#pragma unroll
          for (int k = 0; k < 8; ++k) if (on[k]) gw[k] += acc[k];
        } else if (a.kind[p] == kHeadF32x4) {
          const int c = 4 * u;
          const float4 w = *reinterpret_cast<const float4*>(s_w + a.at[p] + c);
          float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
          const float* z = reinterpret_cast<const float*>(a.src[p]) + (size_t)r0 * a.ld[p] + c;
          float* g = a.grad[p] ? reinterpret_cast<float*>(a.grad[p]) + (size_t)r0 * a.gld[p] + c : nullptr;
#pragma unroll 2
          for (int r = group; r < rows; r += a.groups) {
            const float4 v = *reinterpret_cast<const float4*>(z + (size_t)r * a.ld[p]);
            const float dl = s_dl[r];
            if (g) *reinterpret_cast<float4*>(g + (size_t)r * a.gld[p]) = make_float4(dl * w.x, dl * w.y, dl * w.z, dl * w.w);
            acc.x += dl * v.x; acc.y += dl * v.y; acc.z += dl * v.z; acc.w += dl * v.w;
          }
          float4* gw = reinterpret_cast<float4*>(s_gw + group * a.span + a.at[p] + c);
          const float4 o = *gw;
          *gw = make_float4(o.x + acc.x, o.y + acc.y, o.z + acc.z, o.w + acc.w);
        } else {
          const float w = s_w[a.at[p] + u];
          float acc = 0.f;
          const float* z = reinterpret_cast<const float*>(a.src[p]) + (size_t)r0 * a.ld[p] + u;
          float* g = a.grad[p] ? reinterpret_cast<float*>(a.grad[p]) + (size_t)r0 * a.gld[p] + u : nullptr;
#pragma unroll 4
          for (int r = group; r < rows; r += a.groups) {
            const float dl = s_dl[r];
            acc += dl * z[(size_t)r * a.ld[p]];
            if (g) g[(size_t)r * a.gld[p]] = dl * w;
          }
          s_gw[group * a.span + a.at[p] + u] += acc;
        }
      }
    }
    __syncthreads();
  }
  ls = warp_sum(ls); ys = warp_sum(ys); ps = warp_sum(ps); gb = warp_sum(gb);
  if (lane == 0) { s_sum[0][wib] = ls * invB; s_sum[1][wib] = ys; s_sum[2][wib] = ps; s_sum[3][wib] = gb; }
  __syncthreads();
  const bool alone = gridDim.x == 1;
  if (threadIdx.x < 4) {
    float v = 0.f;
#pragma unroll
    for (int k = 0; k < kWarps; ++k) v += s_sum[threadIdx.x][k];
    if (threadIdx.x < 3) atomicAdd(&a.sums[threadIdx.x], v);
    if (alone) {
      if (threadIdx.x == 0) *a.loss_out = v;
      if (threadIdx.x == 3) a.gw[a.K] += v;
    } else {
      if (threadIdx.x == 0) atomicAdd(&a.scratch[0], v);
      if (threadIdx.x == 3) atomicAdd(&a.scratch[2], v);
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 4) atomicAdd(&a.sums[3], (float)a.B);
  float* copies = a.scratch + 4;
  for (int k = 4 * threadIdx.x; k < a.span; k += 4 * kThreads) {
    float4 v = *reinterpret_cast<const float4*>(s_gw + k);
    for (int q = 1; q < a.groups; ++q) {
      const float4 x = *reinterpret_cast<const float4*>(s_gw + q * a.span + k);
      v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
    }
    if (!alone) red_add_f32x4(copies + (size_t)(blockIdx.x % kHeadCopies) * a.span + k, v);
    else *reinterpret_cast<float4*>(s_gw + k) = v;
  }
  __syncthreads();
  if (!alone) {
    if (threadIdx.x == 0) s_last = publish_loss(a);
    __syncthreads();
    if (!s_last) return;
    if (threadIdx.x == 0) a.gw[a.K] += atomicExch(&a.scratch[2], 0.f);
  }
  for (int k = threadIdx.x; k < a.span; k += kThreads) {
    float sum = 0.f;
    if (alone) {
      sum = s_gw[k];
    } else {
      float x[kHeadCopies];
#pragma unroll
      for (int q = 0; q < kHeadCopies; ++q) x[q] = __ldcg(copies + (size_t)q * a.span + k);
#pragma unroll
      for (int q = 0; q < kHeadCopies; ++q) { sum += x[q]; copies[(size_t)q * a.span + k] = 0.f; }
    }
    for (int p = 0; p < a.n; ++p)
      if (k >= a.at[p] && k < a.at[p] + a.width[p]) a.gw[a.first[p] + (k - a.at[p])] += sum;      // nobody else adds to it meanwhile
  }
}

template <int kRows>
__global__ void __launch_bounds__(kThreads) head_score_kernel(const __grid_constant__ HeadArgs a) {
  pdl_sync();
  extern __shared__ __align__(16) float s_mem[];
  load_weights(a, s_mem);
  const float bias = __ldg(a.w + a.K);
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  __syncthreads();
  for (int r0 = blockIdx.x * kWarps * kRows; r0 < a.B; r0 += gridDim.x * kWarps * kRows) {
    const int b0 = r0 + wib, mine = b0 + lane * kWarps;
    float dot[kRows], sum = 0.f;
    row_dots<kRows>(a, s_mem, b0, kWarps, lane, dot);
#pragma unroll
    for (int q = 0; q < kRows; ++q) if (lane == q) sum = dot[q];
    if (lane < kRows && mine < a.B) a.pred[mine] = sum + bias;
  }
}

// Heads over [h | L | one column] whose row fits the registers of a warp: 64 * kPairs columns of h, 32 * kLin of L.  Every
// piece is read once.  A warp has kR rows on the way at once (packed as they are stored), their scalar mathematics run side by
// side in one lane per row, gradients of the weights are summed in registers, and warps meet in shared memory with plain
// stores (a float add to shared memory is a compare-and-swap loop).
//
// Bound by latency: a quarter of the warps an SM can hold (128 registers), memory at 7 % of its rate.
// 8192 x [400 | 26 | 1] 8.2 us, 4096 x [256 | 200] 7.0, 2999 x [75 | 39 | 1] 5.6, 1024 x 42 3.8, 32 x 260 3.3.  As kernels of
// their own (operand assembled, dot products, loss, gradients, and the copies and fills between them) the last four took
// 36, 47, 12 and 12 us of a step's critical path, seven to eleven launches.
template <int kPairs, int kLin, bool kMask>
__global__ void __launch_bounds__(kThreads, 2) head_loss_rows_kernel(const __grid_constant__ HeadArgs a) {
  pdl_sync();
  constexpr int kR = kLin > 4 ? 2 : kPairs == 8 && kLin > 1 ? 3 : 4;      // (what 128 registers hold)
  extern __shared__ __align__(16) float s_mem[];       // [kWarps][NWp]
  __shared__ float s_sum[3][kWarps];
  __shared__ int s_last;
  const int B = a.B, NH = a.width[0], ldh = a.ld[0];
  const int pl = kLin > 0 ? 1 : 0;                     // piece L; the column follows
  const int NL = kLin > 0 ? a.width[1] : 0;
  const bool col = a.n > 1 + pl;
  const __nv_bfloat16* H = reinterpret_cast<const __nv_bfloat16*>(a.src[0]);
  __nv_bfloat16* dH = reinterpret_cast<__nv_bfloat16*>(a.grad[0]);
  const float* L = reinterpret_cast<const float*>(a.src[1]);
  float* dL = reinterpret_cast<float*>(a.grad[1]);
  const float* F = reinterpret_cast<const float*>(a.src[1 + pl]);
  float* dF = reinterpret_cast<float*>(a.grad[1 + pl]);
  const int NW = a.K + 1, NWp = (NW + 3) & ~3;
  const int warp = (blockIdx.x * kThreads + threadIdx.x) >> 5, lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int nwarps = gridDim.x * kWarps;
  float2 wv[kPairs], acc[kPairs];
#pragma unroll
  for (int i = 0; i < kPairs; ++i) {
    const int c = 64 * i + 2 * lane;
    wv[i].x = c < NH ? __ldg(a.w + c) : 0.f;
    wv[i].y = c + 1 < NH ? __ldg(a.w + c + 1) : 0.f;
    acc[i] = make_float2(0.f, 0.f);
  }
  float wl[kLin > 0 ? kLin : 1], accl[kLin > 0 ? kLin : 1];
#pragma unroll
  for (int i = 0; i < kLin; ++i) {
    wl[i] = lane + 32 * i < NL ? __ldg(a.w + NH + lane + 32 * i) : 0.f;
    accl[i] = 0.f;
  }
  const float wf = col ? __ldg(a.w + NH + NL) : 0.f, bias = __ldg(a.w + a.K);
  float accf = 0.f, accb = 0.f, ls = 0.f, ys = 0.f, ps = 0.f;
  const float invB = 1.f / (float)B;
  for (int b0 = warp; b0 < B; b0 += kR * nwarps) {
    __nv_bfloat162 z[kR][kPairs];
    float lv[kR][kLin > 0 ? kLin : 1], dot[kR];
#pragma unroll
    for (int q = 0; q < kR; ++q) {
      const int b = b0 + q * nwarps;
      const __nv_bfloat162* zr = reinterpret_cast<const __nv_bfloat162*>(H + (size_t)b * ldh);
#pragma unroll
      for (int i = 0; i < kPairs; ++i) z[q][i] = b < B && 64 * i + 2 * lane < NH ? zr[32 * i + lane] : __floats2bfloat162_rn(0.f, 0.f);
#pragma unroll
      for (int i = 0; i < kLin; ++i) lv[q][i] = b < B && lane + 32 * i < NL ? L[(size_t)b * NL + lane + 32 * i] : 0.f;
    }
    if (NH & 1) {                                                 // the last column's neighbour
#pragma unroll
      for (int q = 0; q < kR; ++q)
#pragma unroll
        for (int i = 0; i < kPairs; ++i)
          if (64 * i + 2 * lane == NH - 1) z[q][i].y = __float2bfloat16(0.f);
    }
    const int mine = b0 + lane * nwarps;                          // lane q looks after row q
    const bool own = lane < kR && mine < B;
    const float f = own && col ? F[mine] : 0.f, y = own ? a.label[mine] : 0.f;
#pragma unroll
    for (int q = 0; q < kR; ++q) {
      dot[q] = 0.f;
#pragma unroll
      for (int i = 0; i < kLin; ++i) dot[q] += lv[q][i] * wl[i];
#pragma unroll
      for (int i = 0; i < kPairs; ++i) {
        const float2 zz = __bfloat1622float2(z[q][i]);
        dot[q] += zz.x * wv[i].x + zz.y * wv[i].y;
      }
    }
    float sum = 0.f;
#pragma unroll
    for (int q = 0; q < kR; ++q) {
      const float d = warp_sum(dot[q]);
      if (lane == q) sum = d;
    }
    const float logit = sum + f * wf + bias;
    const float p = 1.f / (1.f + expf(-logit));
    const float dl = (p - y) * invB;
    if (own) {
      ls += fmaxf(logit, 0.f) + log1pf(expf(-fabsf(logit))) - y * logit;
      ys += y; ps += p;
      if (a.pred) a.pred[mine] = p;
      if (a.nbins > 0)
        atomicAdd(reinterpret_cast<unsigned*>(a.sums + 4) + (y > 0.5f ? 0 : a.nbins) + min(a.nbins - 1, (int)(p * (float)a.nbins)), 1u);
      if (col) dF[mine] = dl * wf;
      accf += dl * f;
      accb += dl;
    }
#pragma unroll
    for (int q = 0; q < kR; ++q) {
      const int b = b0 + q * nwarps;
      const float d = __shfl_sync(0xffffffffu, dl, q);
      if (b >= B) continue;
#pragma unroll
      for (int i = 0; i < kLin; ++i) {
        if (lane + 32 * i >= NL) continue;
        dL[(size_t)b * NL + lane + 32 * i] = d * wl[i];
        accl[i] += d * lv[q][i];
      }
      __nv_bfloat162* dz = reinterpret_cast<__nv_bfloat162*>(dH + (size_t)b * ldh);
#pragma unroll
      for (int i = 0; i < kPairs; ++i) {
        const int c = 64 * i + 2 * lane;
        if (c >= ldh) continue;
        const float2 zz = __bfloat1622float2(z[q][i]);
        // (weights beyond NH are zero: the ones and padding columns get no gradient)
        const float gx = !kMask || zz.x > 0.f ? d * wv[i].x : 0.f, gy = !kMask || zz.y > 0.f ? d * wv[i].y : 0.f;
        dz[32 * i + lane] = __floats2bfloat162_rn(gx, gy);
        acc[i].x += d * zz.x;
        acc[i].y += d * zz.y;
      }
    }
  }
  ls = warp_sum(ls); ys = warp_sum(ys); ps = warp_sum(ps); accf = warp_sum(accf); accb = warp_sum(accb);
  float* my_gw = s_mem + wib * NWp;
#pragma unroll
  for (int i = 0; i < kPairs; ++i) {
    const int c = 64 * i + 2 * lane;
    if (c < NH) my_gw[c] = acc[i].x;
    if (c + 1 < NH) my_gw[c + 1] = acc[i].y;
  }
#pragma unroll
  for (int i = 0; i < kLin; ++i)
    if (lane + 32 * i < NL) my_gw[NH + lane + 32 * i] = accl[i];
  if (lane == 0) {
    if (col) my_gw[NH + NL] = accf;
    my_gw[a.K] = accb;
    for (int k = NW; k < NWp; ++k) my_gw[k] = 0.f;
    s_sum[0][wib] = ls * invB; s_sum[1][wib] = ys; s_sum[2][wib] = ps;
  }
  __syncthreads();
  const bool alone = gridDim.x == 1;
  float part = 0.f;
  if (threadIdx.x < 3) {
#pragma unroll
    for (int k = 0; k < kWarps; ++k) part += s_sum[threadIdx.x][k];
    atomicAdd(&a.sums[threadIdx.x], part);
    if (threadIdx.x == 0) {
      if (alone) *a.loss_out = part;
      else atomicAdd(&a.scratch[0], part);
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 3) atomicAdd(&a.sums[3], (float)B);
  float* parts = a.scratch + 4;
  for (int k = 4 * threadIdx.x; k < NWp; k += 4 * kThreads) {
    float4 v = *reinterpret_cast<const float4*>(s_mem + k);
#pragma unroll
    for (int q = 1; q < kWarps; ++q) {
      const float4 x = *reinterpret_cast<const float4*>(s_mem + q * NWp + k);
      v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
    }
    if (a.copies > 0) {
      red_add_f32x4(parts + (size_t)(blockIdx.x % kHeadCopies) * NWp + k, v);
    } else {
      const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) if (k + j < NW) atomicAdd(a.gw + k + j, e[j]);
    }
  }
  if (alone) return;
  if (a.copies > 0) __syncthreads();
  if (threadIdx.x == 0) s_last = publish_loss(a);
  if (a.copies == 0) return;
  __syncthreads();
  if (!s_last) return;
  for (int k = threadIdx.x; k < NW; k += kThreads) {
    float x[kHeadCopies], sum = 0.f;
#pragma unroll
    for (int q = 0; q < kHeadCopies; ++q) x[q] = __ldcg(parts + (size_t)q * NWp + k);
#pragma unroll
    for (int q = 0; q < kHeadCopies; ++q) {
      sum += x[q];
      parts[(size_t)q * NWp + k] = 0.f;
    }
    a.gw[k] += sum;          // nobody else touches the head's gradient while this kernel runs
  }
}

// The same for a head over one operand [z | 1] and a batch that few blocks get through: lane l has the columns l, l + 32, ... and adds
// them up in that order, so that the logits are, bit for bit, those of the layer on its own (gemv_fwd_kernel); the ones column
// takes part.  What counts at such sizes is the one trip through memory, not the width of the loads.
template <int kCols, bool kMask>
__global__ void __launch_bounds__(kThreads, 2) head_loss_small_kernel(const __grid_constant__ HeadArgs a) {
  pdl_sync();
  constexpr int kR = kCols > 10 ? 2 : 4;
  extern __shared__ __align__(16) float s_mem[];       // [kWarps][NWp]
  __shared__ float s_sum[3][kWarps];
  const int B = a.B, ld = a.ld[0], K = a.K, NW = K + 1, NWp = (NW + 3) & ~3;
  const __nv_bfloat16* Z = reinterpret_cast<const __nv_bfloat16*>(a.src[0]);
  __nv_bfloat16* dZ = reinterpret_cast<__nv_bfloat16*>(a.grad[0]);
  const int warp = (blockIdx.x * kThreads + threadIdx.x) >> 5, lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int nwarps = gridDim.x * kWarps;
  float wv[kCols], acc[kCols];
#pragma unroll
  for (int i = 0; i < kCols; ++i) {
    const int c = lane + 32 * i;
    wv[i] = c < NW ? __ldg(a.w + c) : 0.f;
    acc[i] = 0.f;
  }
  float ls = 0.f, ys = 0.f, ps = 0.f;
  const float invB = 1.f / (float)B;
  for (int b0 = warp; b0 < B; b0 += kR * nwarps) {
    __nv_bfloat16 z[kR][kCols];
    float dot[kR];
#pragma unroll
    for (int q = 0; q < kR; ++q) {
      const int b = b0 + q * nwarps;
#pragma unroll
      for (int i = 0; i < kCols; ++i) {
        const int c = lane + 32 * i;
        z[q][i] = __float2bfloat16(c == K ? 1.f : 0.f);
        if (b < B && c < K) z[q][i] = Z[(size_t)b * ld + c];
      }
    }
    const int mine = b0 + lane * nwarps;                          // lane q looks after row q
    const bool own = lane < kR && mine < B;
    const float y = own ? a.label[mine] : 0.f;
    float logit = 0.f;
#pragma unroll
    for (int q = 0; q < kR; ++q) {
      dot[q] = 0.f;
#pragma unroll
      for (int i = 0; i < kCols; ++i) dot[q] += __bfloat162float(z[q][i]) * wv[i];
      const float d = warp_sum(dot[q]);
      if (lane == q) logit = d;
    }
    const float p = 1.f / (1.f + expf(-logit));
    const float dl = (p - y) * invB;
    if (own) {
      ls += fmaxf(logit, 0.f) + log1pf(expf(-fabsf(logit))) - y * logit;
      ys += y; ps += p;
      if (a.pred) a.pred[mine] = p;
      if (a.nbins > 0)
        atomicAdd(reinterpret_cast<unsigned*>(a.sums + 4) + (y > 0.5f ? 0 : a.nbins) + min(a.nbins - 1, (int)(p * (float)a.nbins)), 1u);
    }
#pragma unroll
    for (int q = 0; q < kR; ++q) {
      const int b = b0 + q * nwarps;
      const float d = __shfl_sync(0xffffffffu, dl, q);
      if (b >= B) continue;
#pragma unroll
      for (int i = 0; i < kCols; ++i) {
        const int c = lane + 32 * i;
        const float zz = __bfloat162float(z[q][i]);
        if (c < ld) dZ[(size_t)b * ld + c] = __float2bfloat16(c < K && (!kMask || zz > 0.f) ? d * wv[i] : 0.f);
        acc[i] += d * zz;
      }
    }
  }
  ls = warp_sum(ls); ys = warp_sum(ys); ps = warp_sum(ps);
#pragma unroll
  for (int i = 0; i < kCols; ++i)
    if (lane + 32 * i < NWp) s_mem[wib * NWp + lane + 32 * i] = acc[i];
  if (lane == 0) { s_sum[0][wib] = ls * invB; s_sum[1][wib] = ys; s_sum[2][wib] = ps; }
  __syncthreads();
  const bool alone = gridDim.x == 1;
  if (threadIdx.x < 3) {
    float part = 0.f;
#pragma unroll
    for (int k = 0; k < kWarps; ++k) part += s_sum[threadIdx.x][k];
    atomicAdd(&a.sums[threadIdx.x], part);
    if (threadIdx.x == 0) {
      if (alone) *a.loss_out = part;
      else atomicAdd(&a.scratch[0], part);
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 3) atomicAdd(&a.sums[3], (float)B);
  for (int k = threadIdx.x; k < NW; k += kThreads) {
    float v = 0.f;
#pragma unroll
    for (int q = 0; q < kWarps; ++q) v += s_mem[q * NWp + k];
    atomicAdd(a.gw + k, v);
  }
  if (!alone && threadIdx.x == 0) publish_loss(a);
}

// The instance for a head, or null where none takes it.  By powers of two, but for the padded rows of 256 to 312 units, which would
// fall to the widest one: five pairs (ten columns) a lane in place of eight (17) take 7.03 in place of 7.43 us at 4096 x [256 | 200],
// 4.9 in place of 5.6 at 500 x 256, 3.3 in place of 4.1 at 32 x 260.
using HeadKernel = void (*)(HeadArgs);
template <int kPairs>
HeadKernel rows_kernel_lin(int lin, bool mask) {
  if (lin == 0) return mask ? head_loss_rows_kernel<kPairs, 0, true> : head_loss_rows_kernel<kPairs, 0, false>;
  if (!mask) return nullptr;
  return lin <= 32 ? head_loss_rows_kernel<kPairs, 1, true> : lin <= 64 ? head_loss_rows_kernel<kPairs, 2, true>
       : lin <= 128 ? head_loss_rows_kernel<kPairs, 4, true> : lin <= 256 ? head_loss_rows_kernel<kPairs, 8, true> : nullptr;
}
HeadKernel rows_kernel(const HeadArgs& a) {
  if (a.kind[0] != kHeadBf16 || a.gld[0] != a.ld[0] || a.grad[0] == nullptr) return nullptr;
  for (int p = 1; p < a.n; ++p)
    if (a.kind[p] == kHeadBf16 || a.ld[p] != a.width[p] || a.gld[p] != a.width[p] || a.grad[p] == nullptr) return nullptr;
  const int lin = a.n > 1 && a.width[1] > 1 ? a.width[1] : 0, rest = a.n - 1 - (lin > 0);
  if (rest > 1 || (rest == 1 && a.width[a.n - 1] != 1)) return nullptr;
  const int ld = a.ld[0];
  const bool mask = a.relu_first != 0;
  return ld <= 64 ? rows_kernel_lin<1>(lin, mask) : ld <= 128 ? rows_kernel_lin<2>(lin, mask) : ld <= 256 ? rows_kernel_lin<4>(lin, mask)
       : ld <= 320 ? rows_kernel_lin<5>(lin, mask) : ld <= 512 ? rows_kernel_lin<8>(lin, mask) : nullptr;
}

HeadKernel small_kernel(const HeadArgs& a) {
  const int cols = a.ld[0] > a.K ? a.ld[0] : a.K + 1;
#define TN_SMALL(n) (a.relu_first ? head_loss_small_kernel<n, true> : head_loss_small_kernel<n, false>)
  return cols <= 64 ? TN_SMALL(2) : cols <= 128 ? TN_SMALL(4) : cols <= 320 ? TN_SMALL(10) : TN_SMALL(17);
#undef TN_SMALL
}

// where the pieces lie in shared memory, and their units
const char* lay_out(HeadArgs& a) {
  if (a.n < 1 || a.n > kMaxHeadPieces) return "head: number of pieces";
  int at = 0, first = 0, units = 0;
  for (int p = 0; p < a.n; ++p) {
    if (a.width[p] < 1) return "head: empty piece";
    a.first[p] = first;
    a.at[p] = at;
    first += a.width[p];
    at += (a.width[p] + 7) & ~7;
    const uintptr_t all = reinterpret_cast<uintptr_t>(a.src[p]) | reinterpret_cast<uintptr_t>(a.grad[p]);
    if (a.kind[p] == kHeadBf16) {
      if ((all & 15) || (a.ld[p] & 7) || (a.gld[p] & 7) || a.width[p] > a.ld[p]) return "head: bf16 pieces need rows of whole 16-byte pieces";
      a.units[p] = (a.grad[p] ? a.gld[p] : a.width[p] + 7) >> 3;
      if (8 * a.units[p] > a.ld[p]) return "head: gradient of a bf16 piece wider than the piece";
    } else {
      a.kind[p] = (all & 15) == 0 && ((a.ld[p] | a.gld[p] | a.width[p]) & 3) == 0 ? kHeadF32x4 : kHeadF32;
      a.units[p] = a.kind[p] == kHeadF32x4 ? a.width[p] >> 2 : a.width[p];
    }
    units += a.units[p];
  }
  if (first != a.K) return "head: the pieces' widths do not add up to the weight's";
  a.span = at;
  if (a.span > kMaxHeadSpan) return "head: too wide";
  int slots = 16;
  while (slots < units && slots < kThreads) slots <<= 1;
  a.groups = kThreads / slots;
  return nullptr;
}

}  // namespace

const char* launch_head_loss(HeadArgs a, cudaStream_t st) {
  if (const char* err = lay_out(a)) return err;
  if (a.B < 1) return "head: empty batch";
  if (HeadKernel k = rows_kernel(a)) {
    // Two blocks per SM, which is what the registers leave room for.  Batches that 64 blocks get through in one turn (four rows a
    // warp) take no more: so few add to gw directly, and the fold of the copies, 1.5 us, falls away (1024 x 42: 5.0 -> 3.5 us).
    // 2999 x 115 the same way 5.7, with one row a warp and the fold 5.2.
    int blocks = (a.B + 4 * kWarps - 1) / (4 * kWarps);
    const bool few = blocks <= 64;
    if (!few) blocks = 148 * 2;
    a.copies = few ? 0 : kHeadCopies;
    if (few && a.n == 1) k = small_kernel(a);
    const cudaError_t e = launch_pdl(k, dim3(blocks), dim3(kThreads), kWarps * ((a.K + 4) & ~3) * sizeof(float), st, a);
    return e == cudaSuccess ? nullptr : cudaGetErrorString(e);
  }
  const size_t smem = (size_t)a.span * (1 + a.groups) * sizeof(float);
  const int rows = a.B > 148 * kWarps ? 2 : 1, per_block = kWarps * rows;
  int blocks = (a.B + per_block - 1) / per_block;
  if (blocks > 148 * 4) blocks = 148 * 4;
  if (a.B <= 2 * kWarps) blocks = 1;
  const cudaError_t e = launch_pdl(rows == 2 ? head_loss_kernel<2> : head_loss_kernel<1>, dim3(blocks), dim3(kThreads), smem, st, a);
  return e == cudaSuccess ? nullptr : cudaGetErrorString(e);
}

const char* launch_head_score(HeadArgs a, cudaStream_t st) {
  if (const char* err = lay_out(a)) return err;
  if (a.B < 1) return "head: empty batch";
  const int rows = a.B > 148 * kWarps * 4 ? 4 : 1, per_block = kWarps * rows;
  int blocks = (a.B + per_block - 1) / per_block;
  if (blocks > 148 * 8) blocks = 148 * 8;
  const cudaError_t e = launch_pdl(rows == 4 ? head_score_kernel<4> : head_score_kernel<1>, dim3(blocks), dim3(kThreads), a.span * sizeof(float), st, a);
  return e == cudaSuccess ? nullptr : cudaGetErrorString(e);
}

}  // namespace tn
