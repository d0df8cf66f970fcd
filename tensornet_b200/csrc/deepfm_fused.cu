// DeepFM-specific fusions of the memory-bound glue around the tensor-core towers
// (model structure: examples/models/deepfm.py, examples/common/layers.py:72-103 in the reference).
//
//   deepfm_input_fwd : gather the pulled embedding rows of every slot (single-hot), compute the
//                      second-order FM term and write the padded bf16 operand of the first MLP layer
//                      [emb | dense | 1 | 0] in one pass - replaces pool + FM + concat/cast.
//   deepfm_input_bwd : gradient of that operand (bf16, from the first layer's dgrad) plus the FM
//                      gradient, scattered straight into the unique-gradient rows - replaces
//                      split/cast + FM backward + add + pool backward.
#include <cuda_bf16.h>
#include "sparse_table.cuh"
#include "tn_ops.h"

namespace tn {

namespace {

__device__ __forceinline__ float wsum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// D % 4 == 0, dq = D/4 a power of two <= 32.  One warp per example.  The rows it has read are left in `E` as they are: the
// backward pass then reads them as one run per example instead of gathering them once more (and does not depend on
// what happens to the pulled rows in between); null when there is none.
template <bool kInPlace>
__global__ void __launch_bounds__(256, 6) deepfm_input_fwd_kernel(const RowSource src, const int* __restrict__ inverse, int B, int S, int D,
                                        const float* __restrict__ dense, int Dd, int ld_dense, __nv_bfloat16* __restrict__ X0, int ld,
                                        float* __restrict__ fm, int lin_col, float* __restrict__ Lout, float* __restrict__ E) {
  const PulledRows<kInPlace> rows(src);
  pdl_sync();
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const int dq = D >> 2, nch = S * dq;
  for (int b = warp; b < B; b += nwarps) {
    __nv_bfloat16* xrow = X0 + (size_t)b * ld;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    float sq = 0.f;
    // batches of 4 x 32 chunks: first all row indices, then all row gathers, then the arithmetic, so that a
    // warp has four independent loads in flight at each of the dependent steps
    for (int c0 = 0; c0 < nch; c0 += 128) {
      int r[4];
      float4 x[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int c = c0 + 32 * k + lane;
        r[k] = c < nch ? __ldg(inverse + (size_t)(c / dq) * B + b) : -1;
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) r[k] = rows.row(r[k]);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int c = c0 + 32 * k + lane;
        x[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r[k] >= 0) x[k] = ldcg_f4(rows.base + (size_t)r[k] * rows.stride + 4 * (c % dq));
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int c = c0 + 32 * k + lane;
        if (c >= nch) continue;
        if (E != nullptr) *reinterpret_cast<float4*>(E + (size_t)b * S * D + 4 * c) = x[k];
        s.x += x[k].x; s.y += x[k].y; s.z += x[k].z; s.w += x[k].w;
        sq += x[k].x * x[k].x + x[k].y * x[k].y + x[k].z * x[k].z + x[k].w * x[k].w;
        __nv_bfloat162 lo = __floats2bfloat162_rn(x[k].x, x[k].y), hi = __floats2bfloat162_rn(x[k].z, x[k].w);
        *reinterpret_cast<uint2*>(xrow + 4 * c) = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
      }
    }
    for (int o = 16; o >= dq; o >>= 1) {
      s.x += __shfl_xor_sync(0xffffffffu, s.x, o); s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
      s.z += __shfl_xor_sync(0xffffffffu, s.z, o); s.w += __shfl_xor_sync(0xffffffffu, s.w, o);
    }
    float part = (lane < dq) ? (s.x * s.x + s.y * s.y + s.z * s.z + s.w * s.w) : 0.f;
    part = wsum(part) - wsum(sq);
    if (lane == 0) fm[b] = 0.5f * part;
    if (lin_col >= 0) {   // the slot's linear weight rides in column `lin_col` of the same row
      for (int f = lane; f < S; f += 32) {
        const int r = rows.row(__ldg(inverse + (size_t)f * B + b));
        Lout[(size_t)b * S + f] = r >= 0 ? __ldcg(rows.base + (size_t)r * rows.stride + lin_col) : 0.f;
      }
    }
    const int tail0 = S * D;
    for (int j = lane; j < ld - tail0; j += 32) {
      float v = 0.f;
      if (j < Dd) v = dense[(size_t)b * ld_dense + j];
      else if (j == Dd) v = 1.f;
      xrow[tail0 + j] = __float2bfloat16(v);
    }
  }
}

__global__ void deepfm_input_bwd_kernel(const float* __restrict__ E, const int* __restrict__ inverse, int B, int S, int D,
                                        const __nv_bfloat16* __restrict__ dX0, int ld, const float* __restrict__ gfm,
                                        float* __restrict__ gU, int gstride, int lin_col, const float* __restrict__ dL) {
  pdl_sync();
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const int dq = D >> 2, nch = S * dq;
  for (int b = warp; b < B; b += nwarps) {
    const __nv_bfloat16* grow = dX0 + (size_t)b * ld;
    const float* e = E + (size_t)b * S * D;
    const float gf = gfm[b];
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    if (nch <= 128) {
      // the usual case: the example's rows stay in registers between the field sum and the gradient
      int v[4];
      float4 x[4];
      uint2 raw[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int c = 32 * k + lane;
        v[k] = c < nch ? __ldg(inverse + (size_t)(c / dq) * B + b) : -1;
        raw[k] = c < nch ? *reinterpret_cast<const uint2*>(grow + 4 * c) : make_uint2(0u, 0u);
        x[k] = c < nch ? ldcg_f4(e + 4 * c) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        s.x += x[k].x; s.y += x[k].y; s.z += x[k].z; s.w += x[k].w;
      }
      for (int o = 16; o >= dq; o >>= 1) {
        s.x += __shfl_xor_sync(0xffffffffu, s.x, o); s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
        s.z += __shfl_xor_sync(0xffffffffu, s.z, o); s.w += __shfl_xor_sync(0xffffffffu, s.w, o);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int c = 32 * k + lane;
        if (v[k] < 0) continue;
        const float2 g01 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw[k].x));
        const float2 g23 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw[k].y));
        float4 g;
        g.x = g01.x + gf * (s.x - x[k].x);
        g.y = g01.y + gf * (s.y - x[k].y);
        g.z = g23.x + gf * (s.z - x[k].z);
        g.w = g23.y + gf * (s.w - x[k].w);
        red_add_f32x4(gU + (size_t)v[k] * gstride + 4 * (c % dq), g);
      }
    } else {
      for (int c = lane; c < nch; c += 32) {
        const float4 x = ldcg_f4(e + 4 * c);
        s.x += x.x; s.y += x.y; s.z += x.z; s.w += x.w;
      }
      for (int o = 16; o >= dq; o >>= 1) {
        s.x += __shfl_xor_sync(0xffffffffu, s.x, o); s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
        s.z += __shfl_xor_sync(0xffffffffu, s.z, o); s.w += __shfl_xor_sync(0xffffffffu, s.w, o);
      }
      for (int c = lane; c < nch; c += 32) {
        const int f = c / dq, dc = c - f * dq;
        const int v = __ldg(inverse + (size_t)f * B + b);
        if (v < 0) continue;
        const float4 x = ldcg_f4(e + 4 * c);
        const uint2 raw = *reinterpret_cast<const uint2*>(grow + 4 * c);
        const float2 g01 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
        const float2 g23 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
        float4 g;
        g.x = g01.x + gf * (s.x - x.x);
        g.y = g01.y + gf * (s.y - x.y);
        g.z = g23.x + gf * (s.z - x.z);
        g.w = g23.y + gf * (s.w - x.w);
        red_add_f32x4(gU + (size_t)v * gstride + 4 * dc, g);
      }
    }
    if (lin_col >= 0) {
      for (int f = lane; f < S; f += 32) {
        const int v = __ldg(inverse + (size_t)f * B + b);
        if (v >= 0) atomicAdd(gU + (size_t)v * gstride + lin_col, dL[(size_t)b * S + f]);
      }
    }
  }
}

}  // namespace

const char* launch_deepfm_input_fwd(const RowSource& src, const int* inverse, int B, int S, int D, const float* dense, int Dd, int ld_dense,
                                    void* X0, int ld, float* fm, int lin_col, float* Lout, float* E, cudaStream_t st) {
  const int dq = D >> 2;
  if ((D & 3) || dq < 1 || dq > 32 || (dq & (dq - 1))) return "deepfm_input: embedding dim must be 4 * 2^k, at most 128";
  if (ld < S * D + Dd + 1 || (ld & 3)) return "deepfm_input: operand row too short";
  int blocks = (B + 7) / 8; if (blocks > 148 * 8) blocks = 148 * 8; if (blocks < 1) blocks = 1;
  cudaError_t e = launch_pdl(src.row_of != nullptr ? deepfm_input_fwd_kernel<true> : deepfm_input_fwd_kernel<false>, dim3(blocks), dim3(256), 0,
                             st, src, inverse, B, S, D, dense, Dd, ld_dense, reinterpret_cast<__nv_bfloat16*>(X0), ld, fm, lin_col, Lout, E);
  return e == cudaSuccess ? nullptr : cudaGetErrorString(e);
}
const char* launch_deepfm_input_bwd(const float* E, const int* inverse, int B, int S, int D, const void* dX0, int ld, const float* gfm,
                                    float* gU, int gstride, int lin_col, const float* dL, cudaStream_t st) {
  const int dq = D >> 2;
  if ((D & 3) || dq < 1 || dq > 32 || (dq & (dq - 1))) return "deepfm_input: embedding dim must be 4 * 2^k, at most 128";
  int blocks = (B + 7) / 8; if (blocks > 148 * 8) blocks = 148 * 8; if (blocks < 1) blocks = 1;
  cudaError_t e = launch_pdl(deepfm_input_bwd_kernel, dim3(blocks), dim3(256), 0, st, E, inverse, B, S, D,
                             reinterpret_cast<const __nv_bfloat16*>(dX0), ld, gfm, gU, gstride, lin_col, dL);
  return e == cudaSuccess ? nullptr : cudaGetErrorString(e);
}

}  // namespace tn
