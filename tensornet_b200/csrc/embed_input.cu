// The input of a model's dense part straight from the pulled rows, and its gradient straight into the rows' gradients
// (model structure: examples/models/{wide_deep,deepfm,deep_cross}.py, examples/common/layers.py:72-103 in the reference):
//
//   embed_input_fwd : pool every slot's rows, write the padded bf16 operand of the first layer [emb | dense | 1 | 0] and, where
//                     wanted, the pooled columns in fp32, the second-order FM term and a linear weight that rides in the rows
//   embed_input_bwd : gradient of that operand (bf16, from the first layer), of the FM term and of the pooled columns,
//                     scattered into the unique-gradient rows
//
// in one pass each, in place of pooling, FM, concatenation with its cast, and of split, FM backward, additions, pooling backward.
// Slots hold one id each or ragged bags, and are of any width up to 128 columns; a lane moves four columns (rows are
// whole 16-byte pieces whatever their width), G lanes a slot.
#include <cuda_bf16.h>
#include "sparse_table.cuh"
#include "tn_ops.h"

namespace tn {

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kGradFlight = 4;           // rows a group of lanes has on the way at once in the backward pass

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float bag_scale(int combiner, int len) {
  if (len <= 0) return 0.f;
  if (combiner == 1) return 1.f / (float)len;
  if (combiner == 2) return rsqrtf((float)len);
  return 1.f;
}
// `n` bf16 columns (at most four) to or from an address that is a multiple of SV of them
template <int SV>
__device__ __forceinline__ void store_bf16(__nv_bfloat16* p, const float4& x, int n) {
  const __nv_bfloat162 lo = __floats2bfloat162_rn(x.x, x.y), hi = __floats2bfloat162_rn(x.z, x.w);
  if constexpr (SV == 4) {
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
  } else if constexpr (SV == 2) {
    *reinterpret_cast<__nv_bfloat162*>(p) = lo;
    if (n > 2) *reinterpret_cast<__nv_bfloat162*>(p + 2) = hi;
  } else {
    p[0] = lo.x;
    if (n > 1) p[1] = lo.y;
    if (n > 2) p[2] = hi.x;
    if (n > 3) p[3] = hi.y;
  }
}
template <int SV>
__device__ __forceinline__ float4 load_bf16(const __nv_bfloat16* p, int n) {
  float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
  if constexpr (SV == 4) {
    const uint2 r = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&r.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&r.y));
    x = make_float4(a.x, a.y, b.x, b.y);
  } else if constexpr (SV == 2) {
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p));
    x.x = a.x; x.y = a.y;
    if (n > 2) { const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p + 2)); x.z = b.x; x.w = b.y; }
  } else {
    x.x = __bfloat162float(p[0]);
    if (n > 1) x.y = __bfloat162float(p[1]);
    if (n > 2) x.z = __bfloat162float(p[2]);
    if (n > 3) x.w = __bfloat162float(p[3]);
  }
  return x;
}

// `wpe` warps (a power of two) share an example, each takes a run of its slots; they meet in shared memory for the FM term.  A
// warp first fetches the row numbers of up to 32 slots, a lane each (or the bounds of their bags), hands them to the groups of
// G lanes that read the rows, kFlight at a time: the chain of dependent loads is walked once per 32 slots.
// Bound by the latency of those loads (L2 and memory at 22 and 15 % of their rates).  8192 x 26 slots of 16 with their linear weights 17.8 us.  In place of pooling, FM term
// and concatenation: 2999 x 39 slots of 10, 8.2 us for 18 (and three launches more); 4096 x 20 bags of three ids and 10 columns 24
// for 22.6; 8192 x 100 bags of five ids and 64 columns 330 for 375.  More blocks of fewer registers per SM (five, six, eight):
// 8 to 40 % slower; sixty-four warps per SM by splitting examples: 7 to 50 % slower.
template <bool kInPlace, bool kBags, int SV, int kFlight>
__global__ void __launch_bounds__(kThreads, 4) embed_input_fwd_kernel(const RowSource src, const __grid_constant__ EmbedInput a, int G, int wpe) {
  const PulledRows<kInPlace> rows(src);
  pdl_sync();
  __shared__ float4 s_sum[kWarps][32];
  __shared__ float s_sq[kWarps];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, sub = lane / G, ch = lane % G, np = 32 / G;
  const int S = a.S, D = a.D, B = a.B, ncol = D - 4 * ch;                 // columns of this lane's piece that count
  const bool on = ncol > 0;
  const int per = (S + wpe - 1) / wpe, epb = kWarps / wpe, part = wib % wpe;
  for (int e0 = blockIdx.x * epb; e0 < B; e0 += gridDim.x * epb) {
    const int b = e0 + wib / wpe;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    float sq = 0.f;
    if (b < B) {
      __nv_bfloat16* xrow = reinterpret_cast<__nv_bfloat16*>(a.X0) + (size_t)b * a.ld;
      float* erow = a.E != nullptr ? a.E + (size_t)b * a.ldE : nullptr;
      auto put = [&](int slot, float4 x) {
        if (ncol < 4) {                                                   // what lies behind the columns is not theirs
          if (ncol < 2) x.y = 0.f;
          if (ncol < 3) x.z = 0.f;
          x.w = 0.f;
        }
        s.x += x.x; s.y += x.y; s.z += x.z; s.w += x.w;
        sq += x.x * x.x + x.y * x.y + x.z * x.z + x.w * x.w;
        if (erow != nullptr) store_cols<SV>(erow + slot * D + 4 * ch, x, ncol);
        store_bf16<SV>(xrow + slot * D + 4 * ch, x, ncol);
      };
      const int s_hi = min(S, part * per + per);
      for (int s0 = part * per; s0 < s_hi; s0 += 32) {
        const int n = min(32, s_hi - s0);
        if constexpr (!kBags) {
          const int r_lane = lane < n ? rows.row(__ldg(a.inverse + (size_t)(s0 + lane) * B + b)) : -1;
          float lin = 0.f;
          if (a.lin_col >= 0 && r_lane >= 0) lin = __ldcg(rows.base + (size_t)r_lane * rows.stride + a.lin_col);
          const float sc = bag_scale(a.combiner, 1);
          for (int p = 0; p < n; p += kFlight * np) {
            float4 x[kFlight];
#pragma unroll
            for (int q = 0; q < kFlight; ++q) {
              const int at = p + q * np + sub;
              const int r = __shfl_sync(0xffffffffu, r_lane, at & 31);
              x[q] = make_float4(0.f, 0.f, 0.f, 0.f);
              if (on && at < n && r >= 0) x[q] = rows.load4(r, 4 * ch);
            }
#pragma unroll
            for (int q = 0; q < kFlight; ++q) {
              const int at = p + q * np + sub;
              if (on && at < n) put(s0 + at, make_float4(x[q].x * sc, x[q].y * sc, x[q].z * sc, x[q].w * sc));
            }
          }
          if (a.lin_col >= 0 && lane < n) a.Lout[(size_t)b * S + s0 + lane] = lin * sc;
        } else {
          int k0_lane = 0, k1_lane = 0;
          if (lane < n) {
            k0_lane = __ldg(a.offsets + (size_t)(s0 + lane) * B + b);
            k1_lane = __ldg(a.offsets + (size_t)(s0 + lane) * B + b + 1);
          }
          for (int p = 0; p < n; p += np) {
            const int at = p + sub;
            const int k0 = __shfl_sync(0xffffffffu, k0_lane, at & 31), k1 = __shfl_sync(0xffffffffu, k1_lane, at & 31);
            if (!on || at >= n) continue;
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int k = k0; k < k1; k += kFlight) {
              int r[kFlight];
              float4 x[kFlight];
#pragma unroll
              for (int q = 0; q < kFlight; ++q) r[q] = k + q < k1 ? __ldg(a.inverse + k + q) : -1;
#pragma unroll
              for (int q = 0; q < kFlight; ++q) r[q] = rows.row(r[q]);
#pragma unroll
              for (int q = 0; q < kFlight; ++q)
                if (r[q] >= 0) x[q] = rows.load4(r[q], 4 * ch);
#pragma unroll
              for (int q = 0; q < kFlight; ++q)
                if (r[q] >= 0) { acc.x += x[q].x; acc.y += x[q].y; acc.z += x[q].z; acc.w += x[q].w; }
            }
            const float sc = bag_scale(a.combiner, k1 - k0);
            put(s0 + at, make_float4(acc.x * sc, acc.y * sc, acc.z * sc, acc.w * sc));
          }
          if (a.lin_col >= 0 && lane < n) {
            float lin = 0.f;
            for (int k = k0_lane; k < k1_lane; ++k) {
              const int r = rows.row(__ldg(a.inverse + k));
              if (r >= 0) lin += __ldcg(rows.base + (size_t)r * rows.stride + a.lin_col);
            }
            a.Lout[(size_t)b * S + s0 + lane] = lin * bag_scale(a.combiner, k1_lane - k0_lane);
          }
        }
      }
      if (part == wpe - 1) {
        const int tail0 = S * D;
        for (int j = lane; j < a.ld - tail0; j += 32) {
          float v = 0.f;
          if (j < a.Dd) v = a.dense[(size_t)b * a.ld_dense + j];
          else if (j == a.Dd) v = 1.f;
          xrow[tail0 + j] = __float2bfloat16(v);
          if (erow != nullptr && j < a.ldE - tail0) erow[tail0 + j] = v;
        }
      }
    }
    if (a.fm == nullptr) continue;
    for (int o = 16; o >= G; o >>= 1) {
      s.x += __shfl_xor_sync(0xffffffffu, s.x, o); s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
      s.z += __shfl_xor_sync(0xffffffffu, s.z, o); s.w += __shfl_xor_sync(0xffffffffu, s.w, o);
    }
    sq = warp_sum(sq);
    if (wpe > 1) {
      if (lane < G) s_sum[wib][lane] = s;
      if (lane == 0) s_sq[wib] = sq;
      __syncthreads();
      if (part == 0) {
        for (int w = 1; w < wpe; ++w) {
          const float4 x = s_sum[wib + w][ch];
          s.x += x.x; s.y += x.y; s.z += x.z; s.w += x.w;
          sq += s_sq[wib + w];
        }
      }
      __syncthreads();
    }
    if (part != 0 || b >= B) continue;
    const float t = warp_sum(lane < G ? s.x * s.x + s.y * s.y + s.z * s.z + s.w * s.w : 0.f) - sq;
    if (lane == 0) a.fm[b] = 0.5f * t;
    if (a.fsum != nullptr && lane < G && on) *reinterpret_cast<float4*>(a.fsum + ((size_t)b * ((D + 3) >> 2) + ch) * 4) = s;
  }
}

// One group of G lanes per bag, example after example, so that the operand's gradient and the pooled columns are read as they
// lie; kFlight bags on the way at once when every bag holds one id.  The field sums of the FM term come from the forward pass: no
// bag waits for another.  Columns from `dim` on (show / click) carry no gradient.  Bound by the latency of its loads (for which a
// warp waits ten of its fifteen cycles per instruction; L2 at 22 % of its rate, memory at 28 %): reductions into the rows are not waited for.
// 8192 x 26 slots of 16 with their linear weights 15.1 us (a warp per example 14.6).  In place of split, FM backward, additions and
// pooling backward: 2999 x 39 slots of 10, 8.4 us for 27 and four launches more; 4096 x 20 bags of three ids and 10 columns 9.9 for
// 14.5; 8192 x 100 bags of five ids and 64 columns 422 for 492.
template <bool kBags, int SV>
__global__ void __launch_bounds__(kThreads) embed_input_bwd_kernel(const __grid_constant__ EmbedGrad a, int G) {
  pdl_sync();
  constexpr int kQ = kBags ? 1 : kGradFlight;
  const int ch = threadIdx.x % G, S = a.S, D = a.D, B = a.B;
  const int nq = (D + 3) >> 2, ncol = D - 4 * ch, nred = min(a.dim, D) - 4 * ch;
  const int nbags = B * S;
  const int ngroups = gridDim.x * kThreads / G;
  const __nv_bfloat16* dX = reinterpret_cast<const __nv_bfloat16*>(a.dX0);
  for (int i0 = (blockIdx.x * kThreads + threadIdx.x) / G; i0 < nbags; i0 += kQ * ngroups) {
    int v[kQ], k0[kQ], k1[kQ];
    float4 g[kQ];
    float lin[kQ];
#pragma unroll
    for (int q = 0; q < kQ; ++q) {
      const long long i = i0 + (long long)q * ngroups;
      v[q] = -1; k0[q] = k1[q] = 0;
      lin[q] = 0.f;
      g[q] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (i >= nbags) continue;
      const int b = (int)i / S, s = (int)i - b * S;
      if constexpr (kBags) {
        k0[q] = __ldg(a.offsets + (size_t)s * B + b);
        k1[q] = __ldg(a.offsets + (size_t)s * B + b + 1);
      } else {
        v[q] = __ldg(a.inverse + (size_t)s * B + b);
      }
      if (a.dL != nullptr && ch == 0) lin[q] = a.dL[(size_t)b * S + s];
      if (nred <= 0) continue;
      const int col = s * D + 4 * ch;
      g[q] = load_bf16<SV>(dX + (size_t)b * a.ld + col, ncol);
      if (a.gfm != nullptr) {
        const float gf = __ldg(a.gfm + b);
        const float4 t = ldcg_f4(a.fsum + ((size_t)b * nq + ch) * 4), e = load_cols<SV>(a.E + (size_t)b * a.ldE + col, ncol);
        g[q].x += gf * (t.x - e.x); g[q].y += gf * (t.y - e.y); g[q].z += gf * (t.z - e.z); g[q].w += gf * (t.w - e.w);
      }
      if (a.gE != nullptr) {
        const float4 e = load_cols<SV>(a.gE + (size_t)b * a.ldE + col, ncol);
        g[q].x += e.x; g[q].y += e.y; g[q].z += e.z; g[q].w += e.w;
      }
    }
#pragma unroll
    for (int q = 0; q < kQ; ++q) {
      if constexpr (kBags) {
        const float sc = bag_scale(a.combiner, k1[q] - k0[q]);
        const float4 x = make_float4(g[q].x * sc, g[q].y * sc, g[q].z * sc, g[q].w * sc);
        const float l = lin[q] * sc;
        for (int k = k0[q]; k < k1[q]; k += kGradFlight) {
          int r[kGradFlight];
#pragma unroll
          for (int u = 0; u < kGradFlight; ++u) r[u] = k + u < k1[q] ? __ldg(a.inverse + k + u) : -1;
#pragma unroll
          for (int u = 0; u < kGradFlight; ++u) {
            if (r[u] < 0) continue;
            if (nred > 0) red_add_cols(a.gU + (size_t)r[u] * a.gstride + 4 * ch, x, nred);
            if (a.dL != nullptr && ch == 0) atomicAdd(a.gU + (size_t)r[u] * a.gstride + a.lin_col, l);
          }
        }
      } else {
        if (v[q] < 0) continue;
        const float sc = bag_scale(a.combiner, 1);
        if (nred > 0)
          red_add_cols(a.gU + (size_t)v[q] * a.gstride + 4 * ch, make_float4(g[q].x * sc, g[q].y * sc, g[q].z * sc, g[q].w * sc), nred);
        if (a.dL != nullptr && ch == 0) atomicAdd(a.gU + (size_t)v[q] * a.gstride + a.lin_col, lin[q] * sc);
      }
    }
  }
}

// Columns that move at a time: the operand's, the pooled columns' and their gradient's address allow it.
int cols_at_once(int D, int ld, int ldE, const void* bf16, const void* f32a, const void* f32b) {
  ld |= f32a != nullptr || f32b != nullptr ? ldE : 0;
  const uintptr_t h = reinterpret_cast<uintptr_t>(bf16), f = reinterpret_cast<uintptr_t>(f32a) | reinterpret_cast<uintptr_t>(f32b);
  if (((D | ld) & 3) == 0 && (h & 7) == 0 && (f & 15) == 0) return 4;
  return ((D | ld) & 1) == 0 && (h & 3) == 0 && (f & 7) == 0 ? 2 : 1;
}

template <bool kInPlace, bool kBags, int kFlight>
auto fwd_kernel(int sv) {
  return sv == 4   ? embed_input_fwd_kernel<kInPlace, kBags, 4, kFlight>
         : sv == 2 ? embed_input_fwd_kernel<kInPlace, kBags, 2, kFlight>
                   : embed_input_fwd_kernel<kInPlace, kBags, 1, kFlight>;
}
template <bool kBags>
auto bwd_kernel(int sv) {
  return sv == 4 ? embed_input_bwd_kernel<kBags, 4> : sv == 2 ? embed_input_bwd_kernel<kBags, 2> : embed_input_bwd_kernel<kBags, 1>;
}

}  // namespace

const char* launch_embed_input_fwd(const RowSource& src, const EmbedInput& a, cudaStream_t st) {
  if (a.D < 1 || a.D > kEmbedInputColumns) return "embed_input: slots of 1 to 128 columns";
  if (a.ld < a.S * a.D + a.Dd + 1 || (a.E != nullptr && (a.ldE < a.S * a.D || a.ldE > a.S * a.D + a.Dd))) return "embed_input: row length";
  if (a.B < 1 || a.S < 1) return nullptr;
  const int G = lanes_for_width(a.D);
  // Warps per example: one where that gives every SM sixteen of them, else as many as have a full turn of slots each.
  int wpe = 1;
  while (wpe < kWarps && (long long)a.B * wpe < 148 * 16 && a.S > wpe * 2 * (32 / G)) wpe <<= 1;
  const int epb = kWarps / wpe;
  int blocks = (a.B + epb - 1) / epb;
  if (blocks > 148 * 8) blocks = 148 * 8;
  const int sv = cols_at_once(a.D, a.ld, a.ldE, a.X0, a.E, nullptr);
  const bool in_place = src.tbl != nullptr;
  // Turns of a warp's groups on the way at once: eight groups or four move enough with two (213 K rows of 16: 17.8 us, with four
  // 18.7), wider rows and bags take four (8192 x 100 bags of five ids and 64 columns: 330 us, with two 440).
  auto* k = a.offsets != nullptr ? (in_place ? fwd_kernel<true, true, 4>(sv) : fwd_kernel<false, true, 4>(sv))
            : G <= 8             ? (in_place ? fwd_kernel<true, false, 2>(sv) : fwd_kernel<false, false, 2>(sv))
                                 : (in_place ? fwd_kernel<true, false, 4>(sv) : fwd_kernel<false, false, 4>(sv));
  const cudaError_t e = launch_pdl(k, dim3(blocks), dim3(kThreads), 0, st, src, a, G, wpe);
  return e == cudaSuccess ? nullptr : cudaGetErrorString(e);
}
const char* launch_embed_input_bwd(const EmbedGrad& a, cudaStream_t st) {
  if (a.D < 1 || a.D > kEmbedInputColumns) return "embed_input: slots of 1 to 128 columns";
  if (a.B < 1 || a.S < 1) return nullptr;
  const int G = lanes_for_width(a.D);
  const long long bags = (long long)a.B * a.S;
  // several bags of one id each once one bag per group already fills the chip
  const long long groups = a.offsets == nullptr && bags * G >= 148ll * 2048 * kGradFlight ? (bags + kGradFlight - 1) / kGradFlight : bags;
  long long blocks = (groups * G + kThreads - 1) / kThreads;
  if (blocks > 148 * 16) blocks = 148 * 16;
  const int sv = cols_at_once(a.D, a.ld, a.ldE, a.dX0, a.E, a.gE);
  const cudaError_t e = launch_pdl(a.offsets != nullptr ? bwd_kernel<true>(sv) : bwd_kernel<false>(sv), dim3((unsigned)blocks), dim3(kThreads), 0, st, a, G);
  return e == cudaSuccess ? nullptr : cudaGetErrorString(e);
}

}  // namespace tn
