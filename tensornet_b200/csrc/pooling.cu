// Bag pooling over the per-batch unique-row matrix and its backward into the unique
// gradient matrix, plus the un-pooled sequence gather.  Stands in for TensorFlow's
// safe_embedding_lookup_sparse / sequence lookups that the reference calls on its batch
// variable (tensornet/layers/embedding_features.py:283-284,
// tensornet/layers/sequence_embedding_features.py:99-137).
#include "tn_device.cuh"
#include "tn_ops.h"

namespace tn {

namespace {

__device__ __forceinline__ float bag_scale(int combiner, int len) {
  if (len <= 0) return 0.f;
  if (combiner == 1) return 1.f / (float)len;
  if (combiner == 2) return rsqrtf((float)len);
  return 1.f;
}

// One group of G lanes per bag.  Bag g = s * B + b, its ids are positions
// [offsets[g], offsets[g+1]) of `inverse` (or exactly position g when offsets == nullptr).
__global__ void pool_fwd_kernel(const float* __restrict__ U, int ustride, const int* __restrict__ inverse,
                                const int* __restrict__ offsets, int B, int S, int pd, int combiner,
                                float* __restrict__ out, int out_ld, int G) {
  pdl_sync();
  const int lane = threadIdx.x % G;
  const int gid = (blockIdx.x * blockDim.x + threadIdx.x) / G;
  const int ngroups = (gridDim.x * blockDim.x) / G;
  const int nbags = B * S;
  for (int g = gid; g < nbags; g += ngroups) {
    const int s = g / B, b = g - s * B;
    int k0 = g, k1 = g + 1;
    if (offsets) { k0 = offsets[g]; k1 = offsets[g + 1]; }
    const float sc = bag_scale(combiner, k1 - k0);
    float* o = out + (size_t)b * out_ld + (size_t)s * pd;
    for (int d = lane; d < pd; d += G) {
      float acc = 0.f;
      for (int k = k0; k < k1; ++k) {
        int v = inverse[k];
        if (v >= 0) acc += __ldcg(U + (size_t)v * ustride + d);
      }
      o[d] = acc * sc;
    }
  }
}

// The variants for pd % 4 == 0: every lane moves float4 chunks.  Bound by random row reads (or reductions), so a group of
// lanes keeps kPoolFlight of them in flight: that many bags when every bag holds one id, that many ids of a bag
// otherwise.  Ids of a bag are added in their order, one after the other, whatever the number in flight.
// 2.1 M single-id bags of 128: forward 399 us with one row at a time, 316 now; backward 474 us, 445 now.  0.8 M bags of
// five ids and 64 columns: forward 251 -> 205 us (5.1 to 6.2 TB/s), backward unchanged: the reductions bound it.
constexpr int kPoolFlight = 4;

__global__ void __launch_bounds__(256) pool_fwd_single_vec4_kernel(const float* __restrict__ U, int ustride,
                                                                   const int* __restrict__ inverse, int B, int S, int pd,
                                                                   int combiner, float* __restrict__ out, int out_ld, int G) {
  pdl_sync();
  const int lane = threadIdx.x % G;
  const int gid = (blockIdx.x * blockDim.x + threadIdx.x) / G;
  const int ngroups = (gridDim.x * blockDim.x) / G;
  const int nbags = B * S, nch = pd >> 2;
  const float sc = bag_scale(combiner, 1);
  for (long long g0 = gid; g0 < nbags; g0 += (long long)kPoolFlight * ngroups) {
    int v[kPoolFlight];
    float* o[kPoolFlight];
#pragma unroll
    for (int q = 0; q < kPoolFlight; ++q) {
      const long long gl = g0 + (long long)q * ngroups;
      o[q] = nullptr;
      v[q] = -1;
      if (gl < nbags) {
        const int g = (int)gl, s = g / B, b = g - s * B;
        v[q] = __ldg(inverse + g);
        o[q] = out + (size_t)b * out_ld + (size_t)s * pd;
      }
    }
    for (int ch = lane; ch < nch; ch += G) {
      float4 x[kPoolFlight];
#pragma unroll
      for (int q = 0; q < kPoolFlight; ++q) {
        x[q] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (v[q] >= 0) x[q] = ldcg_f4(U + (size_t)v[q] * ustride + 4 * ch);
      }
#pragma unroll
      for (int q = 0; q < kPoolFlight; ++q) {
        if (o[q] != nullptr)
          *reinterpret_cast<float4*>(o[q] + 4 * ch) = make_float4(x[q].x * sc, x[q].y * sc, x[q].z * sc, x[q].w * sc);
      }
    }
  }
}

__global__ void __launch_bounds__(256) pool_fwd_bags_vec4_kernel(const float* __restrict__ U, int ustride,
                                                                 const int* __restrict__ inverse, const int* __restrict__ offsets,
                                                                 int B, int S, int pd, int combiner, float* __restrict__ out,
                                                                 int out_ld, int G) {
  pdl_sync();
  const int lane = threadIdx.x % G;
  const int gid = (blockIdx.x * blockDim.x + threadIdx.x) / G;
  const int ngroups = (gridDim.x * blockDim.x) / G;
  const int nbags = B * S, nch = pd >> 2;
  for (int g = gid; g < nbags; g += ngroups) {
    const int s = g / B, b = g - s * B;
    const int k0 = offsets[g], k1 = offsets[g + 1];
    const float sc = bag_scale(combiner, k1 - k0);
    float* o = out + (size_t)b * out_ld + (size_t)s * pd;
    for (int ch = lane; ch < nch; ch += G) {
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int k = k0; k < k1; k += kPoolFlight) {
        int v[kPoolFlight];
        float4 x[kPoolFlight];
#pragma unroll
        for (int q = 0; q < kPoolFlight; ++q) v[q] = k + q < k1 ? __ldg(inverse + k + q) : -1;
#pragma unroll
        for (int q = 0; q < kPoolFlight; ++q)
          if (v[q] >= 0) x[q] = ldcg_f4(U + (size_t)v[q] * ustride + 4 * ch);
#pragma unroll
        for (int q = 0; q < kPoolFlight; ++q)
          if (v[q] >= 0) { acc.x += x[q].x; acc.y += x[q].y; acc.z += x[q].z; acc.w += x[q].w; }
      }
      acc.x *= sc; acc.y *= sc; acc.z *= sc; acc.w *= sc;
      *reinterpret_cast<float4*>(o + 4 * ch) = acc;
    }
  }
}

// dim % 4 == 0 and pd % 4 == 0: vector reductions into the unique-gradient rows.
__global__ void __launch_bounds__(256) pool_bwd_single_vec4_kernel(float* __restrict__ gU, int gstride,
                                                                   const int* __restrict__ inverse, int B, int S, int pd, int dim,
                                                                   int combiner, const float* __restrict__ gout, int gout_ld, int G) {
  pdl_sync();
  const int lane = threadIdx.x % G;
  const int gid = (blockIdx.x * blockDim.x + threadIdx.x) / G;
  const int ngroups = (gridDim.x * blockDim.x) / G;
  const int nbags = B * S, nch = dim >> 2;
  const float sc = bag_scale(combiner, 1);
  for (long long g0 = gid; g0 < nbags; g0 += (long long)kPoolFlight * ngroups) {
    int v[kPoolFlight];
    const float* go[kPoolFlight];
#pragma unroll
    for (int q = 0; q < kPoolFlight; ++q) {
      const long long gl = g0 + (long long)q * ngroups;
      v[q] = -1;
      go[q] = gout;
      if (gl < nbags) {
        const int g = (int)gl, s = g / B, b = g - s * B;
        v[q] = __ldg(inverse + g);
        go[q] = gout + (size_t)b * gout_ld + (size_t)s * pd;
      }
    }
    for (int ch = lane; ch < nch; ch += G) {
      float4 x[kPoolFlight];
#pragma unroll
      for (int q = 0; q < kPoolFlight; ++q)
        if (v[q] >= 0) x[q] = *reinterpret_cast<const float4*>(go[q] + 4 * ch);
#pragma unroll
      for (int q = 0; q < kPoolFlight; ++q)
        if (v[q] >= 0)
          red_add_f32x4(gU + (size_t)v[q] * gstride + 4 * ch, make_float4(x[q].x * sc, x[q].y * sc, x[q].z * sc, x[q].w * sc));
    }
  }
}

__global__ void __launch_bounds__(256) pool_bwd_bags_vec4_kernel(float* __restrict__ gU, int gstride,
                                                                 const int* __restrict__ inverse, const int* __restrict__ offsets,
                                                                 int B, int S, int pd, int dim, int combiner,
                                                                 const float* __restrict__ gout, int gout_ld, int G) {
  pdl_sync();
  const int lane = threadIdx.x % G;
  const int gid = (blockIdx.x * blockDim.x + threadIdx.x) / G;
  const int ngroups = (gridDim.x * blockDim.x) / G;
  const int nbags = B * S, nch = dim >> 2;
  for (int g = gid; g < nbags; g += ngroups) {
    const int s = g / B, b = g - s * B;
    const int k0 = offsets[g], k1 = offsets[g + 1];
    const float sc = bag_scale(combiner, k1 - k0);
    const float* go = gout + (size_t)b * gout_ld + (size_t)s * pd;
    for (int ch = lane; ch < nch; ch += G) {
      float4 x = *reinterpret_cast<const float4*>(go + 4 * ch);
      x.x *= sc; x.y *= sc; x.z *= sc; x.w *= sc;
      for (int k = k0; k < k1; k += kPoolFlight) {
        int v[kPoolFlight];
#pragma unroll
        for (int q = 0; q < kPoolFlight; ++q) v[q] = k + q < k1 ? __ldg(inverse + k + q) : -1;
#pragma unroll
        for (int q = 0; q < kPoolFlight; ++q)
          if (v[q] >= 0) red_add_f32x4(gU + (size_t)v[q] * gstride + 4 * ch, x);
      }
    }
  }
}

__global__ void pool_bwd_kernel(float* __restrict__ gU, int gstride, const int* __restrict__ inverse,
                                const int* __restrict__ offsets, int B, int S, int pd, int dim, int combiner,
                                const float* __restrict__ gout, int gout_ld, int G) {
  pdl_sync();
  const int lane = threadIdx.x % G;
  const int gid = (blockIdx.x * blockDim.x + threadIdx.x) / G;
  const int ngroups = (gridDim.x * blockDim.x) / G;
  const int nbags = B * S;
  for (int g = gid; g < nbags; g += ngroups) {
    const int s = g / B, b = g - s * B;
    int k0 = g, k1 = g + 1;
    if (offsets) { k0 = offsets[g]; k1 = offsets[g + 1]; }
    const float sc = bag_scale(combiner, k1 - k0);
    const float* go = gout + (size_t)b * gout_ld + (size_t)s * pd;
    for (int d = lane; d < dim; d += G) {   // CVM columns (d >= dim) carry no gradient
      const float x = go[d] * sc;
      for (int k = k0; k < k1; ++k) {
        int v = inverse[k];
        if (v >= 0) atomicAdd(gU + (size_t)v * gstride + d, x);
      }
    }
  }
}

// Sequence gather of one column: element t of example b -> out[b, t, :]; t >= T is dropped,
// positions past the length stay zero (caller zero-fills).  lengths[b] = min(len, T).
__global__ void seq_fwd_kernel(const float* __restrict__ U, int ustride, const int* __restrict__ inverse,
                               const int* __restrict__ offsets, int B, int T, int pd, float* __restrict__ out,
                               int* __restrict__ lengths, int G) {
  pdl_sync();
  const int lane = threadIdx.x % G;
  const int gid = (blockIdx.x * blockDim.x + threadIdx.x) / G;
  const int ngroups = (gridDim.x * blockDim.x) / G;
  for (int g = gid; g < B * T; g += ngroups) {
    const int b = g / T, tt = g - b * T;
    const int k0 = offsets[b], len = offsets[b + 1] - k0;
    if (tt == 0 && lane == 0 && lengths) lengths[b] = len < T ? len : T;
    if (tt >= len) continue;
    const int v = inverse[k0 + tt];
    float* o = out + ((size_t)b * T + tt) * pd;
    for (int d = lane; d < pd; d += G) o[d] = v >= 0 ? __ldcg(U + (size_t)v * ustride + d) : 0.f;
  }
}

__global__ void seq_bwd_kernel(float* __restrict__ gU, int gstride, const int* __restrict__ inverse,
                               const int* __restrict__ offsets, int B, int T, int pd, int dim,
                               const float* __restrict__ gout, int G) {
  pdl_sync();
  const int lane = threadIdx.x % G;
  const int gid = (blockIdx.x * blockDim.x + threadIdx.x) / G;
  const int ngroups = (gridDim.x * blockDim.x) / G;
  for (int g = gid; g < B * T; g += ngroups) {
    const int b = g / T, tt = g - b * T;
    const int k0 = offsets[b], len = offsets[b + 1] - k0;
    if (tt >= len) continue;
    const int v = inverse[k0 + tt];
    if (v < 0) continue;
    const float* go = gout + ((size_t)b * T + tt) * pd;
    for (int d = lane; d < dim; d += G) atomicAdd(gU + (size_t)v * gstride + d, go[d]);
  }
}

// Per id the label of its example: one thread per bag writes its bag's few entries.
__global__ void expand_bag_labels_kernel(const float* __restrict__ y, const int* __restrict__ offsets, int B, int nbags,
                                         float* __restrict__ out, int room) {
  for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < nbags; g += gridDim.x * blockDim.x) {
    const float v = y[g % B];
    const int k1 = min(offsets[g + 1], room);
    for (int k = max(offsets[g], 0); k < k1; ++k) out[k] = v;
  }
}

__device__ __forceinline__ long long index_at(const void* p, int is64, long long i) {
  return is64 ? reinterpret_cast<const long long*>(p)[i] : (long long)reinterpret_cast<const int*>(p)[i];
}

// Columns -> packed (values, offsets).  blockIdx.y = column; where it starts is the sum of the counts of the columns
// before it, which only the device knows in a captured step: every block adds them up itself (a few hundred L2 reads),
// which is cheaper than a second launch.  `first` columns of an earlier launch end at out_offsets[first * B].
__global__ void pack_columns_kernel(const __grid_constant__ PackColumns a) {
  __shared__ long long s_base;
  const int c = blockIdx.y, B = a.B;
  if (threadIdx.x == 0) s_base = a.first > 0 ? a.out_offsets[(size_t)a.first * B] : 0;
  __syncthreads();
  long long before = 0;
  for (int j = threadIdx.x; j < c; j += blockDim.x)
    before += a.offsets[j] != nullptr ? index_at(a.offsets[j], a.off64[j], B) : (long long)a.len[j] * B;
  for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
  if ((threadIdx.x & 31) == 0 && before) atomicAdd(reinterpret_cast<unsigned long long*>(&s_base), (unsigned long long)before);
  __syncthreads();
  const long long base = s_base;
  const void* off = a.offsets[c];
  long long n = off != nullptr ? index_at(off, a.off64[c], B) : (long long)a.len[c] * B;
  if (n > a.room[c]) n = a.room[c];
  const int t0 = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
  for (long long k = t0; k < n && base + k < a.total_room; k += nt) a.out_values[base + k] = index_at(a.values[c], a.val64[c], k);
  const size_t row = (size_t)(a.first + c) * B;
  for (int b = t0; b < B; b += nt)
    a.out_offsets[row + b] = (int)(base + (off != nullptr ? index_at(off, a.off64[c], b) : (long long)a.len[c] * b));
  if (t0 == 0) a.out_offsets[row + B] = (int)(base + n);       // the next column writes the same value as its start
}

inline int grid_for(long long groups, int G, int threads) {
  long long blocks = (groups * G + threads - 1) / threads;
  if (blocks < 1) blocks = 1;
  if (blocks > 148 * 16) blocks = 148 * 16;
  return (int)blocks;
}

// Groups for bags of one id: several bags each once one bag per group already fills the chip, else one bag each.
inline long long single_groups(long long bags, int G) {
  return bags * G >= 148ll * 2048 * kPoolFlight ? (bags + kPoolFlight - 1) / kPoolFlight : bags;
}

}  // namespace

void launch_expand_bag_labels(const float* y, const int* offsets, int B, int nbags, float* out, int room, cudaStream_t st) {
  expand_bag_labels_kernel<<<grid_for(nbags, 1, 256), 256, 0, st>>>(y, offsets, B, nbags, out, room);
}
void launch_pack_columns(const PackColumns& a, cudaStream_t st) {
  long long most = a.B;
  for (int c = 0; c < a.n; ++c) most = a.room[c] > most ? a.room[c] : most;
  int bx = (int)((most + 1023) / 1024);          // four elements per thread of the longest column
  if (bx > 64) bx = 64;
  pack_columns_kernel<<<dim3(bx < 1 ? 1 : bx, a.n), 256, 0, st>>>(a);
}

void launch_pool_fwd(const float* U, int ustride, const int* inverse, const int* offsets, int B, int S, int pd,
                     int combiner, float* out, int out_ld, cudaStream_t st) {
  if ((pd & 3) == 0 && (out_ld & 3) == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0) {
    const int G = lanes_for_width(pd);
    if (offsets == nullptr)
      launch_pdl(pool_fwd_single_vec4_kernel, dim3(grid_for(single_groups((long long)B * S, G), G, 256)), dim3(256), 0, st, U, ustride,
                 inverse, B, S, pd, combiner, out, out_ld, G);
    else
      launch_pdl(pool_fwd_bags_vec4_kernel, dim3(grid_for((long long)B * S, G, 256)), dim3(256), 0, st, U, ustride, inverse, offsets, B, S,
                 pd, combiner, out, out_ld, G);
    return;
  }
  int G = pd >= 32 ? 32 : (pd >= 16 ? 16 : (pd >= 8 ? 8 : (pd >= 4 ? 4 : (pd >= 2 ? 2 : 1))));
  launch_pdl(pool_fwd_kernel, dim3(grid_for((long long)B * S, G, 256)), dim3(256), 0, st, U, ustride, inverse, offsets, B, S, pd, combiner,
                                                                        out, out_ld, G);
}
void launch_pool_bwd(float* gU, int gstride, const int* inverse, const int* offsets, int B, int S, int pd, int dim,
                     int combiner, const float* gout, int gout_ld, cudaStream_t st) {
  if ((pd & 3) == 0 && (dim & 3) == 0 && (gout_ld & 3) == 0 && (reinterpret_cast<uintptr_t>(gout) & 15) == 0) {
    const int G = lanes_for_width(dim);
    if (offsets == nullptr)
      launch_pdl(pool_bwd_single_vec4_kernel, dim3(grid_for(single_groups((long long)B * S, G), G, 256)), dim3(256), 0, st, gU, gstride,
                 inverse, B, S, pd, dim, combiner, gout, gout_ld, G);
    else
      launch_pdl(pool_bwd_bags_vec4_kernel, dim3(grid_for((long long)B * S, G, 256)), dim3(256), 0, st, gU, gstride, inverse, offsets, B,
                 S, pd, dim, combiner, gout, gout_ld, G);
    return;
  }
  int G = dim >= 32 ? 32 : (dim >= 16 ? 16 : (dim >= 8 ? 8 : (dim >= 4 ? 4 : (dim >= 2 ? 2 : 1))));
  launch_pdl(pool_bwd_kernel, dim3(grid_for((long long)B * S, G, 256)), dim3(256), 0, st, gU, gstride, inverse, offsets, B, S, pd, dim,
                                                                        combiner, gout, gout_ld, G);
}
void launch_seq_fwd(const float* U, int ustride, const int* inverse, const int* offsets, int B, int T, int pd,
                    float* out, int* lengths, cudaStream_t st) {
  int G = pd >= 32 ? 32 : (pd >= 16 ? 16 : (pd >= 8 ? 8 : (pd >= 4 ? 4 : (pd >= 2 ? 2 : 1))));
  launch_pdl(seq_fwd_kernel, dim3(grid_for((long long)B * T, G, 256)), dim3(256), 0, st, U, ustride, inverse, offsets, B, T, pd, out,
                                                                       lengths, G);
}
void launch_seq_bwd(float* gU, int gstride, const int* inverse, const int* offsets, int B, int T, int pd, int dim,
                    const float* gout, cudaStream_t st) {
  int G = dim >= 32 ? 32 : (dim >= 16 ? 16 : (dim >= 8 ? 8 : (dim >= 4 ? 4 : (dim >= 2 ? 2 : 1))));
  launch_pdl(seq_bwd_kernel, dim3(grid_for((long long)B * T, G, 256)), dim3(256), 0, st, gU, gstride, inverse, offsets, B, T, pd, dim, gout, G);
}

}  // namespace tn
