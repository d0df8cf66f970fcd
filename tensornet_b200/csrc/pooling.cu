// Bag pooling over the per-batch unique-row matrix and its backward into the unique
// gradient matrix, plus the un-pooled sequence gather.  Stands in for TensorFlow's
// safe_embedding_lookup_sparse / sequence lookups that the reference calls on its batch
// variable (tensornet/layers/embedding_features.py:283-284,
// tensornet/layers/sequence_embedding_features.py:99-137).
#include "sparse_table.cuh"
#include "tn_ops.h"

namespace tn {

namespace {

__device__ __forceinline__ float bag_scale(int combiner, int len) {
  if (len <= 0) return 0.f;
  if (combiner == 1) return 1.f / (float)len;
  if (combiner == 2) return rsqrtf((float)len);
  return 1.f;
}

// One group of G lanes per bag, a lane moves four columns at a time: rows and gradient rows are whole 16-byte pieces whatever
// their width, only the pooled columns are written (and their gradient read) SV = 4, 2 or 1 at a time, as their address
// allows.  Bag g = s * B + b, its ids are positions [offsets[g], offsets[g+1]) of `inverse` (or exactly position g when
// offsets == nullptr).  Bound by random row reads (or reductions), so a group keeps kPoolFlight of them in flight: that many
// bags when every bag holds one id, that many ids of a bag otherwise.  Ids of a bag are added in their order, one after
// the other, whatever the number in flight.
// 2.1 M single-id bags of 128: forward 399 us with one row at a time, 312 now (326 with the rows read in place, a
// dependent load more but no copy of the rows beforehand); backward 474 us, 445 now.  0.8 M bags of five ids and 64
// columns: forward 251 -> 205 us (5.1 to 6.2 TB/s), backward unchanged: the reductions bound it.
constexpr int kPoolFlight = 4;

template <bool kInPlace, int SV>
__global__ void __launch_bounds__(256, 6) pool_fwd_single_kernel(const RowSource src, const int* __restrict__ inverse, int B, int S,
                                                                 int pd, int combiner, float* __restrict__ out, int out_ld, int G) {
  const PulledRows<kInPlace> rows(src);
  pdl_sync();
  const int lane = threadIdx.x % G;
  const int gid = (blockIdx.x * blockDim.x + threadIdx.x) / G;
  const int ngroups = (gridDim.x * blockDim.x) / G;
  const int nbags = B * S;
  const float sc = bag_scale(combiner, 1);
  for (long long g0 = gid; g0 < nbags; g0 += (long long)kPoolFlight * ngroups) {
    int r[kPoolFlight];
#pragma unroll
    for (int q = 0; q < kPoolFlight; ++q) {
      const long long g = g0 + (long long)q * ngroups;
      r[q] = g < nbags ? __ldg(inverse + g) : -1;
    }
#pragma unroll
    for (int q = 0; q < kPoolFlight; ++q) r[q] = rows.row(r[q]);
    for (int d = 4 * lane; d < pd; d += 4 * G) {
      float4 x[kPoolFlight];
#pragma unroll
      for (int q = 0; q < kPoolFlight; ++q) {
        x[q] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r[q] >= 0) x[q] = rows.load4(r[q], d);
      }
#pragma unroll
      for (int q = 0; q < kPoolFlight; ++q) {
        const long long g = g0 + (long long)q * ngroups;
        if (g >= nbags) continue;
        const int s = (int)g / B, b = (int)g - s * B;
        store_cols<SV>(out + (size_t)b * out_ld + (size_t)s * pd + d, make_float4(x[q].x * sc, x[q].y * sc, x[q].z * sc, x[q].w * sc), pd - d);
      }
    }
  }
}

template <bool kInPlace, int SV>
__global__ void __launch_bounds__(256, 5) pool_fwd_bags_kernel(const RowSource src, const int* __restrict__ inverse,
                                                               const int* __restrict__ offsets, int B, int S, int pd, int combiner,
                                                               float* __restrict__ out, int out_ld, int G) {
  const PulledRows<kInPlace> rows(src);
  pdl_sync();
  const int lane = threadIdx.x % G;
  const int gid = (blockIdx.x * blockDim.x + threadIdx.x) / G;
  const int ngroups = (gridDim.x * blockDim.x) / G;
  const int nbags = B * S;
  for (int g = gid; g < nbags; g += ngroups) {
    const int s = g / B, b = g - s * B;
    const int k0 = offsets[g], k1 = offsets[g + 1];
    const float sc = bag_scale(combiner, k1 - k0);
    float* o = out + (size_t)b * out_ld + (size_t)s * pd;
    for (int d = 4 * lane; d < pd; d += 4 * G) {
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int k = k0; k < k1; k += kPoolFlight) {
        int r[kPoolFlight];
        float4 x[kPoolFlight];
#pragma unroll
        for (int q = 0; q < kPoolFlight; ++q) r[q] = k + q < k1 ? __ldg(inverse + k + q) : -1;
#pragma unroll
        for (int q = 0; q < kPoolFlight; ++q) r[q] = rows.row(r[q]);
#pragma unroll
        for (int q = 0; q < kPoolFlight; ++q)
          if (r[q] >= 0) x[q] = rows.load4(r[q], d);
#pragma unroll
        for (int q = 0; q < kPoolFlight; ++q)
          if (r[q] >= 0) { acc.x += x[q].x; acc.y += x[q].y; acc.z += x[q].z; acc.w += x[q].w; }
      }
      acc.x *= sc; acc.y *= sc; acc.z *= sc; acc.w *= sc;
      store_cols<SV>(o + d, acc, pd - d);
    }
  }
}

// Backward: vector reductions into the unique-gradient rows.  CVM columns (d >= dim) carry no gradient.
template <int SV>
__global__ void __launch_bounds__(256) pool_bwd_single_kernel(float* __restrict__ gU, int gstride, const int* __restrict__ inverse,
                                                              int B, int S, int pd, int dim, int combiner,
                                                              const float* __restrict__ gout, int gout_ld, int G) {
  pdl_sync();
  const int lane = threadIdx.x % G;
  const int gid = (blockIdx.x * blockDim.x + threadIdx.x) / G;
  const int ngroups = (gridDim.x * blockDim.x) / G;
  const int nbags = B * S;
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
    for (int d = 4 * lane; d < dim; d += 4 * G) {
      float4 x[kPoolFlight];
#pragma unroll
      for (int q = 0; q < kPoolFlight; ++q)
        if (v[q] >= 0) x[q] = load_cols<SV>(go[q] + d, dim - d);
#pragma unroll
      for (int q = 0; q < kPoolFlight; ++q)
        if (v[q] >= 0)
          red_add_cols(gU + (size_t)v[q] * gstride + d, make_float4(x[q].x * sc, x[q].y * sc, x[q].z * sc, x[q].w * sc), dim - d);
    }
  }
}

template <int SV>
__global__ void __launch_bounds__(256) pool_bwd_bags_kernel(float* __restrict__ gU, int gstride, const int* __restrict__ inverse,
                                                            const int* __restrict__ offsets, int B, int S, int pd, int dim,
                                                            int combiner, const float* __restrict__ gout, int gout_ld, int G) {
  pdl_sync();
  const int lane = threadIdx.x % G;
  const int gid = (blockIdx.x * blockDim.x + threadIdx.x) / G;
  const int ngroups = (gridDim.x * blockDim.x) / G;
  const int nbags = B * S;
  for (int g = gid; g < nbags; g += ngroups) {
    const int s = g / B, b = g - s * B;
    const int k0 = offsets[g], k1 = offsets[g + 1];
    const float sc = bag_scale(combiner, k1 - k0);
    const float* go = gout + (size_t)b * gout_ld + (size_t)s * pd;
    for (int d = 4 * lane; d < dim; d += 4 * G) {
      float4 x = load_cols<SV>(go + d, dim - d);
      x.x *= sc; x.y *= sc; x.z *= sc; x.w *= sc;
      for (int k = k0; k < k1; k += kPoolFlight) {
        int v[kPoolFlight];
#pragma unroll
        for (int q = 0; q < kPoolFlight; ++q) v[q] = k + q < k1 ? __ldg(inverse + k + q) : -1;
#pragma unroll
        for (int q = 0; q < kPoolFlight; ++q)
          if (v[q] >= 0) red_add_cols(gU + (size_t)v[q] * gstride + d, x, dim - d);
      }
    }
  }
}

// Sequence gather of one column: element t of example b -> out[b, t, :]; t >= T is dropped,
// positions past the length stay zero (caller zero-fills).  lengths[b] = min(len, T).
template <bool kInPlace>
__global__ void seq_fwd_kernel(const RowSource src, const int* __restrict__ inverse, const int* __restrict__ offsets, int B, int T,
                               int pd, float* __restrict__ out, int* __restrict__ lengths, int G) {
  const PulledRows<kInPlace> rows(src);
  pdl_sync();
  const int lane = threadIdx.x % G;
  const int gid = (blockIdx.x * blockDim.x + threadIdx.x) / G;
  const int ngroups = (gridDim.x * blockDim.x) / G;
  for (int g = gid; g < B * T; g += ngroups) {
    const int b = g / T, tt = g - b * T;
    const int k0 = offsets[b], len = offsets[b + 1] - k0;
    if (tt == 0 && lane == 0 && lengths) lengths[b] = len < T ? len : T;
    if (tt >= len) continue;
    const int r = rows.row(inverse[k0 + tt]);
    float* o = out + ((size_t)b * T + tt) * pd;
    for (int d = 4 * lane; d < pd; d += 4 * G)
      store_cols<1>(o + d, r >= 0 ? rows.load4(r, d) : make_float4(0.f, 0.f, 0.f, 0.f), pd - d);
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

// Columns that move at a time where bags lie in memory next to each other: 4, 2 or 1.
static int cols_at_once(int pd, int ld, const void* p) {
  const int all = pd | ld;
  const uintptr_t at = reinterpret_cast<uintptr_t>(p);
  return (all & 3) == 0 && (at & 15) == 0 ? 4 : (all & 1) == 0 && (at & 7) == 0 ? 2 : 1;
}

template <bool kInPlace, int SV>
static void pool_fwd(const RowSource& src, const int* inverse, const int* offsets, int B, int S, int pd, int combiner, float* out,
                     int out_ld, cudaStream_t st) {
  const int G = lanes_for_width(pd);
  const long long bags = (long long)B * S;
  if (offsets == nullptr)
    launch_pdl(pool_fwd_single_kernel<kInPlace, SV>, dim3(grid_for(single_groups(bags, G), G, 256)), dim3(256), 0, st, src, inverse, B, S,
               pd, combiner, out, out_ld, G);
  else
    launch_pdl(pool_fwd_bags_kernel<kInPlace, SV>, dim3(grid_for(bags, G, 256)), dim3(256), 0, st, src, inverse, offsets, B, S, pd,
               combiner, out, out_ld, G);
}
void launch_pool_fwd(const RowSource& src, const int* inverse, const int* offsets, int B, int S, int pd, int combiner, float* out,
                     int out_ld, cudaStream_t st) {
  const bool in_place = src.tbl != nullptr;
  switch (cols_at_once(pd, out_ld, out)) {
    case 4: (in_place ? pool_fwd<true, 4> : pool_fwd<false, 4>)(src, inverse, offsets, B, S, pd, combiner, out, out_ld, st); break;
    case 2: (in_place ? pool_fwd<true, 2> : pool_fwd<false, 2>)(src, inverse, offsets, B, S, pd, combiner, out, out_ld, st); break;
    default: (in_place ? pool_fwd<true, 1> : pool_fwd<false, 1>)(src, inverse, offsets, B, S, pd, combiner, out, out_ld, st);
  }
}

template <int SV>
static void pool_bwd(float* gU, int gstride, const int* inverse, const int* offsets, int B, int S, int pd, int dim, int combiner,
                     const float* gout, int gout_ld, cudaStream_t st) {
  const int G = lanes_for_width(dim);
  const long long bags = (long long)B * S;
  if (offsets == nullptr)
    launch_pdl(pool_bwd_single_kernel<SV>, dim3(grid_for(single_groups(bags, G), G, 256)), dim3(256), 0, st, gU, gstride, inverse, B, S, pd,
               dim, combiner, gout, gout_ld, G);
  else
    launch_pdl(pool_bwd_bags_kernel<SV>, dim3(grid_for(bags, G, 256)), dim3(256), 0, st, gU, gstride, inverse, offsets, B, S, pd, dim,
               combiner, gout, gout_ld, G);
}
void launch_pool_bwd(float* gU, int gstride, const int* inverse, const int* offsets, int B, int S, int pd, int dim,
                     int combiner, const float* gout, int gout_ld, cudaStream_t st) {
  switch (cols_at_once(pd, gout_ld, gout)) {
    case 4: pool_bwd<4>(gU, gstride, inverse, offsets, B, S, pd, dim, combiner, gout, gout_ld, st); break;
    case 2: pool_bwd<2>(gU, gstride, inverse, offsets, B, S, pd, dim, combiner, gout, gout_ld, st); break;
    default: pool_bwd<1>(gU, gstride, inverse, offsets, B, S, pd, dim, combiner, gout, gout_ld, st);
  }
}
void launch_seq_fwd(const RowSource& src, const int* inverse, const int* offsets, int B, int T, int pd, float* out, int* lengths,
                    cudaStream_t st) {
  const int G = lanes_for_width(pd);
  launch_pdl(src.tbl != nullptr ? seq_fwd_kernel<true> : seq_fwd_kernel<false>, dim3(grid_for((long long)B * T, G, 256)), dim3(256), 0, st,
             src, inverse, offsets, B, T, pd, out, lengths, G);
}
void launch_seq_bwd(float* gU, int gstride, const int* inverse, const int* offsets, int B, int T, int pd, int dim,
                    const float* gout, cudaStream_t st) {
  int G = dim >= 32 ? 32 : (dim >= 16 ? 16 : (dim >= 8 ? 8 : (dim >= 4 ? 4 : (dim >= 2 ? 2 : 1))));
  launch_pdl(seq_bwd_kernel, dim3(grid_for((long long)B * T, G, 256)), dim3(256), 0, st, gU, gstride, inverse, offsets, B, T, pd, dim, gout, G);
}

}  // namespace tn
