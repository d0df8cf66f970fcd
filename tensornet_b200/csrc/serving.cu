// Serving-side lookup: read-only dictionary probe + per-slot pooling + cast into the padded bf16
// operand of the first dense layer, in one kernel.  The reference's online demo looks every id up
// in a dictionary service, mean-pools multi-valued slots and copies the result into the dense
// graph's feeds (examples/online_serving/main.cc:42-91, graph.cc:25-71); its lookup is a stub
// that returns random vectors.  Signs missing from the dictionary contribute zeros.
#include <cuda_bf16.h>
#include "sparse_table.cuh"
#include "tn_ops.h"

namespace tn {

namespace {

// Bag g = s * B + b holds ids [offsets[g], offsets[g+1]) (or exactly id g when offsets == nullptr).
// dim % 4 == 0; G lanes per bag, each lane owns float4 chunks of the embedding.
__global__ void dict_lookup_pool_kernel(TableView t, const long long* __restrict__ ids, const int* __restrict__ offsets, int B,
                                        int S, int combiner, __nv_bfloat16* __restrict__ out, int ld_out, int ones_col, int G) {
  const int lane = threadIdx.x % G;
  const int gid = (blockIdx.x * blockDim.x + threadIdx.x) / G;
  const int ngroups = (gridDim.x * blockDim.x) / G;
  const int dim = t.dim, nch = dim >> 2, nbags = B * S;
  for (int g = gid; g < nbags; g += ngroups) {
    const int s = g / B, b = g - s * B;
    int k0 = g, k1 = g + 1;
    if (offsets) { k0 = offsets[g]; k1 = offsets[g + 1]; }
    const int len = k1 - k0;
    const float sc = len <= 0 ? 0.f : (combiner == 1 ? 1.f / (float)len : (combiner == 2 ? rsqrtf((float)len) : 1.f));
    __nv_bfloat16* o = out + (size_t)b * ld_out + (size_t)s * dim;
    for (int ch = lane; ch < nch; ch += G) {
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int k = k0; k < k1; ++k) {
        const int r = table_find(t, canon_key((unsigned long long)ids[k]));
        if (r >= 0) {
          const float4 x = *reinterpret_cast<const float4*>(t.rows + (size_t)r * t.stride + 4 * ch);
          acc.x += x.x; acc.y += x.y; acc.z += x.z; acc.w += x.w;
        }
      }
      __nv_bfloat162 lo = __floats2bfloat162_rn(acc.x * sc, acc.y * sc), hi = __floats2bfloat162_rn(acc.z * sc, acc.w * sc);
      *reinterpret_cast<uint2*>(o + 4 * ch) = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
    }
  }
  // tail columns of every row: constant one (bias input of the first layer) and zero padding
  const int tail0 = S * dim, ntail = ld_out - tail0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < B * ntail; i += gridDim.x * blockDim.x) {
    const int b = i / ntail, c = tail0 + (i - b * ntail);
    out[(size_t)b * ld_out + c] = __float2bfloat16(c == ones_col ? 1.f : 0.f);
  }
}

// ---------------------------------------------------------------------------------------------------------------------
// The request path of InferenceEngine: lookup -> layers -> head, a handful of kernels chained as programmatic
// dependents.  What bounds a request is latency, so every stage is shaped for parallel misses: one lane per id probes
// (its key and its row index are loaded together, not one behind the other), then all rows of a warp's bags are in
// flight at once.  The ids of a small request (128 KB at most) may be read straight from pinned host memory, which takes
// the copy and the wait for it out of the chain: the PCIe reads of all warps are in flight together.  Larger ones are
// copied first, beside the conversion of the weights where there is one.
// The first kernel of the chain is launched the ordinary way: it starts when everything before the request is complete,
// so that the ones behind it may write their buffers and read weights before their own predecessor is done.
// 200 slots x 512 examples, dim 32 (102 K ids, 2 M rows): lookup 17.3 us as one probe after the other, 9.4 to 9.9 now,
// behind a copy of 18 to 36 us (the host link differs from machine to machine).
// ---------------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ int find_row(const TableView& t, unsigned long long key) {
  unsigned h = table_home(t, key);
  for (unsigned probes = 0; probes <= t.cap_mask; ++probes) {
    const unsigned long long k = __ldg(&t.keys[h]);
    const int r = __ldg(&t.slots[h]);
    if (k == key) return r;
    if (k == kEmptyKey) return -1;
    h = (h + 1) & t.cap_mask;
  }
  return -1;
}

__device__ __forceinline__ uint2 pack4(float4 v) {
  __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
  return make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
}

// the constant-one column and the zero padding behind the S * dim columns of every row
__device__ __forceinline__ void write_tail(__nv_bfloat16* out, int B, int tail0, int ld_out, int ones_col) {
  const int ntail = ld_out - tail0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < B * ntail; i += gridDim.x * blockDim.x) {
    const int b = i / ntail, c = tail0 + (i - b * ntail);
    out[(size_t)b * ld_out + c] = __float2bfloat16(c == ones_col ? 1.f : 0.f);
  }
}

// One id per bag.  A warp takes `wb` consecutive bags (a power of two, 32 / G at least): fewer when the request is small,
// so that its ids spread over many SMs.
__global__ void __launch_bounds__(256) serve_lookup_single_kernel(TableView t, const long long* __restrict__ ids, int B, int S,
                                                                  __nv_bfloat16* __restrict__ out, int ld_out, int ones_col, int G, int wb) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int lane = threadIdx.x & 31, sub = lane / G, gl = lane % G, rpp = 32 / G;
  const int dim = t.dim, nch = dim >> 2, nbags = B * S;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  for (int g0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * wb; g0 < nbags; g0 += nwarps * wb) {
    int r = -1;
    if (lane < wb && g0 + lane < nbags) r = find_row(t, canon_key((unsigned long long)__ldg(ids + g0 + lane)));
#pragma unroll 4
    for (int p = 0; p < wb; p += rpp) {
      const int rr = __shfl_sync(0xffffffffu, r, p + sub);
      const int g = g0 + p + sub;
      if (g >= nbags) continue;
      const int s = g / B, b = g - s * B;
      __nv_bfloat16* o = out + (size_t)b * ld_out + (size_t)s * dim;
      for (int ch = gl; ch < nch; ch += G) {
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (rr >= 0) x = __ldg(reinterpret_cast<const float4*>(t.rows + (size_t)rr * t.stride + 4 * ch));
        *reinterpret_cast<uint2*>(o + 4 * ch) = pack4(x);
      }
    }
  }
  write_tail(out, B, S * dim, ld_out, ones_col);
  asm volatile("griddepcontrol.wait;" ::: "memory");      // whatever precedes this kernel is complete once this kernel is
}

// Ragged bags, first half: row index of every id; offsets and ids come from wherever the caller has them.
__global__ void __launch_bounds__(256) serve_probe_kernel(TableView t, const long long* __restrict__ ids, int n, const int* __restrict__ offsets,
                                                          int n_off, int* __restrict__ rows, int* __restrict__ offsets_out) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int t0 = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
  for (int i = t0; i < n; i += nt) rows[i] = find_row(t, canon_key((unsigned long long)__ldg(ids + i)));
  if (offsets_out != nullptr)
    for (int i = t0; i < n_off; i += nt) offsets_out[i] = __ldg(offsets + i);
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
// second half: a group of G lanes per bag, the lanes fetch the bag's row indices side by side and keep four rows in flight
__global__ void __launch_bounds__(256) serve_pool_kernel(TableView t, const int* __restrict__ rows, int n, const int* __restrict__ offsets, int B,
                                                         int S, int combiner, __nv_bfloat16* __restrict__ out, int ld_out, int ones_col, int G) {
  pdl_sync();
  const int lane = threadIdx.x & 31, gl = lane % G, first = lane - gl;
  const unsigned gmask = G >= 32 ? 0xffffffffu : (((1u << G) - 1u) << first);
  const int dim = t.dim, nch = dim >> 2, nbags = B * S;
  const int ngroups = (gridDim.x * blockDim.x) / G;
  for (int g = (blockIdx.x * blockDim.x + threadIdx.x) / G; g < nbags; g += ngroups) {
    const int s = g / B, b = g - s * B;
    const int k0 = max(__ldcg(offsets + g), 0), k1 = min(__ldcg(offsets + g + 1), n), len = k1 - k0;
    const float sc = len <= 0 ? 0.f : (combiner == 1 ? 1.f / (float)len : (combiner == 2 ? rsqrtf((float)len) : 1.f));
    __nv_bfloat16* o = out + (size_t)b * ld_out + (size_t)s * dim;
    for (int ch0 = 0; ch0 < nch; ch0 += G) {
      const int ch = ch0 + gl;
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int kb = k0; kb < k1; kb += G) {
        const int mine = kb + gl < k1 ? __ldcg(rows + kb + gl) : -1;
        const int m = min(G, k1 - kb);
        for (int j = 0; j < m; j += 4) {
          float4 x[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int rr = __shfl_sync(gmask, mine, first + min(j + u, G - 1));
            x[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (j + u < m && rr >= 0 && ch < nch) x[u] = __ldg(reinterpret_cast<const float4*>(t.rows + (size_t)rr * t.stride + 4 * ch));
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) { acc.x += x[u].x; acc.y += x[u].y; acc.z += x[u].z; acc.w += x[u].w; }
        }
      }
      if (ch < nch) *reinterpret_cast<uint2*>(o + 4 * ch) = pack4(make_float4(acc.x * sc, acc.y * sc, acc.z * sc, acc.w * sc));
    }
  }
  write_tail(out, B, S * dim, ld_out, ones_col);
}

// fp32 weights -> bf16 operands, all layers in one launch (28.8 MB at 6400-1024-512-256); runs under the lookup.
__global__ void __launch_bounds__(256) serve_cast_kernel(const __grid_constant__ ServeCast a) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const long long t0 = blockIdx.x * (long long)blockDim.x + threadIdx.x, nt = (long long)gridDim.x * blockDim.x;
  for (int l = 0; l < a.n; ++l) {
    const float4* src = reinterpret_cast<const float4*>(a.src[l]);
    uint4* dst = reinterpret_cast<uint4*>(a.dst[l]);
    for (long long i = t0; i < a.n8[l]; i += nt) {
      const uint2 lo = pack4(__ldg(src + 2 * i)), hi = pack4(__ldg(src + 2 * i + 1));
      dst[i] = make_uint4(lo.x, lo.y, hi.x, hi.y);
    }
  }
}

__device__ __forceinline__ float4 bf16x4(uint2 v) {
  const float2 a = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&v.x)), b = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&v.y));
  return make_float4(a.x, a.y, b.x, b.y);
}

// A layer of a request of at most kServeSkinnyRows rows, y[m, n] = relu(sum_k x[m, k] w[n, k]): a 128-row MMA tile would be all
// padding, and what counts is streaming the weights once through every SM.  A warp takes kRows weight rows, eight loads
// in flight per lane; a block's warps share a group of rows and split K (`ksplit` ways), the parts meet in shared
// memory.  fp32 weights are rounded to bf16 on the way, as the MMA operands are.  The bias sits in column K - 1.
template <int kM, bool kF32>
__global__ void __launch_bounds__(256) serve_skinny_kernel(const __nv_bfloat16* __restrict__ x, int ldx, const void* __restrict__ w, int ldw, int M,
                                                           int N, int K, int relu, __nv_bfloat16* __restrict__ y, int ldy, int n_store, int ksplit) {
  constexpr int kRows = 2;
  __shared__ float s_part[8][kRows * kM];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int groups = 8 / ksplit;                                 // row groups per block
  const int rg = warp / ksplit, kp = warp % ksplit;
  const int n0 = (blockIdx.x * groups + rg) * kRows;
  float acc[kRows][kM];
#pragma unroll
  for (int r = 0; r < kRows; ++r)
#pragma unroll
    for (int m = 0; m < kM; ++m) acc[r][m] = 0.f;
  const int n4 = (K + 3) >> 2;                                   // ldw and ldx are multiples of 8: the last chunk is readable
  const int per = (n4 + ksplit - 1) / ksplit;
  const int c0 = kp * per, c1 = min(n4, c0 + per);
  // the weights do not depend on the kernel before this one: the first ones are on their way before its results are waited for
  constexpr int kUn = 4;
  float4 wv[kRows][kUn];
  auto load_w = [&](int c) {
#pragma unroll
    for (int u = 0; u < kUn; ++u) {
      const int cc = c + 32 * u + lane;
#pragma unroll
      for (int r = 0; r < kRows; ++r) {
        wv[r][u] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (cc < c1 && n0 + r < N) {
          if (kF32) wv[r][u] = __ldg(reinterpret_cast<const float4*>(reinterpret_cast<const float*>(w) + (size_t)(n0 + r) * ldw) + cc);
          else wv[r][u] = bf16x4(__ldg(reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(w) + (size_t)(n0 + r) * ldw) + cc));
        }
      }
    }
  };
  load_w(c0);
  pdl_sync();
  for (int c = c0; c < c1; c += 32 * kUn) {
    if (c != c0) load_w(c);
#pragma unroll
    for (int u = 0; u < kUn; ++u) {
      const int cc = c + 32 * u + lane;
      if (cc < c1) {
        const int k = 4 * cc;
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
          if (kF32) wv[r][u] = bf16x4(pack4(wv[r][u]));
          if (k + 4 > K) { if (k + 1 >= K) wv[r][u].y = 0.f; if (k + 2 >= K) wv[r][u].z = 0.f; wv[r][u].w = 0.f; }
        }
#pragma unroll
        for (int m = 0; m < kM; ++m) {
          if (m < M) {
            const float4 xv = bf16x4(__ldcg(reinterpret_cast<const uint2*>(x + (size_t)m * ldx) + cc));
#pragma unroll
            for (int r = 0; r < kRows; ++r)
              acc[r][m] += wv[r][u].x * xv.x + wv[r][u].y * xv.y + wv[r][u].z * xv.z + wv[r][u].w * xv.w;
          }
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < kRows; ++r)
#pragma unroll
    for (int m = 0; m < kM; ++m) {
      float v = acc[r][m];
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) s_part[warp][r * kM + m] = v;
    }
  __syncthreads();
  for (int i = threadIdx.x; i < groups * kRows * kM; i += blockDim.x) {
    const int g = i / (kRows * kM), j = i - g * (kRows * kM), r = j / kM, m = j - r * kM;
    const int n = (blockIdx.x * groups + g) * kRows + r;
    if (n >= n_store || m >= M) continue;
    float v = 0.f;
    for (int q = 0; q < ksplit; ++q) v += s_part[g * ksplit + q][j];
    if (relu) v = fmaxf(v, 0.f);
    if (n >= N) v = n == N ? 1.f : 0.f;                          // ones column and padding
    y[(size_t)m * ldy + n] = __float2bfloat16(v);
  }
}

// logit and probability of every row: a warp per row
__global__ void __launch_bounds__(256) serve_head_kernel(const __nv_bfloat16* __restrict__ z, int ld, int B, int K, const float* __restrict__ w,
                                                         float* __restrict__ prob) {
  pdl_sync();
  const int lane = threadIdx.x & 31, nwarps = (gridDim.x * blockDim.x) >> 5;
  for (int b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; b < B; b += nwarps) {
    float acc = 0.f;
    for (int c = lane; 4 * c < K; c += 32) {
      const float4 v = bf16x4(__ldcg(reinterpret_cast<const uint2*>(z + (size_t)b * ld) + c));
      const int k = 4 * c;
      acc += v.x * __ldg(w + k);
      if (k + 1 < K) acc += v.y * __ldg(w + k + 1);
      if (k + 2 < K) acc += v.z * __ldg(w + k + 2);
      if (k + 3 < K) acc += v.w * __ldg(w + k + 3);
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) prob[b] = 1.f / (1.f + expf(-acc));
  }
}

__global__ void sigmoid_kernel(const float* __restrict__ x, float* __restrict__ y, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) y[i] = 1.f / (1.f + expf(-x[i]));
}

}  // namespace

void launch_dict_lookup_pool(const TableView& t, const long long* ids, const int* offsets, int B, int S, int combiner, void* out,
                             int ld_out, int ones_col, cudaStream_t st) {
  int G = lanes_for_width(t.dim);
  long long blocks = ((long long)B * S * G + 255) / 256;
  if (blocks < 1) blocks = 1;
  if (blocks > 148 * 16) blocks = 148 * 16;
  dict_lookup_pool_kernel<<<(int)blocks, 256, 0, st>>>(t, ids, offsets, B, S, combiner, reinterpret_cast<__nv_bfloat16*>(out), ld_out,
                                                     ones_col, G);
}
void launch_sigmoid(const float* x, float* y, int n, cudaStream_t st) {
  int blocks = (n + 255) / 256; if (blocks > 148 * 4) blocks = 148 * 4; if (blocks < 1) blocks = 1;
  sigmoid_kernel<<<blocks, 256, 0, st>>>(x, y, n);
}


static int capped(long long blocks, int most) { return (int)(blocks < 1 ? 1 : (blocks > most ? most : blocks)); }

void launch_serve_cast(const ServeCast& a, cudaStream_t st) {
  long long n8 = 0;
  for (int l = 0; l < a.n; ++l) n8 = a.n8[l] > n8 ? a.n8[l] : n8;
  serve_cast_kernel<<<capped((n8 + 255) / 256, 148 * 4), 256, 0, st>>>(a);
}
void launch_serve_lookup_single(const TableView& t, const long long* ids, int B, int S, void* out, int ld_out, int ones_col, bool behind_cast,
                                cudaEvent_t read, cudaStream_t st) {
  const int G = lanes_for_width(t.dim);
  const long long nbags = (long long)B * S;
  int wb = 32;                                                   // enough warps for every SM to have a few
  while (wb > 32 / G && nbags / wb < 148 * 40) wb >>= 1;
  const dim3 grid(capped((nbags + wb * 8 - 1) / (wb * 8), 148 * 8));
  __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(out);
  if (behind_cast) launch_pdl(serve_lookup_single_kernel, grid, dim3(256), 0, st, t, ids, B, S, o, ld_out, ones_col, G, wb);
  else serve_lookup_single_kernel<<<grid, 256, 0, st>>>(t, ids, B, S, o, ld_out, ones_col, G, wb);
  if (read != nullptr) cudaEventRecord(read, st);
}
void launch_serve_lookup_ragged(const TableView& t, const long long* ids, int n, const int* offsets, int B, int S, int combiner, int* rows,
                                int* offsets_dev, void* out, int ld_out, int ones_col, bool behind_cast, cudaEvent_t read, cudaStream_t st) {
  const int G = lanes_for_width(t.dim);
  const long long nbags = (long long)B * S;
  const dim3 grid(capped(((n > nbags ? n : nbags) + 255) / 256, 148 * 8));
  if (behind_cast) launch_pdl(serve_probe_kernel, grid, dim3(256), 0, st, t, ids, n, offsets, (int)nbags + 1, rows, offsets_dev);
  else serve_probe_kernel<<<grid, 256, 0, st>>>(t, ids, n, offsets, (int)nbags + 1, rows, offsets_dev);
  if (read != nullptr) cudaEventRecord(read, st);
  launch_pdl(serve_pool_kernel, dim3(capped((nbags * G + 255) / 256, 148 * 8)), dim3(256), 0, st, t, rows, n,
             static_cast<const int*>(offsets_dev != nullptr ? offsets_dev : offsets), B, S, combiner, reinterpret_cast<__nv_bfloat16*>(out), ld_out, ones_col, G);
}
template <int kM>
static void skinny(const void* x, int ldx, const void* w, int w_f32, int ldw, int M, int N, int K, int relu, void* y, int ldy, int n_store,
                   cudaStream_t st) {
  constexpr int kRows = 2;               // as in the kernel
  // long rows are split over the warps of a block until every SM has a block (a row group is read by one warp otherwise)
  int ks = 1;
  while (ks < 8 && (n_store + (8 / ks) * kRows - 1) / ((8 / ks) * kRows) < 148 && K / (2 * ks) >= 256) ks *= 2;
  const dim3 grid((n_store + (8 / ks) * kRows - 1) / ((8 / ks) * kRows));
  const __nv_bfloat16* xb = reinterpret_cast<const __nv_bfloat16*>(x);
  __nv_bfloat16* yb = reinterpret_cast<__nv_bfloat16*>(y);
  if (w_f32) launch_pdl(serve_skinny_kernel<kM, true>, grid, dim3(256), 0, st, xb, ldx, w, ldw, M, N, K, relu, yb, ldy, n_store, ks);
  else launch_pdl(serve_skinny_kernel<kM, false>, grid, dim3(256), 0, st, xb, ldx, w, ldw, M, N, K, relu, yb, ldy, n_store, ks);
}
void launch_serve_skinny(const void* x, int ldx, const void* w, int w_f32, int ldw, int M, int N, int K, int relu, void* y, int ldy, int n_store,
                         cudaStream_t st) {
  static_assert(kServeSkinnyRows == 2, "one instantiation per row count");
  if (M <= 1) skinny<1>(x, ldx, w, w_f32, ldw, M, N, K, relu, y, ldy, n_store, st);
  else skinny<2>(x, ldx, w, w_f32, ldw, M, N, K, relu, y, ldy, n_store, st);
}
void launch_serve_head(const void* z, int ld, int B, int K, const float* w, float* prob, cudaStream_t st) {
  launch_pdl(serve_head_kernel, dim3(capped((B + 7) / 8, 148 * 4)), dim3(256), 0, st, reinterpret_cast<const __nv_bfloat16*>(z), ld, B, K, w, prob);
}

}  // namespace tn
