// GPU-resident hashed embedding table: open-addressing key array -> row index into a
// dense row slab.  Replaces the reference's 8 mutex-guarded unordered_maps per rank
// (core/ps/optimizer/optimizer_kernel.h:254-437) and its slab allocator
// (core/utility/allocator.h:26-129).
#pragma once
#include "tn_device.cuh"
#include "tn_types.h"

namespace tn {

constexpr unsigned long long kTagNew = 1ull << 31;
constexpr int kReqNewOwner = 1 << 31;   // this request created the row and must initialise it
constexpr int kReqNewCopy = 1 << 30;    // row was created this step by someone else: recompute init, do not read
constexpr int kReqRowMask = (1 << 30) - 1;
constexpr int kReqPending = -2;         // lost the insert race before the row index was published
constexpr int kReqNone = -1;            // no row (table full)

__device__ __forceinline__ unsigned table_home(const TableView& t, unsigned long long key) {
  return (unsigned)mix64(key) & t.cap_mask;
}

// Read-only probe.  Returns row index or -1.
__device__ __forceinline__ int table_find(const TableView& t, unsigned long long key) {
  unsigned h = table_home(t, key);
  for (unsigned probes = 0; probes <= t.cap_mask; ++probes) {
    unsigned long long k = __ldcg(&t.keys[h]);
    if (k == key) return ld_volatile_s32(&t.slots[h]);
    if (k == kEmptyKey) return -1;
    h = (h + 1) & t.cap_mask;
  }
  return -1;
}

// Row field offsets.
__device__ __forceinline__ int off_g2sum(int dim) { return dim; }
__device__ __forceinline__ int off_show(int kind, int dim) { return kind == kAdaGrad ? dim + 1 : 3 * dim; }
__device__ __forceinline__ int off_click(int dim) { return dim + 2; }           // AdaGrad only
__device__ __forceinline__ int off_noshow(int dim) { return dim + 3; }          // AdaGrad only (int32)
__device__ __forceinline__ int off_delta_show(int dim) { return 3 * dim + 1; }  // Adam / Ftrl (int32)

// ---- pulled rows as the pooling kernels read them (RowSource) ---------------------------------------------------
template <bool kInPlace> struct PulledRows {
  const float* base;
  size_t stride;
  const int* row_of;
  int dim, cvm;
  __device__ __forceinline__ explicit PulledRows(const RowSource& s)
      : base(kInPlace ? reinterpret_cast<const float*>(__ldg(reinterpret_cast<const unsigned long long*>(&s.tbl->rows))) : s.U),
        stride(kInPlace ? s.stride : s.ustride), row_of(s.row_of), dim(s.dim), cvm(s.cvm) {}
  // index of the row of position v (negative: none)
  __device__ __forceinline__ int row(int v) const { return kInPlace && row_of != nullptr && v >= 0 ? __ldg(row_of + v) : v; }
  // Four columns of it from d on, a multiple of four.  A row is a whole number of 16-byte pieces and longer than its pulled
  // columns (the optimizer's state follows), so this never leaves it; what lies beyond the pulled columns is not to be used.
  __device__ __forceinline__ float4 load4(int r, int d) const {
    const float* p = base + (size_t)r * stride;
    float4 x = ldcg_f4(p + d);
    if (kInPlace && cvm != 0 && d + 4 > dim) {
      float e[4] = {x.x, x.y, x.z, x.w};
      float show = 0.f, ratio = 0.f;
      if (cvm == 1) {
        show = __ldcg(p + dim + 1);
        ratio = logf(__ldcg(p + dim + 2) + 1.f) - logf(show + 1.f);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (d + k == dim) e[k] = show;
        if (d + k == dim + 1) e[k] = ratio;
      }
      x = make_float4(e[0], e[1], e[2], e[3]);
    }
    return x;
  }
};

// `n` columns (at most four) to or from an address that is a multiple of SV floats.
template <int SV>
__device__ __forceinline__ void store_cols(float* p, const float4& x, int n) {
  if constexpr (SV == 4) {
    *reinterpret_cast<float4*>(p) = x;
  } else if constexpr (SV == 2) {
    *reinterpret_cast<float2*>(p) = make_float2(x.x, x.y);
    if (n > 2) *reinterpret_cast<float2*>(p + 2) = make_float2(x.z, x.w);
  } else {
    p[0] = x.x;
    if (n > 1) p[1] = x.y;
    if (n > 2) p[2] = x.z;
    if (n > 3) p[3] = x.w;
  }
}
template <int SV>
__device__ __forceinline__ float4 load_cols(const float* p, int n) {
  float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
  if constexpr (SV == 4) {
    x = *reinterpret_cast<const float4*>(p);
  } else if constexpr (SV == 2) {
    const float2 a = *reinterpret_cast<const float2*>(p);
    x.x = a.x; x.y = a.y;
    if (n > 2) { const float2 c = *reinterpret_cast<const float2*>(p + 2); x.z = c.x; x.w = c.y; }
  } else {
    x.x = p[0];
    if (n > 1) x.y = p[1];
    if (n > 2) x.z = p[2];
    if (n > 3) x.w = p[3];
  }
  return x;
}
// Adds the first `n` columns of x to a row of gradients whose rows are whole 16-byte pieces.
__device__ __forceinline__ void red_add_cols(float* p, const float4& x, int n) {
  if (n >= 4) { red_add_f32x4(p, x); return; }
  if (n >= 2) asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(x.x), "f"(x.y) : "memory");
  if (n == 1) atomicAdd(p, x.x);
  if (n == 3) atomicAdd(p + 2, x.z);
}

}  // namespace tn
