// Epilogue of the tcgen05 bf16 GEMM kernels (gemm_tcgen05.cu, gemm_2sm.cu): one warp drains its 32 TMEM lanes of an
// accumulator, applies the fused epilogue (bias, ReLU, ReLU mask of the backward pass, "ones" bias column,
// Hadamard / residual step of DCN-v2, fp32 accumulate) and writes whole 64-byte row segments to global memory.
#pragma once
#include "gemm_tcgen05.h"
#include "tc_primitives.cuh"

namespace tn {
namespace gemm_epi {

constexpr int kBytesPerWarp = 6144;   // out block + two auxiliary blocks of 32 rows x 64 B

enum Mode { kPlain, kMask, kResidual };      // kResidual: the Hadamard step, or a residual alone

// What the epilogues below have in common.  `tm_lane`: TMEM address of the warp's lane quarter at the accumulator's first
// column; `row_base`: global row of TMEM lane 0 of that quarter; `n0`: global column of accumulator column 0; the warp takes
// column chunks sub, sub + nsubs, ... (32 columns each for bf16 outputs, 16 for fp32); `sm_out`: kBytesPerWarp bytes of
// shared memory private to the warp.  TMEM gives a lane one ROW of the tile, global memory wants a warp on whole lines:
// blocks of 32 rows x 64 bytes go through shared memory (16-byte pieces, XOR-swizzled so both the row-wise writes and the
// line-wise reads are bank-conflict free) and leave as 64-byte row segments, eight rows per store.
//
// Small problems spend a third to a half of their time here, and the four warps of a scheduler keep it busy with
// instructions, not with waiting.  So there is code per epilogue, ReLU and its mask work on packed pairs (rounding
// commutes with both), and the mask is applied where its 16-byte pieces have the layout of the stores, which spares it the
// way through shared memory.  Auxiliary operands are asked for before the accumulator is waited for (`ready`; false: it
// will not come), those of the next chunk while the present one is worked on.  8192 x 400 x 430, from the last MMA to the
// last store: forward 3.3 -> 2.6 us, backward with its mask 5.1 -> 3.2 (launch to launch 8.5 -> 8.3 and 10.7 -> 9.4).
struct Lines {                       // the line-wise mapping: 4 lanes per row of 64 bytes, rows lrow, lrow + 8, ...
  int lpc, nrows;                    // 16-byte piece, rows that exist from this lane's first one on
  int so;                            // shared-memory offset of piece lpc of row lrow; the next row is 512 bytes on
  size_t row;
  __device__ __forceinline__ Lines(int lane, int row_base, int M) {
    const int lrow = lane >> 2;
    lpc = lane & 3;
    row = (size_t)(row_base + lrow);
    nrows = M - row_base - lrow;
    so = lrow * 64 + ((lpc ^ ((lrow >> 1) & 3)) << 4);
  }
};

__device__ __forceinline__ uint32_t relu2(uint32_t x) {
  const __nv_bfloat162 r = __hmax2(*reinterpret_cast<const __nv_bfloat162*>(&x), __floats2bfloat162_rn(0.f, 0.f));
  return *reinterpret_cast<const uint32_t*>(&r);
}
// all ones where the bf16 half is above zero (not for NaN)
__device__ __forceinline__ uint32_t positive2(uint32_t x) {
  return __hgt2_mask(*reinterpret_cast<const __nv_bfloat162*>(&x), __floats2bfloat162_rn(0.f, 0.f));
}

template <Mode kMode, class Ready>
__device__ __forceinline__ bool store_bf16(const GemmParams& p, uint32_t tm_lane, int row_base, int n0, int BN, int sub, int nsubs,
                                           int lane, uint8_t* sm_out, Ready&& ready) {
  using namespace tc;
  uint8_t* sm_a0 = sm_out + 2048;
  uint8_t* sm_a1 = sm_out + 4096;
  const int n_store = p.n_store;
  const Lines ln(lane, row_base, p.M);
  const int my_off = lane * 64, my_sw = (lane >> 1) & 3;
  const bool relu = p.relu != 0;
  uint4 va[4], vb[4];
  // auxiliary operands of chunk c0 (ReLU mask, or x0 / xl of the Hadamard step): global -> registers
  auto load_aux = [&](int c0) {
    if (kMode == kPlain) return;
    const int gcol = n0 + c0 + ln.lpc * 8;
    const size_t off = ln.row * p.ld_aux + gcol;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      va[i] = vb[i] = make_uint4(0u, 0u, 0u, 0u);
      if (8 * i < ln.nrows && gcol + 8 <= p.ld_aux) {
        const size_t o = off + (size_t)(8 * i) * p.ld_aux;
        if (kMode == kMask) va[i] = *reinterpret_cast<const uint4*>(p.mask_aux + o);
        else {
          if (p.had_x0) va[i] = *reinterpret_cast<const uint4*>(p.had_x0 + o);
          vb[i] = *reinterpret_cast<const uint4*>(p.had_xl + o);
        }
      }
    }
  };
  const int step = 32 * nsubs;
  auto live = [&](int c0) { return c0 < BN && n0 + c0 < n_store; };      // warp-uniform
  int c0 = 32 * sub;
  if (live(c0)) load_aux(c0);
  if (!ready()) return false;
  for (; live(c0); c0 += step) {
    uint32_t acc[32];
    if (c0 + 16 < BN) {
      tmem_ld32_nowait(tm_lane + (uint32_t)c0, acc);
    } else {
      tmem_ld16_nowait(tm_lane + (uint32_t)c0, acc);
#pragma unroll
      for (int j = 16; j < 32; ++j) acc[j] = 0u;
    }
    if (kMode == kResidual) {          // registers -> the warp's shared-memory blocks, where the row-wise pass finds them
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        *reinterpret_cast<uint4*>(sm_a0 + ln.so + 512 * i) = va[i];
        *reinterpret_cast<uint4*>(sm_a1 + ln.so + 512 * i) = vb[i];
      }
      __syncwarp();
      if (live(c0 + step)) load_aux(c0 + step);
    }
    tmem_ld_wait();
#pragma unroll
    for (int pc = 0; pc < 4; ++pc) {
      const int nb = n0 + c0 + pc * 8;
      const int so = my_off + ((pc ^ my_sw) << 4);
      if (p.bias != nullptr) {
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (nb + j < p.N) acc[pc * 8 + j] = __float_as_uint(__uint_as_float(acc[pc * 8 + j]) + __ldg(p.bias + nb + j));
      }
      uint32_t o[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) o[k] = pack_bf16(__uint_as_float(acc[pc * 8 + 2 * k]), __uint_as_float(acc[pc * 8 + 2 * k + 1]));
      if (relu) {
#pragma unroll
        for (int k = 0; k < 4; ++k) o[k] = relu2(o[k]);
      }
      if (kMode == kResidual) {       // DCN-v2: x0 * (acc + bias) + xl, or just + xl when there is no x0
        const uint4 a0 = *reinterpret_cast<const uint4*>(sm_a0 + so), a1 = *reinterpret_cast<const uint4*>(sm_a1 + so);
        const __nv_bfloat162* h0 = reinterpret_cast<const __nv_bfloat162*>(&a0);
        const __nv_bfloat162* h1 = reinterpret_cast<const __nv_bfloat162*>(&a1);
        // keep u = acc + bias for the backward pass; this lane owns the slot it just read
        if (p.aux_out) *reinterpret_cast<uint4*>(sm_a1 + so) = make_uint4(o[0], o[1], o[2], o[3]);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          float vx = __uint_as_float(acc[pc * 8 + 2 * k]), vy = __uint_as_float(acc[pc * 8 + 2 * k + 1]);
          if (relu) { vx = fmaxf(vx, 0.f); vy = fmaxf(vy, 0.f); }
          const float2 xl = __bfloat1622float2(h1[k]);
          if (p.had_x0) {
            const float2 x0 = __bfloat1622float2(h0[k]);
            vx = x0.x * vx + xl.x; vy = x0.y * vy + xl.y;
          } else {
            vx += xl.x; vy += xl.y;
          }
          o[k] = pack_bf16(vx, vy);
        }
      }
      if (nb + 8 > p.N) {             // only the piece that straddles N pays for the ones / padding columns
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int n = nb + 2 * k;
          if (n >= p.N) o[k] = (o[k] & 0xffff0000u) | (n == p.ones_col ? 0x3f80u : 0u);
          if (n + 1 >= p.N) o[k] = (o[k] & 0xffffu) | (n + 1 == p.ones_col ? 0x3f800000u : 0u);
        }
      }
      *reinterpret_cast<uint4*>(sm_out + so) = make_uint4(o[0], o[1], o[2], o[3]);
    }
    __syncwarp();
    const int gcol = n0 + c0 + ln.lpc * 8;
    if (gcol < n_store && c0 + ln.lpc * 8 < BN) {
      __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(p.C) + ln.row * p.ldc + gcol;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (8 * i >= ln.nrows) continue;
        uint4 o = *reinterpret_cast<const uint4*>(sm_out + ln.so + 512 * i);
        if (kMode == kMask) {         // backward of ReLU: keep the gradient where the forward activation was positive
          uint4 m = make_uint4(positive2(va[i].x), positive2(va[i].y), positive2(va[i].z), positive2(va[i].w));
          if (gcol + 8 > p.N) {       // (columns beyond N are what the row-wise pass has made them)
            uint32_t* mk = reinterpret_cast<uint32_t*>(&m);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              if (gcol + 2 * k >= p.N) mk[k] |= 0xffffu;
              if (gcol + 2 * k + 1 >= p.N) mk[k] |= 0xffff0000u;
            }
          }
          o.x &= m.x; o.y &= m.y; o.z &= m.z; o.w &= m.w;
        }
        __nv_bfloat16* d = dst + (size_t)(8 * i) * p.ldc;
        if (gcol + 8 <= n_store) {
          *reinterpret_cast<uint4*>(d) = o;
        } else {
          const __nv_bfloat16* ob = reinterpret_cast<const __nv_bfloat16*>(&o);
          for (int j = 0; j < n_store - gcol; ++j) d[j] = ob[j];
        }
        if (kMode == kResidual && p.aux_out && gcol + 8 <= p.ld_aux)
          *reinterpret_cast<uint4*>(p.aux_out + (ln.row + 8 * i) * p.ld_aux + gcol) =
              *reinterpret_cast<const uint4*>(sm_a1 + ln.so + 512 * i);
      }
    }
    if (kMode == kMask && live(c0 + step)) load_aux(c0 + step);
    __syncwarp();
  }
  return true;
}

template <class Ready>
__device__ __forceinline__ bool store_f32(const GemmParams& p, uint32_t tm_lane, int row_base, int n0, int BN, int sub, int nsubs,
                                          int lane, uint8_t* sm_out, Ready&& ready) {
  using namespace tc;
  const int n_store = p.n_store;
  const Lines ln(lane, row_base, p.M);
  const int my_off = lane * 64, my_sw = (lane >> 1) & 3;
  const bool plain = p.bias == nullptr && p.relu == 0;
  if (!ready()) return false;
  const int step = 16 * nsubs;
  for (int c0 = 16 * sub; c0 < BN && n0 + c0 < n_store; c0 += step) {      // warp-uniform
    uint32_t acc[16];
    tmem_ld16_nowait(tm_lane + (uint32_t)c0, acc);
    tmem_ld_wait();
    if (!plain || n0 + c0 + 16 > p.N) {
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const int n = n0 + c0 + j;
        float v = __uint_as_float(acc[j]);
        if (p.bias != nullptr && n < p.N) v += __ldg(p.bias + n);
        if (p.relu) v = fmaxf(v, 0.f);
        if (n >= p.N) v = n == p.ones_col ? 1.f : 0.f;
        acc[j] = __float_as_uint(v);
      }
    }
#pragma unroll
    for (int pc = 0; pc < 4; ++pc)
      *reinterpret_cast<uint4*>(sm_out + my_off + ((pc ^ my_sw) << 4)) =
          make_uint4(acc[4 * pc], acc[4 * pc + 1], acc[4 * pc + 2], acc[4 * pc + 3]);
    __syncwarp();
    const int gcol = n0 + c0 + ln.lpc * 4;
    if (gcol < n_store && c0 + ln.lpc * 4 < BN) {
      float* dst = reinterpret_cast<float*>(p.C) + ln.row * p.ldc + gcol;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (8 * i >= ln.nrows) continue;
        const float4 o = *reinterpret_cast<const float4*>(sm_out + ln.so + 512 * i);
        float* d = dst + (size_t)(8 * i) * p.ldc;
        if (gcol + 4 <= n_store) {
          if (p.accumulate) red_add_f32x4(d, o); else *reinterpret_cast<float4*>(d) = o;
        } else {
          const float ov[4] = {o.x, o.y, o.z, o.w};
          for (int j = 0; j < n_store - gcol; ++j) {
            if (p.accumulate) atomicAdd(d + j, ov[j]); else d[j] = ov[j];
          }
        }
      }
    }
    __syncwarp();
  }
  return true;
}

// Asks L2 for the auxiliary operands of a warp's share of a tile, to be called a tile's worth of MMAs before they are needed.
__device__ __forceinline__ void prefetch_aux(const GemmParams& p, int row_base, int n0, int BN, int sub, int nsubs, int lane) {
  const int row = row_base + lane;
  if (row >= p.M) return;
  for (int c0 = 64 * sub; c0 < BN && n0 + c0 < p.ld_aux; c0 += 64 * nsubs) {
    const size_t off = (size_t)row * p.ld_aux + n0 + c0;
    for (const __nv_bfloat16* a : {p.mask_aux, p.had_x0, p.had_xl})
      if (a != nullptr) asm volatile("prefetch.global.L2 [%0];" ::"l"(a + off));
  }
}

// What a kernel's epilogue has to be ready for.
enum Kinds { kBf16, kNoAux, kGrad, kAny };   // a plain bf16 output; no auxiliary operands; fp32 or masked; everything
template <Kinds kKinds, class Ready>
__device__ __forceinline__ bool store_rows(const GemmParams& p, uint32_t tm_lane, int row_base, int n0, int BN, int sub, int nsubs,
                                           int lane, uint8_t* sm_out, Ready&& ready) {
  if (kKinds != kBf16 && p.out_f32) return store_f32(p, tm_lane, row_base, n0, BN, sub, nsubs, lane, sm_out, ready);
  if (kKinds == kBf16 || kKinds == kNoAux) return store_bf16<kPlain>(p, tm_lane, row_base, n0, BN, sub, nsubs, lane, sm_out, ready);
  if (kKinds == kGrad || p.mask_aux != nullptr) return store_bf16<kMask>(p, tm_lane, row_base, n0, BN, sub, nsubs, lane, sm_out, ready);
  if (p.had_xl != nullptr) return store_bf16<kResidual>(p, tm_lane, row_base, n0, BN, sub, nsubs, lane, sm_out, ready);
  return store_bf16<kPlain>(p, tm_lane, row_base, n0, BN, sub, nsubs, lane, sm_out, ready);
}

}  // namespace gemm_epi
}  // namespace tn
