// bf16 GEMM for problems with few output tiles and a long contraction (the towers of a request batch, the layers of a
// small training batch): the CTAs of a thread-block cluster share one output tile, each contracts its part of K on the
// tensor cores, and the partial tiles are summed through distributed shared memory before one fused epilogue.
//
// What bounds it: one SM takes in operands at about 120 GB/s, so a 512 x 1024 x 6401 layer on the 40 tiles that the
// plain kernel makes of it waits 36 us for 101 k-blocks per CTA while 108 SMs idle.  With eight CTAs per tile every SM
// has 13 k-blocks.  The sum is deterministic (fixed order over the cluster) and in fp32, as one accumulator would be.
//
// Every mbarrier wait is bounded; after an expiry the CTA still takes part in the cluster barriers, skips its stores
// and leaves an error in the status words.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cstdint>
#include <cstdlib>
#include "gemm_tcgen05.h"
#include "tc_primitives.cuh"

namespace tn {

using namespace tc;

namespace {

constexpr int kBM = 128, kBK = 64, kUmmaK = 16;
constexpr int kABytes = kBM * kBK * 2;
constexpr int kWarps = 10;                  // warp 0 TMA, warp 1 MMA + TMEM owner, 2..9 drain the accumulator; all reduce
constexpr int kThreads = 32 * kWarps;
constexpr int kMaxStages = kGemmMaxStages;

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
  return v;
}

// Position of the 16-byte piece `pc` of row `r` in a block of 128 rows of 2^lp pieces: rows follow one another without
// gaps, so that a warp reads 512 contiguous bytes of another CTA's block, and the pieces of a row are permuted so that
// eight lanes that write one piece each of eight successive rows hit eight different bank groups.
__device__ __forceinline__ int piece_at(int r, int pc, int lp) {
  const int sw = lp >= 3 ? (r & 7) : ((r >> (3 - lp)) & ((1 << lp) - 1));
  return (r << lp) + (pc ^ sw);
}

__global__ void __launch_bounds__(kThreads, 1)
gemm_bf16_splitk_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const GemmParams p,
                        const int S, const int kStages) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t s_full[kMaxStages];
  __shared__ __align__(8) uint64_t s_empty[kMaxStages];
  __shared__ __align__(8) uint64_t s_accum;
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort_i;
  volatile int* s_abort = &s_abort_i;

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;      // (known to be one per warp)
  const int BN = p.BN;
  const uint32_t b_bytes = (uint32_t)BN * kBK * 2;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t a_smem = base, b_smem = base + kStages * kABytes;
  const int rank = (int)__shfl_sync(0xffffffffu, cluster_ctarank(), 0);
  const int n0 = ((int)blockIdx.x / S) * BN, m0 = (int)blockIdx.y * kBM;
  const int kt_total = (p.K + kBK - 1) / kBK;
  const int kt0 = rank * p.k_tiles_per_split;
  int nk = kt_total - kt0;
  if (nk > p.k_tiles_per_split) nk = p.k_tiles_per_split;      // > 0 for every rank (host side)

  uint32_t tmem_cols = 32;
  while ((int)tmem_cols < BN) tmem_cols <<= 1;
  if (threadIdx.x == 0) {
    *s_abort = 0;
    for (int s = 0; s < kStages; ++s) { mbar_init(smem_u32(&s_full[s]), 1); mbar_init(smem_u32(&s_empty[s]), 1); }
    mbar_init(smem_u32(&s_accum), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmA)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmB)) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(tmem_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s_tmem;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  // (whole warps with one elected lane that issues, as in gemm_tcgen05.cu)
  if (warp == 0) {
    const bool lead = elect_one();
    int s = 0;
    uint32_t ph = 1u;
    for (int i = 0; i < nk; ++i) {
      if (i >= kStages && !mbar_wait_warp(smem_u32(&s_empty[s]), ph, s_abort)) { *s_abort = 1; break; }
      const uint32_t full = smem_u32(&s_full[s]);
      const int kc = (kt0 + i) * kBK;
      const uint32_t a_dst = a_smem + s * kABytes, b_dst = b_smem + s * b_bytes;
      if (lead) {
        mbar_expect_tx(full, kABytes + b_bytes);
        if (!p.a_mn) {
          tma_load_2d(a_dst, &tmA, kc, m0, full);
        } else {
          tma_load_2d(a_dst, &tmA, m0, kc, full);
          tma_load_2d(a_dst + 8192, &tmA, m0 + 64, kc, full);
        }
        if (!p.b_mn) {
          tma_load_2d(b_dst, &tmB, kc, n0, full);
        } else {
          for (int c = 0; c < BN / 64; ++c) tma_load_2d(b_dst + c * 8192, &tmB, n0 + 64 * c, kc, full);
        }
      }
      __syncwarp();
      if (++s == kStages) { s = 0; ph ^= 1u; }
    }
  } else if (warp == 1) {
    const bool lead = elect_one();
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(p.a_mn ? 1 : 0) << 15) |
                           ((uint32_t)(p.b_mn ? 1 : 0) << 16) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);
    const uint32_t a_lbo = p.a_mn ? 8192u : 16u, b_lbo = p.b_mn ? 8192u : 16u;
    const uint32_t a_kstep = p.a_mn ? 2048u : 32u, b_kstep = p.b_mn ? 2048u : 32u;
    bool ok = true;
    int s = 0;
    uint32_t ph = 0u;
    for (int i = 0; i < nk; ++i) {
      if (!mbar_wait_warp(smem_u32(&s_full[s]), ph, s_abort)) { *s_abort = 1; ok = false; break; }
      tc_fence_after();
      if (lead) {
#pragma unroll
        for (int k = 0; k < kBK / kUmmaK; ++k) {
          const uint64_t ad = make_smem_desc(a_smem + s * kABytes + k * a_kstep, a_lbo, 1024u);
          const uint64_t bd = make_smem_desc(b_smem + s * b_bytes + k * b_kstep, b_lbo, 1024u);
          umma_f16(tm, ad, bd, idesc, (i > 0 || k > 0) ? 1u : 0u);
        }
        if (i + kStages < nk) umma_commit(smem_u32(&s_empty[s]));
      }
      __syncwarp();
      if (++s == kStages) { s = 0; ph ^= 1u; }
    }
    if (ok && lead) umma_commit(smem_u32(&s_accum));
    __syncwarp();
  }

  // ---- partial tile -> this CTA's shared memory (the stage ring is free once the accumulator barrier has fired) -----
  // fp32, one block of 128 rows x (BN / S) columns per CTA of the cluster.
  const int cw = BN / S, lp = 31 - __clz(cw >> 2);               // columns per CTA, log2 of the 16-byte pieces per row
  uint8_t* part = smem_raw + (base - smem_u32(smem_raw));
  if (warp >= 2) {
    const int q = warp & 3, sub = (warp - 2) >> 2, r = q * 32 + lane;
    if (mbar_wait(smem_u32(&s_accum), 0u, s_abort)) {
      tc_fence_after();
      const uint32_t tl = tmem + ((uint32_t)(q * 32) << 16);
      for (int c0 = 32 * sub; c0 < BN; c0 += 64) {
        uint32_t acc[32];
        tmem_ld32_nowait(tl + (uint32_t)c0, acc);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int pc = (c0 >> 2) + j, slice = pc >> lp;
          *reinterpret_cast<uint4*>(part + (((size_t)slice * kBM << lp) + piece_at(r, pc & ((1 << lp) - 1), lp)) * 16) =
              make_uint4(acc[4 * j], acc[4 * j + 1], acc[4 * j + 2], acc[4 * j + 3]);
        }
      }
      tc_fence_before();
    } else {
      *s_abort = 1;
    }
  }
  cluster_sync_all();
  tc_fence_after();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols) : "memory");

  // ---- this CTA's share of the columns: sum over the cluster, epilogue, store ---------------------------------------
  const uint32_t block = base + (uint32_t)(((size_t)rank * kBM << lp) * 16);
  if (!*s_abort) {
    const int rows = min(kBM, p.M - m0);
    for (int it = threadIdx.x; it < (rows << lp); it += kThreads) {
      const int r = it >> lp, pc = piece_at(0, it & ((1 << lp) - 1), lp) ^ (piece_at(r, 0, lp) - (r << lp));
      const int grow = m0 + r, gcol = n0 + rank * cw + 4 * pc;
      float4 x[8];
#pragma unroll
      for (int s = 0; s < 8; ++s)
        if (s < S) x[s] = ld_cluster_f4(map_to_cta(block + (uint32_t)it * 16u, (uint32_t)s));
      float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int s = 0; s < 8; ++s)
        if (s < S) { v[0] += x[s].x; v[1] += x[s].y; v[2] += x[s].z; v[3] += x[s].w; }
      if (gcol >= p.n_store) continue;
      if (p.bias) {
#pragma unroll
        for (int j = 0; j < 4; ++j) if (gcol + j < p.N) v[j] += __ldg(p.bias + gcol + j);
      }
      if (p.relu) {
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = fmaxf(v[j], 0.f);
      }
      if (p.mask_aux) {
        uint2 a0 = make_uint2(0u, 0u);
        if (gcol + 4 <= p.ld_aux) a0 = *reinterpret_cast<const uint2*>(p.mask_aux + (size_t)grow * p.ld_aux + gcol);
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&a0);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const float2 m2 = __bfloat1622float2(h[k]);
          if (!(m2.x > 0.f)) v[2 * k] = 0.f;
          if (!(m2.y > 0.f)) v[2 * k + 1] = 0.f;
        }
      }
      if (gcol + 4 > p.N) {
#pragma unroll
        for (int j = 0; j < 4; ++j) if (gcol + j >= p.N) v[j] = gcol + j == p.ones_col ? 1.f : 0.f;
      }
      const uint2 o = make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]));
      __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(p.C) + (size_t)grow * p.ldc + gcol;
      if (gcol + 4 <= p.n_store) {
        *reinterpret_cast<uint2*>(dst) = o;
      } else {
        const __nv_bfloat16* ob = reinterpret_cast<const __nv_bfloat16*>(&o);
        for (int j = 0; j < p.n_store - gcol; ++j) dst[j] = ob[j];
      }
    }
    // the constant-one and padding columns that lie beyond the last tile (a tile of their own would cost a cluster)
    const int pad0 = n0 + BN;
    if (n0 < p.N && pad0 >= p.N && rank == S - 1 && pad0 < p.n_store) {
      const int np = p.n_store - pad0;
      for (int it = threadIdx.x; it < kBM * np; it += kThreads) {
        const int r = it / np, c = pad0 + (it - r * np);
        if (m0 + r < p.M) reinterpret_cast<__nv_bfloat16*>(p.C)[(size_t)(m0 + r) * p.ldc + c] = __float2bfloat16(c == p.ones_col ? 1.f : 0.f);
      }
    }
  } else {
    if (threadIdx.x == 0) set_status(p.status, kMbarTimeout, 31, (int)blockIdx.x);
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);            // copies in flight land before the shared memory goes away
  }
  cluster_sync_all();                                            // nobody leaves while its partial tile is still being read
}

}  // namespace

// Cost (in ns, without the launch) of the best cluster split of this problem; fills BN and S.  Fitted on B200 to
// 16..1024 x 1024 x 6401, 512 x 512 x 1025, 4096 x 512 x 201 and smaller: a k-block costs what gemm_kblock_ns says, the
// reduction and the two cluster barriers 1.7 us + 5 ns per column, growing to 23 ns per column when the chip is full (the
// partial tiles then cross the SM-to-SM network together).  Clusters stay inside a GPC, so that fewer than 148 CTAs of large
// clusters run at a time (16 clusters of eight were measured to take two turns).
double gemm_splitk_plan(const GemmDesc& d, int* best_bn, int* best_s) {
  const int kt = (d.K + kBK - 1) / kBK, mt = (d.M + kBM - 1) / kBM;
  double best = 1e30;
  for (int bn = 64; bn <= 256; bn *= 2) {
    const int nt = (d.N + bn - 1) / bn;
    for (int s = 2; s <= 8; s *= 2) {
      if (kt < 2 * s) break;                                     // at least two k-blocks for every CTA
      const int ktps = (kt + s - 1) / s;
      if ((kt + ktps - 1) / ktps != s) continue;                 // every CTA of the cluster has work
      const int fit = s == 8 ? 96 : (s == 4 ? 128 : 148);
      const long long ctas = (long long)mt * nt * s;
      const double load = ctas <= 32 ? 0.0 : (ctas >= 128 ? 1.0 : (ctas - 32) / 96.0);
      const double per_cta = ktps * gemm_kblock_ns(bn, gemm_ring_stages(bn)) + bn * (5.0 + 18.0 * load) + 1700.0;
      const double cost = (double)((ctas + fit - 1) / fit) * per_cta;
      if (cost < best) { best = cost; *best_bn = bn; *best_s = s; }
    }
  }
  return best;
}

const char* gemm_bf16_splitk(const GemmDesc& d, GemmParams p, int BN, int S, cudaStream_t stream) {
  const int kt = (d.K + kBK - 1) / kBK, ktps = (kt + S - 1) / S;
  if (S < 2 || S > 8 || (S & (S - 1)) || (BN != 64 && BN != 128 && BN != 256) || (kt + ktps - 1) / ktps != S) return "gemm_bf16: bad cluster split";
  CUtensorMap tmA, tmB;
  bool ok;
  if (!d.a_mn) ok = get_tensor_map(d.A, d.M, d.K, d.lda, kBM, &tmA);
  else         ok = get_tensor_map(d.A, d.K, d.M, d.lda, kBK, &tmA);
  if (!ok) return "gemm_bf16: cuTensorMapEncodeTiled failed for A";
  if (!d.b_mn) ok = get_tensor_map(d.B, d.N, d.K, d.ldb, BN, &tmB);
  else         ok = get_tensor_map(d.B, d.K, d.N, d.ldb, kBK, &tmB);
  if (!ok) return "gemm_bf16: cuTensorMapEncodeTiled failed for B";
  p.BN = BN; p.k_tiles_per_split = ktps;
  const int stages = gemm_ring_stages(BN);
  size_t smem = (size_t)stages * (kABytes + (size_t)BN * kBK * 2);
  const size_t tile = (size_t)kBM * BN * 4;
  if (tile > smem) smem = tile;
  smem += 1024;
  static bool attr_set = false;
  if (!attr_set) {
    cudaFuncSetAttribute(gemm_bf16_splitk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
    attr_set = true;
  }
  static const bool use_pdl = []() { const char* e = getenv("TN_PDL"); return e == nullptr || atoi(e) != 0; }();
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(((d.N + BN - 1) / BN) * S, (d.M + kBM - 1) / kBM, 1);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = S; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = use_pdl ? 2 : 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_bf16_splitk_kernel, tmA, tmB, p, S, stages);
  if (e == cudaSuccess) e = cudaGetLastError();
  return e == cudaSuccess ? nullptr : cudaGetErrorString(e);
}

}  // namespace tn
