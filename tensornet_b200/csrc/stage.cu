// Small inputs of a captured step from page-locked host memory to their static buffers, many in one launch.
#include "tn_ops.h"

namespace tn {

namespace {

constexpr int kThreads = 256;
constexpr int kFlight = 2;                      // 16-byte pieces a thread has on the way at once

// blockIdx.x walks the blocks of all pieces; a piece's first block is where the one before it ends.  Bound by the round trip over
// the host link (1 to 2 us), then by its rate; the copy engine takes 3.5 to 4 us for each of these however small, one behind the
// other with 2 us in between, and 2.5 to 3.4 us of the host for each call.  Twelve inputs of 8 KB (ten columns of ids,
// dense features, labels) 5.3 us, as copies 62.
__global__ void __launch_bounds__(kThreads) stage_inputs_kernel(const __grid_constant__ StagePieces a) {
  int p = 0;
  while (p + 1 < a.n && (int)blockIdx.x >= a.first[p + 1]) ++p;
  const char* src = static_cast<const char*>(a.src[p]);
  char* dst = static_cast<char*>(a.dst[p]);
  const int bytes = a.bytes[p], lo = ((int)blockIdx.x - a.first[p]) * kStageBlockBytes, hi = min(bytes, lo + kStageBlockBytes);
  const uintptr_t both = reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst);
  int done = lo;
  if ((both & 15) == 0) {
    const int n16 = (hi - lo) >> 4;
    const uint4* s = reinterpret_cast<const uint4*>(src + lo);
    uint4* d = reinterpret_cast<uint4*>(dst + lo);
    for (int i = threadIdx.x; i < n16; i += kFlight * kThreads) {
      uint4 x[kFlight];
#pragma unroll
      for (int q = 0; q < kFlight; ++q)
        if (i + q * kThreads < n16) x[q] = __ldcv(s + i + q * kThreads);        // (the host writes here between launches)
#pragma unroll
      for (int q = 0; q < kFlight; ++q)
        if (i + q * kThreads < n16) d[i + q * kThreads] = x[q];
    }
    done = lo + (n16 << 4);
  } else if ((both & 3) == 0) {
    const int n4 = (hi - lo) >> 2;
    for (int i = threadIdx.x; i < n4; i += kThreads) reinterpret_cast<unsigned*>(dst + lo)[i] = __ldcv(reinterpret_cast<const unsigned*>(src + lo) + i);
    done = lo + (n4 << 2);
  }
  for (int i = done + threadIdx.x; i < hi; i += kThreads) dst[i] = __ldcv(src + i);
}

}  // namespace

cudaError_t launch_stage_inputs(StagePieces& a, cudaStream_t st) {
  int blocks = 0;
  for (int p = 0; p < a.n; ++p) {
    a.first[p] = blocks;
    blocks += (a.bytes[p] + kStageBlockBytes - 1) / kStageBlockBytes;
  }
  if (blocks == 0) return cudaSuccess;
  stage_inputs_kernel<<<blocks, kThreads, 0, st>>>(a);
  return cudaGetLastError();
}

}  // namespace tn
