// Host side of the few-row block-scaled fp8 GEMM (gemm_narrow_fp8_sm100.cuh).
#include "gemm_narrow_fp8_sm100.cuh"

#include <algorithm>

#include "gemm_host.h"

namespace b200 {
namespace gemmn8 {
namespace {

template <int TN, bool SWIGLU>
cudaError_t launch(const Params& p, int tiles, int groups, int S, bool early, cudaStream_t s) {
  auto kernel = gemmNarrowFp8Kernel<TN, SWIGLU>;
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg<TN>::kSmemBytes);
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  cudaLaunchConfig_t q{};
  q.gridDim = dim3((unsigned)(S * tiles), (unsigned)((p.M + TN - 1) / TN), (unsigned)groups);
  q.blockDim = dim3(kThreads);
  q.dynamicSmemBytes = Cfg<TN>::kSmemBytes;
  q.stream = s;
  cudaLaunchAttribute at[2] = {};
  unsigned n = 0;
  if (S > 1) {
    at[n].id = cudaLaunchAttributeClusterDimension;
    at[n].val.clusterDim.x = (unsigned)S;
    at[n].val.clusterDim.y = 1;
    at[n++].val.clusterDim.z = 1;
  }
  if (early) {
    at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  q.attrs = at;
  q.numAttrs = n;
  return cudaLaunchKernelEx(&q, kernel, p, S);
}

template <bool SWIGLU>
cudaError_t dispatch(const Params& p, int tn, int tiles, int groups, int S, bool early, cudaStream_t s) {
  switch (tn) {
    case 16: return launch<16, SWIGLU>(p, tiles, groups, S, early, s);
    case 32: return launch<32, SWIGLU>(p, tiles, groups, S, early, s);
    default: return launch<64, SWIGLU>(p, tiles, groups, S, early, s);
  }
}

}  // namespace

// Where this kernel is the faster one, measured over M 1 .. 512, N 1024 .. 28672, K 512 .. 14336 with the weights out of the L2: up
// to 64 rows (4096 x 14336: 16 - 18 us against 41 on 128 x 128 tiles; 28672 x 4096: 24 against 41, at 64 rows level at 31), above
// only while the tiles leave half of the device idle, because every 64 rows read W again (128 x 4096 x 4096 12 us against 16, but
// 256 x 4096 x 4096 17 against 16).
bool prefersNarrow(int M, int N, int K) {
  const int tiles = (N + BF - 1) / BF * ((M + 63) / 64);
  const int S = std::max(1, std::min(kMaxSplit, 256 / tiles));
  if (K / BK > kMaxBlocks * S) return false;  // the scales of a CTA's part of K do not fit its table
  return M <= 64 || 2 * tiles <= gemm::smCount();
}

// C [M, N or N / 2] = X8 [M, K] * W8 [N, K]^T, ldx / ldw in bytes; sX[kb * sXBlock + row * sXRow]. early: the kernel in front is the
// quantiser of X, launched without the early start itself, and lets this one begin before it ends.
cudaError_t gemmNarrowFp8(const void* X8, const float* sX, size_t sXBlock, size_t sXRow, const void* W8, const float* sW, void* C, int M, int N, int K, int ldx,
                          int ldw, int ldc, bool swiglu, bool early, cudaStream_t s) {
  if ((reinterpret_cast<uintptr_t>(C) & 15) || (ldc & 7)) return cudaErrorInvalidValue;
  Params p{};
  p.sX = sX;
  p.sXBlock = sXBlock;
  p.sXRow = sXRow;
  p.sW = sW;
  p.C = (__nv_bfloat16*)C;
  p.ldc = ldc;
  p.M = M;
  p.N = N;
  p.kBlocks = K / BK;
  const int tn = M <= 16 ? 16 : M <= 32 ? 32 : 64;
  if (!gemm::makeTileMap(&p.mapW, W8, N, K, ldw, BF, 1) || !gemm::makeTileMap(&p.mapX, X8, M, K, ldx, tn, 1)) return cudaErrorInvalidValue;
  p.err = gemm::errWord();
  if (!p.err) return cudaErrorMemoryAllocation;
  // K is split until two CTAs share every SM (4096 x 14336 on 16 rows: 28 us with 2 splits, 17 with 4, 15.7 with 7 or 8).
  const int tiles = (N + BF - 1) / BF, tokTiles = (M + tn - 1) / tn;
  const int S = std::max(1, std::min({kMaxSplit, p.kBlocks, 256 / (tiles * tokTiles)}));
  return swiglu ? dispatch<true>(p, tn, tiles, 1, S, early, s) : dispatch<false>(p, tn, tiles, 1, S, early, s);
}

// C [groups * cap, N or N / 2] = X8 [groups * cap, K] * W8_g^T over the first cnt[g] rows of every group, `avg` of them as a rule;
// sX [groups * cap][K / 128], N % 128 == 0, K at most kMaxBlocks blocks.
cudaError_t gemmNarrowGroupedFp8(const void* X8, const float* sX, const void* W8, const float* sW, void* C, const uint32_t* cnt, int groups, int cap, int avg, int N,
                                 int K, bool swiglu, cudaStream_t s) {
  if (reinterpret_cast<uintptr_t>(C) & 15) return cudaErrorInvalidValue;
  Params p{};
  p.sX = sX;
  p.sXBlock = 1;
  p.sXRow = K / BK;
  p.sW = sW;
  p.C = (__nv_bfloat16*)C;
  p.ldc = swiglu ? N / 2 : N;
  p.M = cap;
  p.N = N;
  p.kBlocks = K / BK;
  p.group.count = cnt;
  p.group.cap = cap;
  const int tn = 3 * avg <= 2 * 32 ? 32 : 64;
  if (p.kBlocks > kMaxBlocks || !gemm::makeTileMap(&p.mapW, W8, (uint64_t)groups * N, K, K, BF, 1) || !gemm::makeTileMap(&p.mapX, X8, (uint64_t)groups * cap, K, K, tn, 1))
    return cudaErrorInvalidValue;
  p.err = gemm::errWord();
  if (!p.err) return cudaErrorMemoryAllocation;
  const int S = std::max(1, std::min({kMaxSplit, p.kBlocks, 256 / (N / BF * groups)}));
  return swiglu ? dispatch<true>(p, tn, N / BF, groups, S, false, s) : dispatch<false>(p, tn, N / BF, groups, S, false, s);
}

}  // namespace gemmn8
}  // namespace b200
