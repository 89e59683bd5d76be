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

int tokensPerTile(int M) { return M <= 16 ? 16 : M <= 32 ? 32 : 64; }

// CTAs along K for `ctas` tiles: as many as put two CTAs on every SM (4096 x 14336 on 16 rows: 28 us with 2 splits, 17 with 4, 15.7 with 7
// or 8). Up to 2048 steps of K the exchange of many or uneven parts outweighs the shorter loop, so at most four, as even as they come (3072 x 1024 on
// 48 rows: 7.6 us in eight, 6.0 in four; x 2048 8.4, 7.5), and none for 512 steps of many tiles (8192 x 512 on 16 rows 6.3 in four, 5.8
// in one), unless a dozen tiles leave most of the device free (512 x 2048 on 16 rows: 4.9 us in eight, 5.7 in four).
int splitsFor(int ctas, int kBlocks) {
  const int S = std::max(1, std::min({kMaxSplit, kBlocks, 256 / ctas}));
  if (kBlocks > 16 || ctas <= (kBlocks <= 6 ? 16 : 12)) return S;
  if (kBlocks <= 4 && ctas >= 48) return 1;
  const int per = (kBlocks + std::min(S, 4) - 1) / std::min(S, 4);
  return (kBlocks + per - 1) / per;
}

// Where this kernel is the faster one, measured over M 1 .. 512, N 512 .. 28672, K 512 .. 8192 with the weights out of the L2 (graphs of
// GEMMs), against a CTA per 128 x 128 tile. Up to 64 rows one tile holds them all, and it is ahead nearly everywhere (4096 x 4096
// on 16 rows 1.7 times, 28672 x 2048 1.5 times), except where 80 to 148 tiles are one round of the other kernel and too many to split here
// (14336 x 1024 on 64 rows: 11.1 us against 8.8), and with up to 1024 steps from 48 tiles on (6144 x 512 on 64 rows 7.5 against 6.5). Above, every
// 64 rows read W again: it takes few tiles and long reductions (128 x 4096 x 4096, 64 tiles: 1.3 times ahead; 128 x 6144 x
// 4096, 96 tiles: 0.96; 192 x 3072 x 512: 8.3 us against 6.2).
bool prefersNarrow(int M, int N, int K) {
  const int tokTiles = (M + tokensPerTile(M) - 1) / tokensPerTile(M), ctas = (N + BF - 1) / BF * tokTiles;
  if (K / BK > kMaxBlocks * splitsFor(ctas, K / BK)) return false;  // the scales of a CTA's part of K do not fit its table
  if (M <= 16) return true;
  if (M <= 32) return K >= 1536 || ctas < 80 || ctas > gemm::smCount();
  const bool between = K > 512 && K < 1024;  // 5 to 7 blocks do not split evenly
  if (M <= 64) return ctas <= 64 ? K >= 1536 || ctas < (between ? 17 : 48) : ctas <= 85 ? K >= 4096 : ctas > gemm::smCount();
  return ctas <= (K >= 4096 ? 80 : K >= 1536 ? 64 : K >= 1024 ? (tokTiles == 2 ? 48 : 32) : between ? 16 : 32);
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
  const int tn = tokensPerTile(M);
  if (!gemm::makeTileMap(&p.mapW, W8, N, K, ldw, BF, 1) || !gemm::makeTileMap(&p.mapX, X8, M, K, ldx, tn, 1)) return cudaErrorInvalidValue;
  p.err = gemm::errWord();
  if (!p.err) return cudaErrorMemoryAllocation;
  const int tiles = (N + BF - 1) / BF, S = splitsFor(tiles * ((M + tn - 1) / tn), p.kBlocks);
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
  const int S = splitsFor(N / BF * groups, p.kBlocks);
  return swiglu ? dispatch<true>(p, tn, N / BF, groups, S, false, s) : dispatch<false>(p, tn, N / BF, groups, S, false, s);
}

}  // namespace gemmn8
}  // namespace b200
