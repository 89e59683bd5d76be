// Host side of the block-scaled fp8 GEMM on CTA pairs (gemm_fp8_pair_sm100.cuh).
#include "gemm_fp8_pair_sm100.cuh"

#include <algorithm>

#include "gemm_host.h"

namespace b200 {
namespace gemm8p {
namespace {

template <bool GROUPED, bool SWIGLU>
auto pairKernel() {
  if constexpr (GROUPED) return &gemmFp8PairGroupedKernel;
  else return &gemmFp8PairKernel<SWIGLU>;
}

template <bool GROUPED, bool SWIGLU>
cudaError_t launch(const Params& p, int tiles, cudaStream_t s) {
  auto kernel = pairKernel<GROUPED, SWIGLU>();
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes);
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  kernel<<<2 * std::min(tiles, gemm2::pairsOnDevice()), kThreads, kSmemBytes, s>>>(p);  // cluster shape (2, 1, 1) is part of the kernel
  return cudaGetLastError();
}

}  // namespace

// Where pairs are faster than one CTA per 128 x 128 tile, from sweeps of M 136 .. 4096, N 512 .. 28672, K 512 .. 8192: a round of pairs
// (one 256 x 256 tile each) takes 1.66 - 1.77 times as long as a round of single CTAs, so they win where the other kernel needs at
// least 1.75 times the rounds. 4096 x 28672 x 8192: 1.09 ms against 1.39; 512 x 8192 x 8192 (one round against two): 53 us against 64;
// but 768 x 8192 x 4096 (two against three) 48.4 against 41.3 and 640 x 28672 x 4096 (five against eight) 115 against 105. A short
// reduction is mostly prologue and epilogue: with K 512 and two rounds 136 x 28672 takes 20.3 us against 18.7, from three on pairs are level or ahead.
bool prefersPair(int M, int N, int K) {
  auto rounds = [](long long tiles, int at) { return (tiles + at - 1) / at; };
  const long long two = rounds((long long)((M + BT - 1) / BT) * ((N + BT - 1) / BT), gemm2::pairsOnDevice());
  const long long one = rounds((long long)((M + 127) / 128) * ((N + 127) / 128), gemm::smCount());
  return 7 * two <= 4 * one && (K >= 1024 || two >= 3);
}

// C [M, N or N / 2] = A8 [M, K] * B8 [N, K]^T, lda / ldb in bytes; sA[kb * sABlock + row * sARow]. swiglu: B holds 64 gate and 64 up
// rows in turn, N is a multiple of 128.
cudaError_t gemmFp8Pair(const void* A8, const float* sA, size_t sABlock, size_t sARow, const void* B8, const float* sB, void* C, int M, int N, int K, int lda,
                        int ldb, int ldc, bool swiglu, cudaStream_t s) {
  if ((reinterpret_cast<uintptr_t>(C) & 15) || (ldc & 7)) return cudaErrorInvalidValue;  // rows of C are written in 16-byte pieces
  Params p{};
  if (!gemm::makeTileMap(&p.mapA, A8, M, K, lda, 128, 1) || !gemm::makeTileMap(&p.mapB, B8, N, K, ldb, 128, 1)) return cudaErrorInvalidValue;
  p.sA = sA;
  p.sABlock = sABlock;
  p.sARow = sARow;
  p.sB = sB;
  p.C = (__nv_bfloat16*)C;
  p.ldc = ldc;
  p.M = M;
  p.N = N;
  p.kBlocks = K / 128;
  p.tilesM = (M + BT - 1) / BT;
  p.tilesN = (N + BT - 1) / BT;
  p.err = gemm::errWord();
  if (!p.err) return cudaErrorMemoryAllocation;
  const int tiles = p.tilesM * p.tilesN;
  return swiglu ? launch<false, true>(p, tiles, s) : launch<false, false>(p, tiles, s);
}

// C [groups * cap, N / 2] = SwiGLU over A8 [groups * cap, K] * B8_g [N, K]^T on the first cnt[g] rows of every group; sA [groups * cap][K / 128],
// 64 gate and 64 up rows in turn, N % 256 == 0.
cudaError_t gemmFp8PairGroupedSwiglu(const void* A8, const float* sA, const void* B8, const float* sB, void* C, const uint32_t* cnt, int groups, int cap, int N, int K,
                                     cudaStream_t s) {
  if (reinterpret_cast<uintptr_t>(C) & 15) return cudaErrorInvalidValue;
  Params p{};
  if (groups > kMaxGroups || N % BT || !gemm::makeTileMap(&p.mapA, A8, (uint64_t)groups * cap, K, K, 128, 1) ||
      !gemm::makeTileMap(&p.mapB, B8, (uint64_t)groups * N, K, K, 128, 1))
    return cudaErrorInvalidValue;
  p.sA = sA;
  p.sABlock = 1;
  p.sARow = K / 128;
  p.sB = sB;
  p.C = (__nv_bfloat16*)C;
  p.ldc = N / 2;
  p.N = N;
  p.kBlocks = K / 128;
  p.tilesN = N / BT;
  p.cnt = cnt;
  p.groups = groups;
  p.cap = cap;
  p.err = gemm::errWord();
  if (!p.err) return cudaErrorMemoryAllocation;
  return launch<true, true>(p, groups * ((cap + BT - 1) / BT) * p.tilesN, s);  // at most so many tiles
}

}  // namespace gemm8p
}  // namespace b200
