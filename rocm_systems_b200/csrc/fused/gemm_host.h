// Host-side helpers shared by the tcgen05 GEMM and the fused GEMM+collective launchers.
#pragma once

#include <cuda.h>
#include <cuda_runtime_api.h>
#include <stdint.h>

namespace b200 {
namespace gemm {

bool makeTileMap(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t boxRows, uint32_t elemBytes);
int* errWord();   // per-device error word of the tcgen05 kernels (device memory)
int smCount();
cudaError_t gemmBf16TN(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc, int bn, int maxCtas, cudaStream_t s);

}  // namespace gemm
namespace gemm2 {
int pairsOnDevice();
cudaError_t gemmPairBf16(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc, bool aMn, bool bMn, int bn, int maxCtas,
                         cudaStream_t s);
cudaError_t gemmPairSwiglu(const void* A, const void* W, void* C, int M, int N, int K, cudaStream_t s);
cudaError_t gemmPairGroupedRows(const void* A, const void* W, void* C, const uint32_t* cnt, int groups, int cap, int N, int K, bool wMn, bool swiglu, cudaStream_t s);
cudaError_t gemmPairGroupedSum(const void* A, const void* B, void* C, const uint32_t* cnt, int groups, int cap, int M, int N, cudaStream_t s);
}  // namespace gemm2
namespace gemmn {
bool prefersNarrow(int M, int N, int K);
cudaError_t gemmNarrowBf16(const void* X, const void* W, void* C, int M, int N, int K, int ldx, int ldw, int ldc, bool wMn, int gateUpTile, cudaStream_t s);
cudaError_t gemmNarrowGroupedBf16(const void* X, const void* W, void* C, const uint32_t* cnt, int groups, int cap, int avg, int N, int K, bool wMn, int gateUpTile,
                                  cudaStream_t s);
}  // namespace gemmn
namespace gemmn8 {
bool prefersNarrow(int M, int N, int K);
cudaError_t gemmNarrowFp8(const void* X8, const float* sX, size_t sXBlock, size_t sXRow, const void* W8, const float* sW, void* C, int M, int N, int K, int ldx,
                          int ldw, int ldc, bool swiglu, bool early, cudaStream_t s);
cudaError_t gemmNarrowGroupedFp8(const void* X8, const float* sX, const void* W8, const float* sW, void* C, const uint32_t* cnt, int groups, int cap, int avg, int N,
                                 int K, bool swiglu, cudaStream_t s);
}  // namespace gemmn8
namespace gemm8p {
bool prefersPair(int M, int N, int K);
cudaError_t gemmFp8Pair(const void* A8, const float* sA, size_t sABlock, size_t sARow, const void* B8, const float* sB, void* C, int M, int N, int K, int lda,
                        int ldb, int ldc, bool swiglu, cudaStream_t s);
cudaError_t gemmFp8PairGroupedSwiglu(const void* A8, const float* sA, const void* B8, const float* sB, void* C, const uint32_t* cnt, int groups, int cap, int N, int K,
                                     cudaStream_t s);
}  // namespace gemm8p
}  // namespace b200
