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
}  // namespace gemm2
namespace gemmn {
bool prefersNarrow(int M, int N);
cudaError_t gemmNarrowBf16(const void* X, const void* W, void* C, int M, int N, int K, int ldx, int ldw, int ldc, bool wMn, int gateUpTile, cudaStream_t s);
}  // namespace gemmn
namespace gemmn8 {
bool prefersNarrow(int M, int N, int K);
cudaError_t gemmNarrowFp8(const void* X8, const float* sX, size_t sXBlock, size_t sXRow, const void* W8, const float* sW, void* C, int M, int N, int K, int ldx,
                          int ldw, int ldc, bool swiglu, bool early, cudaStream_t s);
}  // namespace gemmn8
}  // namespace b200
