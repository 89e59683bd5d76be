// Block-scaled fp8 (e4m3) GEMM (main loop in gemm_fp8_sm100.cuh) as a plain kernel, and the quantisers that feed it.
#include "gemm_fp8_sm100.cuh"
#include "gemm_host.h"

namespace b200 {
namespace gemm8 {

__global__ void __launch_bounds__(kThreads, 1) gemmFp8BlockKernel(const __grid_constant__ Params p) {
  extern __shared__ uint8_t smemRaw[];
  PlainPolicy8 pol{p};
  gemmFp8Cta(p, pol, blockIdx.x, gridDim.x, smemRaw);
}

// ---- quantisers ------------------------------------------------------------------------------------------------
// Activations: one scale per row and 128 channels. A CTA takes 8 rows (a warp each, so that the 8 scales of a group, neighbours in
// the table, go to one 32-byte sector) and up to 4 rounds of 256 channels: lane l holds channels (32 j + l) * 8 .. + 8 of round j, a
// half-warp is one group, and all its loads are in flight at once. With a whole row per warp, one round after the other,
// 32 rows of 14336 channels took 31 us, 56 round trips to memory; 4096 x 4096 took 20 us, half of it in the divisions.
constexpr int kQuantRounds = 4;
__global__ void __launch_bounds__(256) quantRows1x128(const __nv_bfloat16* __restrict__ x, uint8_t* __restrict__ q, float* __restrict__ s, int M, int K, int ldx,
                                                      int ldq, int lds) {
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5);
  sm100::gridLaunchDependents();
  if (row >= M) return;
  const int groups = K / 128;
  const uint4* xr = reinterpret_cast<const uint4*>(x + (size_t)row * ldx);
  uint2* qr = reinterpret_cast<uint2*>(q + (size_t)row * ldq);
  const int j0 = blockIdx.y * kQuantRounds;
  uint4 raw[kQuantRounds];
#pragma unroll
  for (int j = 0; j < kQuantRounds; j++) {
    raw[j] = make_uint4(0, 0, 0, 0);
    if ((j0 + j) * 2 + (lane >> 4) < groups) raw[j] = xr[(j0 + j) * 32 + lane];
  }
#pragma unroll
  for (int j = 0; j < kQuantRounds; j++) {
    const int g = (j0 + j) * 2 + (lane >> 4);
    float f[8], amax = 0.f;
    unpackBf16x8(raw[j], f, amax);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    const QuantScale qs(amax);
    if (g < groups) {
      qr[(j0 + j) * 32 + lane] = qs.codes(f);
      if ((lane & 15) == 0) s[(size_t)g * lds + row] = qs.scale;
    }
  }
}

// Weights: one scale per 128 x 128 block. One CTA of 256 threads per block; thread t holds 8 channels of rows
// (t / 16) + 16 i, i = 0..7.
__global__ void __launch_bounds__(256) quantBlocks128x128(const __nv_bfloat16* w, uint8_t* q, float* s, int N, int K, int ldw, int ldq) {
  __shared__ float red[8];
  const int kb = blockIdx.x, nb = blockIdx.y;
  const int t = threadIdx.x, sub = t & 15, r0 = t >> 4;
  uint4 raw[8];
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int row = nb * 128 + r0 + 16 * i;
    raw[i] = make_uint4(0, 0, 0, 0);
    if (row < N) raw[i] = *reinterpret_cast<const uint4*>(w + (size_t)row * ldw + (size_t)kb * 128 + sub * 8);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw[i]);
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const float2 pr = __bfloat1622float2(h[e]);
      amax = fmaxf(amax, fmaxf(fabsf(pr.x), fabsf(pr.y)));
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if ((t & 31) == 0) red[t >> 5] = amax;
  __syncthreads();
  amax = red[0];
#pragma unroll
  for (int i = 1; i < 8; i++) amax = fmaxf(amax, red[i]);
  const QuantScale qs(amax);
  if (t == 0) s[(size_t)nb * gridDim.x + kb] = qs.scale;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int row = nb * 128 + r0 + 16 * i;
    if (row >= N) continue;
    float f[8], unused = 0.f;
    unpackBf16x8(raw[i], f, unused);
    *reinterpret_cast<uint2*>(q + (size_t)row * ldq + (size_t)kb * 128 + sub * 8) = qs.codes(f);
  }
}

}  // namespace gemm8
}  // namespace b200

using namespace b200;

static int gemmFp8BlockTn(const void* A8, const float* sA, const void* B8, const float* sB, void* C, int M, int N, int K, int lda, int ldb, int ldc, int maxCtas,
                          bool early, cudaStream_t st);

extern "C" {

// q[M, K] (e4m3, row stride ldq bytes) and s[K / 128][lds] from x[M, K] (bf16, row stride ldx elements). K % 128 == 0.
// lds >= M is the row stride of the scale table: a rank that owns rows [r0, r0 + M) of a larger matrix passes the table's
// full width and s + r0.
int b200ops_quant_e4m3_1x128_strided(const void* x, void* q, float* s, int M, int K, int ldx, int ldq, int lds, cudaStream_t st) {
  if (M <= 0 || K <= 0) return 0;
  if ((K & 127) || (ldx & 7) || (ldq & 7) || lds < M || ((uintptr_t)x & 15) || ((uintptr_t)q & 7)) return (int)cudaErrorInvalidValue;
  gemm8::quantRows1x128<<<dim3((M + 7) / 8, (K + 256 * gemm8::kQuantRounds - 1) / (256 * gemm8::kQuantRounds)), 256, 0, st>>>((const __nv_bfloat16*)x, (uint8_t*)q, s, M, K, ldx, ldq, lds);
  return (int)cudaGetLastError();
}
int b200ops_quant_e4m3_1x128(const void* x, void* q, float* s, int M, int K, int ldx, int ldq, cudaStream_t st) {
  return b200ops_quant_e4m3_1x128_strided(x, q, s, M, K, ldx, ldq, M, st);
}

// q[N, K] (e4m3) and s[ceil(N / 128)][K / 128] from w[N, K] (bf16). K % 128 == 0.
int b200ops_quant_e4m3_128x128(const void* w, void* q, float* s, int N, int K, int ldw, int ldq, cudaStream_t st) {
  if (N <= 0 || K <= 0) return 0;
  if ((K & 127) || (ldw & 7) || (ldq & 7) || ((uintptr_t)w & 15) || ((uintptr_t)q & 7)) return (int)cudaErrorInvalidValue;
  dim3 grid(K / 128, (N + 127) / 128);
  gemm8::quantBlocks128x128<<<grid, 256, 0, st>>>((const __nv_bfloat16*)w, (uint8_t*)q, s, N, K, ldw, ldq);
  return (int)cudaGetLastError();
}

// C[M, N] (bf16, ldc) = block-scaled A8[M, K] (lda bytes) * B8[N, K]^T (ldb bytes); sA [K / 128][M], sB [ceil(N / 128)][K / 128].
int b200ops_gemm_fp8_block_tn(const void* A8, const float* sA, const void* B8, const float* sB, void* C, int M, int N, int K, int lda, int ldb, int ldc,
                              int maxCtas, cudaStream_t st) {
  return gemmFp8BlockTn(A8, sA, B8, sB, C, M, N, K, lda, ldb, ldc, maxCtas, false, st);
}

// C[M, N] (bf16, row stride N) = x[M, K] (bf16, row stride ldx) * B8[N, K]^T with x quantised on the way; `scratch` holds the codes and
// behind them the scales: M * K + M * (K / 128) * 4 bytes, 16-byte aligned.
int b200ops_fp8_linear(const void* x, void* scratch, const void* B8, const float* sB, void* C, int M, int N, int K, int ldx, int ldb, cudaStream_t st) {
  float* s = reinterpret_cast<float*>((uint8_t*)scratch + (size_t)M * K);
  const int e = b200ops_quant_e4m3_1x128(x, scratch, s, M, K, ldx, K, st);
  return e ? e : gemmFp8BlockTn(scratch, s, B8, sB, C, M, N, K, K, ldb, N, 0, true, st);
}

}  // extern "C"

static int gemmFp8BlockTn(const void* A8, const float* sA, const void* B8, const float* sB, void* C, int M, int N, int K, int lda, int ldb, int ldc, int maxCtas,
                          bool early, cudaStream_t st) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((K & 127) || ((uintptr_t)C & 15) || (ldc & 7)) return (int)cudaErrorInvalidValue;
  if (maxCtas == 0 && gemmn8::prefersNarrow(M, N, K))
    return (int)gemmn8::gemmNarrowFp8(A8, sA, (size_t)M, 1, B8, sB, C, M, N, K, lda, ldb, ldc, false, early, st);
  if (maxCtas == 0 && gemm8p::prefersPair(M, N, K))
    return (int)gemm8p::gemmFp8Pair(A8, sA, (size_t)M, 1, B8, sB, C, M, N, K, lda, ldb, ldc, false, st);
  gemm8::Params p{};
  if (!gemm::makeTileMap(&p.mapA, A8, M, K, lda, gemm::BM, 1) || !gemm::makeTileMap(&p.mapB, B8, N, K, ldb, gemm8::BN, 1)) return (int)cudaErrorInvalidValue;
  p.sA = sA;
  p.sB = sB;
  p.C = (__nv_bfloat16*)C;
  p.M = M;
  p.N = N;
  p.K = K;
  p.ldc = ldc;
  p.tilesM = (M + gemm::BM - 1) / gemm::BM;
  p.tilesN = (N + gemm8::BN - 1) / gemm8::BN;
  p.kBlocks = K / 128;
  p.err = gemm::errWord();
  if (!p.err) return (int)cudaErrorMemoryAllocation;
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(gemm8::gemmFp8BlockKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gemm8::kSmemBytes);
    if (e != cudaSuccess) return (int)e;
    configured[dev] = true;
  }
  int ctas = gemm::smCount();
  if (maxCtas > 0 && maxCtas < ctas) ctas = maxCtas;
  const int tiles = p.tilesM * p.tilesN;
  if (tiles < ctas) ctas = tiles;
  gemm8::gemmFp8BlockKernel<<<ctas, gemm8::kThreads, gemm8::kSmemBytes, st>>>(p);
  return (int)cudaGetLastError();
}
