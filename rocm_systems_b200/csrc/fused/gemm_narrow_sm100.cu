// Host side of the few-row bf16 GEMM (gemm_narrow_sm100.cuh): which shapes it takes, tile and split choice, cluster launch.
#include "gemm_narrow_sm100.cuh"

#include <algorithm>

#include "gemm_host.h"

namespace b200 {
namespace gemmn {
namespace {

template <int TN, bool W_MN, bool SWIGLU>
cudaError_t launch(const Params& p, int tiles, int groups, int S, cudaStream_t s) {
  auto kernel = gemmNarrowKernel<TN, W_MN, SWIGLU>;
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
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = (unsigned)S;
  at.val.clusterDim.y = 1;
  at.val.clusterDim.z = 1;
  q.attrs = &at;
  q.numAttrs = S > 1 ? 1 : 0;
  return cudaLaunchKernelEx(&q, kernel, p, S);
}

template <bool W_MN, bool SWIGLU>
cudaError_t dispatch(const Params& p, int tn, int tiles, int groups, int S, cudaStream_t s) {
  switch (tn) {
    case 16: return launch<16, W_MN, SWIGLU>(p, tiles, groups, S, s);
    case 32: return launch<32, W_MN, SWIGLU>(p, tiles, groups, S, s);
    case 64: return launch<64, W_MN, SWIGLU>(p, tiles, groups, S, s);
    default: return launch<128, W_MN, SWIGLU>(p, tiles, groups, S, s);
  }
}

}  // namespace

// Where this kernel is the faster one, measured over M 1 .. 1024, N 512 .. 28672, K 512 .. 14336 with the weights out of
// the L2. Up to 128 rows nearly everywhere (N 28672, K 4096, 128 rows: 48 us against 56 on CTA pairs; N 1024, K 512: 4 - 5 against
// 9). Above, W is read again for every 128 rows, and it pays only while the 256 x 256 tiles would leave half of the
// device idle: 512 x 4096 x 4096 23 us against 27, 512 x 4096 x 14336 58 against 73, but 512 x 6144 x 4096 31 against 28. Above 512
// rows never (768 x 4096 x 4096 30 against 28). Of those tiles, more than 128 CTAs are not split along K, which pays for a short
// reduction only (256 x 9216 x 512 9.7 us against 10.8, x 4096 32.9 against 29.6, 512 x 4608 x 4096 28.9 against 27.5), and below 1024
// steps of K two splits of 80 CTAs or more do not (256 x 8192 x 512 11.4 against 10.7, 512 x 4096 x 768 12.1 against 11.8).
bool prefersNarrow(int M, int N, int K) {
  if (M <= 128) return true;
  const int tiles = ((M + 255) / 256) * ((N + 255) / 256);
  if (M > 512 || 2 * tiles > gemm2::pairsOnDevice()) return false;
  const int ctas = ((M + 127) / 128) * ((N + BF - 1) / BF);
  if (ctas > 128) return K <= 1024;
  return K >= 1024 || ctas < 80;
}

// CTAs along K: as many as fill the device two to an SM. 4096 x 4096 on 16 rows takes 14.8 us with 2 splits, 10.8 - 11.4 with 4 - 8.
// One token tile: at most 240 CTAs, because from 128 feature tiles up the exchange costs more than the second CTA of an SM gives
// (16384 x 2048 on 16 rows: 15.2 us unsplit, 16.1 in two). A cluster beyond that number waits for a second wave (6144 x 4096: 13.5 us
// with 240 CTAs, 18.6 with 288). Up to 1024 steps of K the exchange of many or uneven parts outweighs the shorter loop: 1, 2 or 4 even
// parts (4096 x 512 on 128 rows: 12.1 us in seven, 10.4 on CTA pairs, 8.1 in four; 8192 x 1024 on 64 rows 10.7 in three, 9.7 in two),
// except where a dozen tiles leave most of the device free (512 x 1024 on one row: 4.4 us in eight, 4.9 in four).
int splitsFor(int tiles, int tokTiles, int kSteps) {
  const int S = std::max(1, std::min({kMaxSplit, kSteps, (tokTiles == 1 ? 240 : 256) / (tiles * tokTiles)}));
  if (kSteps > 16 || tiles * tokTiles <= 12) return S;
  return S >= 4 ? 4 : S >= 2 ? 2 : 1;
}

namespace {

cudaError_t run(Params& p, const void* X, const void* W, int xRows, int groups, int tn, int ldx, int ldw, bool wMn, cudaStream_t s) {
  if ((reinterpret_cast<uintptr_t>(p.C) & 15) || (p.ldc & 7)) return cudaErrorInvalidValue;  // as for the CTA-pair kernel, which stores wider pieces
  const bool okW = wMn ? gemm::makeTileMap(&p.mapW, W, (uint64_t)groups * p.K, p.N, ldw, 64, 2) : gemm::makeTileMap(&p.mapW, W, (uint64_t)groups * p.N, p.K, ldw, 64, 2);
  if (!okW || !gemm::makeTileMap(&p.mapX, X, xRows, p.K, ldx, tn, 2)) return cudaErrorInvalidValue;
  p.err = gemm::errWord();
  if (!p.err) return cudaErrorMemoryAllocation;
  const int tiles = (p.N + BF - 1) / BF, tokTiles = groups > 1 ? 1 : (p.M + tn - 1) / tn;
  const int S = splitsFor(tiles * groups, tokTiles, (p.K + BK - 1) / BK);
  if (p.gateUpTile) return dispatch<false, true>(p, tn, tiles, groups, S, s);
  return wMn ? dispatch<true, false>(p, tn, tiles, groups, S, s) : dispatch<false, false>(p, tn, tiles, groups, S, s);
}

}  // namespace

// C [M, N or N / 2] = X [M, K] * W [N, K]^T; wMn: W is stored [K, N]. gateUpTile != 0: SwiGLU over the interleaved rows of W (K-major).
cudaError_t gemmNarrowBf16(const void* X, const void* W, void* C, int M, int N, int K, int ldx, int ldw, int ldc, bool wMn, int gateUpTile, cudaStream_t s) {
  if (wMn && gateUpTile) return cudaErrorInvalidValue;
  Params p{};
  p.C = (__nv_bfloat16*)C;
  p.ldc = ldc;
  p.M = M;
  p.N = N;
  p.K = K;
  p.gateUpTile = gateUpTile;
  return run(p, X, W, M, 1, M <= 16 ? 16 : M <= 32 ? 32 : M <= 64 ? 64 : 128, ldx, ldw, wMn, s);
}

// C [groups * cap, N or N / 2] = X [groups * cap, K] * W_g^T over the first cnt[g] rows of every group, `avg` of them as a rule (it sizes the
// token tile: most groups fit one, and W is read again for every further one). wMn: W_g is stored [K, N], K % 64 == 0.
cudaError_t gemmNarrowGroupedBf16(const void* X, const void* W, void* C, const uint32_t* cnt, int groups, int cap, int avg, int N, int K, bool wMn, int gateUpTile,
                                  cudaStream_t s) {
  if (wMn && (gateUpTile || K % BK)) return cudaErrorInvalidValue;
  Params p{};
  p.C = (__nv_bfloat16*)C;
  p.ldc = gateUpTile ? N / 2 : N;
  p.M = cap;
  p.N = N;
  p.K = K;
  p.gateUpTile = gateUpTile;
  p.group.count = cnt;
  p.group.cap = cap;
  return run(p, X, W, groups * cap, groups, 3 * avg <= 2 * 32 ? 32 : 3 * avg <= 2 * 64 ? 64 : 128, K, wMn ? N : K, wMn, s);
}

}  // namespace gemmn
}  // namespace b200
