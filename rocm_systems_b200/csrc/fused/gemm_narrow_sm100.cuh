// bf16 GEMM for few rows of activations (a decode step, a small batch, a short prompt):
//   C[M, N] = X[M, K] * W[N, K]^T,  fp32 accumulation, bf16 out.
// The work is reading W once. The roles of the operands are swapped against the CTA-pair kernel: the 128 rows of the MMA
// are output FEATURES and its columns are the TN tokens, so a handful of tokens pads to 16 columns and not to 256 rows, and
// N / 128 tiles times the split of K give every SM a share of the weights however few tokens there are.
//
// The split of K: S CTAs of a cluster (S <= 8) multiply consecutive ranges of K for the same tile, park their fp32 partial
// tiles in their own shared memory, and after a cluster barrier each sums its share of the tile over the S partials through
// distributed shared memory, in the order of K: no workspace in device memory, no counters, one launch, and the result does not
// depend on timing.
//
// SWIGLU: W holds gate and up rows interleaved per `gateUpTile` rows (half of them gate, then the up rows of the same outputs);
// a tile is 64 gate rows and their 64 up rows, and its output 64 features of silu(gate) * up.
//
// Bound by the reads of W: 28672 x 4096 against 16 tokens 43 us = 5.4 TB/s (CTA-pair kernel 53 us), 6144 x 4096 13.5 us (26.2),
// 4096 x 14336 24 us (71). On the small ones the launch, the fill of the ring and the exchange of the partials (together about
// 4 us) are what is left above the reads.
//
// Warp 0 feeds a ring of stages of 64 reduction steps by TMA, warp 1 issues tcgen05.mma (M = 128, N = TN), warps 2..5 read
// the accumulator back. The output row segments of a tile are 256 contiguous bytes. Every wait is bounded.
#pragma once

#include "gemm_sm100.cuh"

namespace b200 {
namespace gemmn {

using gemm::BK;
constexpr int BF = 128;        // output features per tile
constexpr int kThreads = 192;
constexpr uint32_t kHalfBytes = 64 * BK * 2;  // one TMA box of W: 64 features x 64 reduction steps, either major
constexpr int kMaxSplit = 8;

template <int TN> struct Cfg {
  static constexpr uint32_t kWBytes = 2 * kHalfBytes;
  static constexpr uint32_t kXBytes = TN * BK * 2;
  static constexpr uint32_t kStageBytes = kWBytes + kXBytes;
  // Two CTAs share an SM, each with about 100 KB of loads in flight.
  static constexpr int kStages = TN == 16 ? 6 : TN == 32 ? 5 : TN == 64 ? 4 : 3;
  static constexpr uint32_t kTmemCols = TN < 32 ? 32 : TN;
  static constexpr size_t kSmemBytes = (size_t)kStages * kStageBytes + 1024 + 256;
  static_assert((size_t)TN * BF * 4 <= (size_t)kStages * kStageBytes, "the partial tile reuses the ring");
};

// Grouped form (the experts of a mixture): blockIdx.z is the group g, which owns rows [g * cap, g * cap + count[g]) of X and C and
// rows [g * N, (g + 1) * N) of W (stored [K, N]: rows [g * K, (g + 1) * K), K a multiple of 64). count == nullptr: one group of all M rows.
struct Group {
  const uint32_t* count;
  int cap;
};

struct Params {
  CUtensorMap mapW;  // K-major: [groups * N, K], box {64, 64}. MN-major: [groups * K, N], box {64, 64}
  CUtensorMap mapX;  // [M, K], box {64, TN}
  __nv_bfloat16* C;
  int ldc;
  int M, N, K;      // M: rows of X of the one group, N: rows of W per group
  int gateUpTile;   // SWIGLU: rows of W per interleaved block (half gate, half up)
  Group group;
  int* err;
};

__device__ __forceinline__ float4 ldSharedCluster4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

// Every CTA of the cluster has parked its partial tile, `part` [TN tokens][128 features] fp32, in its shared memory: this CTA adds
// up its share of the tile's pieces of 4 output features over the S partials, in the order of K, and stores them as bf16.
// C: the tile's first token row, n0: its first output feature, nOut: output features there are.
template <bool SWIGLU>
__device__ __forceinline__ void sumSplitsAndStore(const float* part, int S, int split, int tokens, __nv_bfloat16* C, int ldc, int n0, int nOut) {
  constexpr int kPerTok = (SWIGLU ? BF / 2 : BF) / 4;
  const int pieces = tokens * kPerTok;
  const int lo = (int)((long long)pieces * split / S), hi = (int)((long long)pieces * (split + 1) / S);
  const uint32_t base = sm100::smemAddr(part);
  auto sum4 = [&](int at) {  // `at`: float index into the partial tiles
    float4 v = *reinterpret_cast<const float4*>(part + at);
    if (S > 1) {
      v = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int s = 0; s < S; s++) {
        const float4 a = ldSharedCluster4(sm100::mapToCta(base + (uint32_t)at * 4, (uint32_t)s));
        v.x += a.x;
        v.y += a.y;
        v.z += a.z;
        v.w += a.w;
      }
    }
    return v;
  };
  for (int i = lo + (int)threadIdx.x; i < hi; i += kThreads) {
    const int tok = i / kPerTok, f = (i % kPerTok) * 4;
    float4 v = sum4(tok * BF + f);
    if constexpr (SWIGLU) {
      const float4 u = sum4(tok * BF + 64 + f);
      v.x = v.x / (1.f + __expf(-v.x)) * u.x;
      v.y = v.y / (1.f + __expf(-v.y)) * u.y;
      v.z = v.z / (1.f + __expf(-v.z)) * u.z;
      v.w = v.w / (1.f + __expf(-v.w)) * u.w;
    }
    const int n = n0 + f;
    if (n >= nOut) continue;
    __nv_bfloat16* dst = C + (size_t)tok * ldc + n;
    const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
    if (n + 4 <= nOut) {
      uint2 o;
      o.x = *reinterpret_cast<const uint32_t*>(&a);
      o.y = *reinterpret_cast<const uint32_t*>(&b);
      *reinterpret_cast<uint2*>(dst) = o;
    } else {
      dst[0] = a.x;
      if (n + 1 < nOut) dst[1] = a.y;
      if (n + 2 < nOut) dst[2] = b.x;
    }
  }
}

// Grid: x = split rank + S * feature tile, y = token tile, z = group; cluster (S, 1, 1).
template <int TN, bool W_MN, bool SWIGLU>
__global__ void __launch_bounds__(kThreads, 2) gemmNarrowKernel(const __grid_constant__ Params p, int S) {
  using C = Cfg<TN>;
  using namespace sm100;
  extern __shared__ uint8_t smemRaw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~(uintptr_t)1023);
  uint8_t* smemW = smem;
  uint8_t* smemX = smem + (size_t)C::kStages * C::kWBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (size_t)C::kStages * C::kStageBytes);
  uint64_t* full = bars;
  uint64_t* empty = bars + C::kStages;
  uint64_t* accFull = bars + 2 * C::kStages;
  uint32_t* tmemSlot = reinterpret_cast<uint32_t*>(accFull + 1);
  float* part = reinterpret_cast<float*>(smem);  // [TN][128] once the ring is done with

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  volatile int* err = p.err;
  const int split = blockIdx.x % S;
  const int tile = blockIdx.x / S;
  constexpr int kOut = SWIGLU ? BF / 2 : BF;  // output features of the tile
  const int n0 = tile * kOut;                 // the first of them
  // Rows of W in the two halves of the tile.
  int row0 = n0, row1 = n0 + 64;
  if constexpr (SWIGLU) {
    const int half = p.gateUpTile / 2;
    row0 = n0 / half * p.gateUpTile + n0 % half;
    row1 = row0 + half;
  }
  int kOff = 0;  // reduction steps of W before those of this group
  if constexpr (W_MN) {
    kOff = (int)blockIdx.z * p.K;
  } else {
    row0 += (int)blockIdx.z * p.N;
    row1 += (int)blockIdx.z * p.N;
  }
  const int tok0 = blockIdx.y * TN;
  const int xRow0 = (int)blockIdx.z * p.group.cap;
  const int rows = p.group.count ? min((int)p.group.count[blockIdx.z], p.group.cap) : p.M;
  if (tok0 >= rows) return;  // the same for the whole cluster
  const int kAll = (p.K + BK - 1) / BK;
  const int k0 = (int)((long long)kAll * split / S), k1 = (int)((long long)kAll * (split + 1) / S);

  if (threadIdx.x == 0) {
    prefetchTensorMap(&p.mapW);
    prefetchTensorMap(&p.mapX);
    for (int s = 0; s < C::kStages; s++) {
      mbarInit(&full[s], 1);
      mbarInit(&empty[s], 1);
    }
    mbarInit(accFull, 1);
    fenceBarrierInit();
  }
  if (warp == 1) {
    tmemAlloc(tmemSlot, C::kTmemCols);
    tmemRelinquish();
  }
  tcFenceBefore();
  __syncthreads();
  tcFenceAfter();
  const uint32_t tmem = *tmemSlot;

  if (warp == 0) {
    if (lane == 0) {
      bool ok = true;
      int stage = 0;
      uint32_t phase = 0;
      for (int k = k0; k < k1; k++) {
        if (!mbarWait(&empty[stage], phase ^ 1, err, gemm::ERR_PRODUCER_EMPTY)) { ok = false; break; }
        mbarArriveExpectTx(&full[stage], C::kStageBytes);
        uint8_t* sw = smemW + (size_t)stage * C::kWBytes;
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int row = h == 0 ? row0 : row1;
          if constexpr (W_MN) tmaLoad2d(sw + h * kHalfBytes, &p.mapW, row, kOff + k * BK, &full[stage]);
          else tmaLoad2d(sw + h * kHalfBytes, &p.mapW, k * BK, row, &full[stage]);
        }
        tmaLoad2d(smemX + (size_t)stage * C::kXBytes, &p.mapX, k * BK, xRow0 + tok0, &full[stage]);
        if (++stage == C::kStages) { stage = 0; phase ^= 1; }
      }
      if (!ok)
        for (int s = 0; s < C::kStages; s++) mbarWait(&full[s], 0, err, 0, 2000u);  // let loads in flight land
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = instrDescMajor(BF, TN, 1 /*bf16*/, W_MN ? 1u : 0u, 0u);
      bool ok = true;
      int stage = 0;
      uint32_t phase = 0;
      for (int k = k0; k < k1; k++) {
        if (!mbarWait(&full[stage], phase, err, gemm::ERR_MMA_FULL)) { ok = false; break; }
        tcFenceAfter();
        const uint32_t wAddr = smemAddr(smemW + (size_t)stage * C::kWBytes);
        const uint32_t xAddr = smemAddr(smemX + (size_t)stage * C::kXBytes);
#pragma unroll
        for (int kk = 0; kk < BK / 16; kk++) {
          const uint64_t dw = W_MN ? smemDescSw128Mn(wAddr + kk * 2048, kHalfBytes) : smemDescSw128(wAddr + kk * 32);
          mmaF16(tmem, dw, smemDescSw128(xAddr + kk * 32), idesc, k > k0 || kk > 0);
        }
        mmaCommit(&empty[stage]);
        if (++stage == C::kStages) { stage = 0; phase ^= 1; }
      }
      if (ok) mmaCommit(accFull);
    }
    __syncwarp();
  } else {
    const int q = warp & 3;
    if (mbarWait(accFull, 0, err, gemm::ERR_EPI_ACC_FULL)) {
      tcFenceAfter();
      const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16);
      float* dst = part + q * 32 + lane;
      constexpr int kChunk = TN < 32 ? 16 : 32;
#pragma unroll 1
      for (int c = 0; c < TN; c += kChunk) {
        uint32_t acc[kChunk];
        if constexpr (TN < 32) tmemLoad16(taddr + c, acc);
        else tmemLoad32(taddr + c, acc);
        tmemLoadWait();
#pragma unroll
        for (int i = 0; i < kChunk; i++) dst[(c + i) * BF] = __uint_as_float(acc[i]);
      }
    }
    __syncwarp();
  }
  tcFenceBefore();
  if (S > 1) {
    clusterArrive();
    clusterWait();
  } else {
    __syncthreads();
  }
  sumSplitsAndStore<SWIGLU>(part, S, split, min(TN, rows - tok0), p.C + (size_t)(xRow0 + tok0) * p.ldc, p.ldc, n0, SWIGLU ? p.N / 2 : p.N);
  if (S > 1) {
    clusterArrive();  // no CTA leaves while a peer still reads its partial tile
    clusterWait();
  } else {
    __syncthreads();
  }
  if (warp == 1) tmemDealloc(tmem, C::kTmemCols);
}

}  // namespace gemmn
}  // namespace b200
