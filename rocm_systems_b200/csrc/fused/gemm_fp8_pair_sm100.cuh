// Block-scaled fp8 (e4m3) GEMM on CTA pairs (tcgen05 cta_group::2): the arithmetic of gemm_fp8_sm100.cuh (one fp32 scale per
// activation row and 128 channels, one per 128 x 128 weight block, every 128-deep partial product folded into fp32 registers in the
// order of K) on 256 x 256 tiles shared by two CTAs as in gemm_pair_sm100.cuh.
//
// Why pairs: a K block of a 128 x 128 tile moves 32 KB through shared memory for the load and 32 KB again for the MMAs, twice what
// an SM can move in the 256 cycles the MMAs take. In a 256 x 256 tile each CTA loads and reads 32 KB for 512 cycles of MMAs,
// which just fits. The price is tensor memory: a partial product takes 256 of the 512 columns, so only two are in flight,
// and the eight epilogue warps of each CTA have one block's MMA time to fold a block: 128 columns per thread, the next
// block's scales already loaded, the buffer given back before the last FMAs.
//
// Bound by that fold: 4096 x 8192 x 4096 takes 184 us, 135 without the FMAs (packed two to an instruction they took 207, as they cost moves
// and spills); 4096 x 28672 x 4096 551 us = 1.75 PFLOP/s, 622 on the one-CTA kernel.
//
// Warp 0 of each CTA loads its 128 rows of A and its half of B's 256 rows, the even CTA's warp 1 issues the MMAs, and one commit per
// block, addressed to both CTAs, says that the stage is free AND the product is ready. Every wait is bounded.
//
// GROUPED: the rows are those of the experts of a mixture, `cap` rows reserved per expert of which cnt[e] hold tokens; the
// persistent CTAs share a list of 256-row blocks that hold tokens.
#pragma once

#include "gemm_fp8_sm100.cuh"

namespace b200 {
namespace gemm8p {

using gemm8::BK;
constexpr int kThreads = 384;  // a warpgroup whose warps 0 and 1 load and multiply, two of epilogue warps
// Registers per thread of the two kinds: launched with 168 (384 x 168 = 64512), 128 x 40 + 256 x 232 = 64512 afterwards.
constexpr int kMainRegs = 40, kEpiRegs = 232;
constexpr int BT = 256;    // tile rows and columns
constexpr int kStages = 6;
constexpr int kAccBufs = 2;
static_assert(kAccBufs <= kStages, "a product that is not folded yet keeps its stage's barrier from completing a second time");
constexpr int kFold = 32;      // columns loaded and folded at a time
constexpr int kAccCols = 128;  // accumulator columns per epilogue thread: one half of the tile, one weight scale
constexpr uint32_t kABytes = 128 * BK;
constexpr uint32_t kStageBytes = 2 * kABytes;  // this CTA's rows of A and its half of B
constexpr uint32_t kTmemCols = kAccBufs * BT;
constexpr uint32_t kEpiBytesPerWarp = 32 * 64 * 2;
constexpr size_t kSmemBytes = (size_t)kStages * kStageBytes + 1024 + 256 + 8 * kEpiBytesPerWarp;
constexpr int kMaxGroups = 64;

struct Params {
  CUtensorMap mapA;  // [rows, K] bytes, box {128, 128}
  CUtensorMap mapB;  // [groups * N, K] bytes, box {128, 128}
  const float* sA;   // scale of row r, block kb: sA[kb * sABlock + r * sARow]
  size_t sABlock, sARow;
  const float* sB;   // [groups * ceil(N / 128)][kBlocks]
  __nv_bfloat16* C;
  int ldc;
  int M, N, kBlocks;      // M: rows (not grouped); N: weight rows (per group)
  int tilesM, tilesN;
  const uint32_t* cnt;    // GROUPED: rows of every group (may exceed cap)
  int groups, cap;
  int* err;
};

template <bool GROUPED, bool SWIGLU>
__device__ __forceinline__ void gemmFp8PairCta(const Params& p, uint8_t* smemRaw) {
  using namespace sm100;
  __shared__ int prefix[GROUPED ? kMaxGroups + 1 : 1];  // row blocks with tokens before group g
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~(uintptr_t)1023);
  uint8_t* smemA = smem;
  uint8_t* smemB = smem + (size_t)kStages * kABytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (size_t)kStages * kStageBytes);
  uint64_t* full = bars;                   // used in the even CTA only: both CTAs' loads of a stage have landed
  uint64_t* done = bars + kStages;         // one set per CTA: the MMAs of a stage are complete
  uint64_t* accEmpty = bars + 2 * kStages; // used in the even CTA only: all 16 epilogue warps have read a product
  uint32_t* tmemSlot = reinterpret_cast<uint32_t*>(accEmpty + kAccBufs);
  uint8_t* epiStage = reinterpret_cast<uint8_t*>(bars) + 256;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t cr = clusterCtaRank();
  volatile int* err = p.err;

  if constexpr (GROUPED) {  // the counts are read side by side, then summed
    for (int g = threadIdx.x; g <= p.groups; g += kThreads) prefix[g] = g == 0 ? 0 : (min((int)p.cnt[g - 1], p.cap) + BT - 1) / BT;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    prefetchTensorMap(&p.mapA);
    prefetchTensorMap(&p.mapB);
    for (int s = 0; s < kStages; s++) {
      mbarInit(&full[s], 1);
      mbarInit(&done[s], 1);
    }
    for (int b = 0; b < kAccBufs; b++) mbarInit(&accEmpty[b], 16);
    fenceBarrierInit();
    if constexpr (GROUPED)
      for (int g = 0; g < p.groups; g++) prefix[g + 1] += prefix[g];
  }
  if (warp == 1) {
    tmemAllocPair(tmemSlot, kTmemCols);
    tmemRelinquishPair();
  }
  tcFenceBefore();
  __syncthreads();
  clusterArrive();  // the partner's barriers exist before anything arrives on them
  clusterWait();
  tcFenceAfter();
  const uint32_t tmem = *tmemSlot;

  const int numTiles = GROUPED ? prefix[p.groups] * p.tilesN : p.tilesM * p.tilesN;
  const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
  // First row of A, rows of A end, first row of B, first row of weight blocks, output column block of tile t.
  struct Tile {
    int aRow, aEnd, bRow, sRow, tn;
  };
  auto tileAt = [&](int t) {
    Tile o;
    if constexpr (GROUPED) {
      const int rb = t / p.tilesN;
      o.tn = t - rb * p.tilesN;
      int g = 0;
      while (prefix[g + 1] <= rb) g++;
      o.aRow = g * p.cap + (rb - prefix[g]) * BT;
      o.aEnd = g * p.cap + min((int)p.cnt[g], p.cap);
      o.bRow = g * p.N + o.tn * BT;
      o.sRow = g * (p.N / 128) + o.tn * 2;
    } else {
      int tm;
      gemm::bandedCoord(t, p.tilesM, p.tilesN, tm, o.tn);
      o.aRow = tm * BT;
      o.aEnd = p.M;
      o.bRow = o.tn * BT;
      o.sRow = o.tn * 2;
    }
    return o;
  };

  if (warp < 4) {
    setMaxRegsDown<kMainRegs>();
    if (warp == 0 && lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = pair; t < numTiles && ok; t += npairs) {
        const Tile o = tileAt(t);
        const int aRow = o.aRow + (int)cr * 128, bRow = o.bRow + (int)cr * 128;
        for (int kb = 0; kb < p.kBlocks; kb++) {
          if (!mbarWait(&done[stage], phase ^ 1, err, gemm::ERR_PRODUCER_EMPTY)) { ok = false; break; }
          const uint32_t fullAddr = mapToCta(smemAddr(&full[stage]), 0);
          if (cr == 0) mbarArriveExpectTx(&full[stage], 2 * kStageBytes);  // both CTAs' bytes land here
          tmaLoad2dPair(smemA + (size_t)stage * kABytes, &p.mapA, kb * BK, aRow, fullAddr);
          tmaLoad2dPair(smemB + (size_t)stage * kABytes, &p.mapB, kb * BK, bRow, fullAddr);
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
      }
      if (!ok && cr == 0)
        for (int s = 0; s < kStages; s++) mbarWait(&full[s], 0, err, 0, 2000u);  // let loads in flight land
    }
    if (warp == 1 && lane == 0 && cr == 0) {
      constexpr uint32_t idesc = instrDesc(BT, BT, 0 /*e4m3*/);
      int stage = 0;
      uint32_t phase = 0, n = 0;
      bool ok = true;
      for (int t = pair; t < numTiles && ok; t += npairs) {
        for (int kb = 0; kb < p.kBlocks; kb++, n++) {
          const uint32_t b = n % kAccBufs;
          if (!mbarWait(&full[stage], phase, err, gemm::ERR_MMA_FULL)) { ok = false; break; }
          if (!mbarWait(&accEmpty[b], ((n / kAccBufs) & 1) ^ 1, err, gemm::ERR_MMA_ACC_EMPTY)) { ok = false; break; }
          tcFenceAfter();
          const uint32_t aAddr = smemAddr(smemA + (size_t)stage * kABytes), bAddr = smemAddr(smemB + (size_t)stage * kABytes);
#pragma unroll
          for (int kk = 0; kk < BK / 32; kk++) mmaF8Pair(tmem + b * BT, smemDescSw128(aAddr + kk * 32), smemDescSw128(bAddr + kk * 32), idesc, kk != 0);
          mmaCommitBoth(smemAddr(&done[stage]));
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
      }
    }
    __syncwarp();
  } else {
    setMaxRegsUp<kEpiRegs>();
    const int q = warp & 3, h = (warp - 4) >> 2;  // lanes 32 q .. of tensor memory, columns 128 h .. of the tile
    uint8_t* sw = epiStage + (size_t)(warp - 4) * kEpiBytesPerWarp;
    const uint32_t release = mapToCta(smemAddr(accEmpty), 0);
    int stage = 0;
    uint32_t phase = 0, n = 0;
    bool ok = true;
    for (int t = pair; t < numTiles && ok; t += npairs) {
      const Tile o = tileAt(t);
      const int row0 = o.aRow + (int)cr * 128 + q * 32, row = row0 + lane;
      // A row or a block of weight rows beyond the edge: nothing of it is stored, its scale is not read.
      const bool live = row < o.aEnd && o.tn * BT + h * 128 < p.N;
      const float* sA = p.sA + (size_t)(live ? row : 0) * p.sARow;
      const float* sB = p.sB + (size_t)(live ? o.sRow + h : 0) * p.kBlocks;
      float acc[kAccCols];
#pragma unroll
      for (int i = 0; i < kAccCols; i++) acc[i] = 0.f;
      float a = live ? __ldg(sA) : 0.f, b = live ? __ldg(sB) : 0.f;
      for (int kb = 0; kb < p.kBlocks; kb++, n++) {
        const float s = a * b;
        if (kb + 1 < p.kBlocks && live) {  // in flight across the fold of this block
          a = __ldg(sA + (size_t)(kb + 1) * p.sABlock);
          b = __ldg(sB + kb + 1);
        }
        if (!mbarWait(&done[stage], phase, err, gemm::ERR_EPI_ACC_FULL)) { ok = false; break; }
        if (++stage == kStages) { stage = 0; phase ^= 1; }
        tcFenceAfter();
        const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + (n % kAccBufs) * BT + h * 128;
        // Two loads take turns, so that one is under way while the other's columns are folded.
        uint32_t x[2][kFold];
        tmemLoad32(taddr, x[0]);
#pragma unroll
        for (int c = 0; c < kAccCols / kFold; c++) {
          tmemLoadWait();
          if (c + 1 < kAccCols / kFold) {
            tmemLoad32(taddr + (c + 1) * kFold, x[(c + 1) & 1]);
          } else {
            tcFenceBefore();
            __syncwarp();
            if (lane == 0) mbarArriveCluster(release + (n % kAccBufs) * 8);
          }
#pragma unroll
          for (int i = 0; i < kFold; i++) acc[c * kFold + i] = fmaf(s, __uint_as_float(x[c & 1][i]), acc[c * kFold + i]);
        }
      }
      if (!ok) break;
      if (row0 >= o.aEnd) continue;
      if constexpr (SWIGLU) {  // 64 gate columns, then the 64 up columns of the same outputs
        if (live) {            // not on the zeros of rows past the end, whose division takes the slow path
#pragma unroll
          for (int i = 0; i < 64; i++) acc[i] = acc[i] / (1.f + __expf(-acc[i])) * acc[64 + i];
        }
        gemm8::storeCols<64>(
            sw, lane, p.N / 2 - o.tn * (BT / 2), acc,
            [&](int r) -> __nv_bfloat16* { return row0 + r < o.aEnd ? p.C + (size_t)(row0 + r) * p.ldc + (size_t)o.tn * (BT / 2) : nullptr; },
            [&](int g) { return h * 64 + g * 32; });
      } else {
#pragma unroll
        for (int half = 0; half < 2; half++)
          gemm8::storeCols<64>(
              sw, lane, p.N - o.tn * BT, acc + half * 64,
              [&](int r) -> __nv_bfloat16* { return row0 + r < o.aEnd ? p.C + (size_t)(row0 + r) * p.ldc + (size_t)o.tn * BT : nullptr; },
              [&](int g) { return h * 128 + half * 64 + g * 32; });
      }
    }
  }
  tcFenceBefore();
  __syncthreads();
  clusterArrive();  // no arrival may land on a CTA that has left, and no MMA may read the shared memory of one
  clusterWait();
  if (warp == 1) tmemDeallocPair(tmem, kTmemCols);
}

template <bool SWIGLU>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1) gemmFp8PairKernel(const __grid_constant__ Params p) {
  extern __shared__ uint8_t smemRaw[];
  gemmFp8PairCta<false, SWIGLU>(p, smemRaw);
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1) gemmFp8PairGroupedKernel(const __grid_constant__ Params p) {
  extern __shared__ uint8_t smemRaw[];
  gemmFp8PairCta<true, true>(p, smemRaw);
}

}  // namespace gemm8p
}  // namespace b200
