// bf16 GEMM on CTA pairs (tcgen05 cta_group::2) with either operand K-major or MN-major:
//   C[M, N] = A * B^T,  A logical [M, K], B logical [N, K], fp32 accumulation, bf16 out.
// "K-major": the operand is stored [rows, K] row-major (the reduction index is contiguous). "MN-major": it is stored
// [K, rows] row-major (the row index is contiguous), which is how the operands of a backward pass lie in memory:
//   y  = x  w^T      A = x  (K-major)   B = w  (K-major)
//   dx = dy w        A = dy (K-major)   B = w  read as [N_red, K_out]: MN-major
//   dw = dy^T x      A = dy read as [T_red, N]: MN-major   B = x read as [T_red, K]: MN-major
// so no transposed copy of anything is ever made.
//
// Two CTAs of a cluster work on one 256 x BN output tile. Each loads its own 128 rows of A and its own half of the B
// tile (BN / 2 rows) with ordinary TMA tile loads into its own shared memory; the even CTA's elected thread issues one
// 256 x BN x 16 MMA per step that reads both halves and writes 128 accumulator rows into each CTA's tensor memory.
// Against one CTA per tile that halves the shared-memory traffic of B (three stages of 128 reduction steps fit). The byte count of
// both CTAs' loads lands on the even CTA's `full` barrier; the MMA thread's commits arrive on the `empty` barriers of both
// CTAs (one commit addressed to both) and, at the end of a tile, on both `accFull` barriers; the epilogue warps of both CTAs
// arrive on the even CTA's `accEmpty`. Four epilogue warps per CTA drain tensor memory through a swizzled staging buffer
// into 256-byte row segments while the next tile's main loop runs (two accumulators). Every wait is bounded; a CTA that
// gives up still reaches the cluster barriers at the end.
//
// SWIGLU: B holds gate and up rows in turn per tile (BN / 2 gate rows, then the BN / 2 up rows of the same outputs) and the epilogue
// writes silu(gate) * up, BN / 2 columns per tile.
//
// Two forms for the experts of a mixture, `cap` rows reserved per expert of which cnt[e] hold tokens (read on the device, so no
// host round trip), each one launch whose persistent CTA pairs share the tiles of all experts:
//   kRows  C[rows of e] = A[rows of e] * B_e^T over the 256-row blocks that hold tokens.
//   kSum   C_e[M, N] = A[rows of e]^T * B[rows of e] (a weight gradient), reduced over the rows that hold tokens; the rows up to the
//          next multiple of 16 must be zeros in both operands.
// 32 experts, 4096 tokens, top-8, hidden 4096, ffn 1024, forward and backward (seven launches): the SwiGLU form of the gate/up GEMM 0.40 ms, the
// down GEMM and the recomputed gate/up GEMM 0.64, the two rows' gradients 0.62, the two weight gradients 0.67 (64 launches of
// the plain form 1.11). The SwiGLU form for 4096 x 28672 x 4096 0.60 ms (1.00 on one CTA per 128 x 256 tile).
#pragma once

#include "gemm_sm100.cuh"

namespace b200 {
namespace gemm2 {

using gemm::BK;
using gemm::BM;
using gemm::kThreads;

// A stage holds 128 reduction steps (two TMA boxes of 64 per operand): eight MMAs per barrier round trip. With 64 the
// issuing thread spent as long on the wait / commit pair of a stage as the tensor cores on its four MMAs.
constexpr int kStages = 3;
constexpr int kSub = 2;                        // 64-wide reduction slices per stage
constexpr uint32_t kChunkBytes = 64 * BK * 2;  // one MN-major TMA box: 64 reduction rows of 64 elements

template <int BN> struct Cfg {
  static constexpr uint32_t kASub = BM * BK * 2;            // this CTA's 128 rows of A, 64 reduction steps
  static constexpr uint32_t kBSub = (BN / 2) * BK * 2;      // this CTA's half of the B tile, 64 reduction steps
  static constexpr uint32_t kABytes = kSub * kASub;
  static constexpr uint32_t kBBytes = kSub * kBSub;
  static constexpr uint32_t kStageBytes = kABytes + kBBytes;
  static constexpr uint32_t kTmemCols = 2 * BN;
  static constexpr uint32_t kEpiBytesPerWarp = 32 * 128 * 2;
  static constexpr size_t kSmemBytes = (size_t)kStages * kStageBytes + 1024 + 256 + 4 * kEpiBytesPerWarp;
};

enum Mode { kPlain, kRows, kSum };
constexpr int kMaxGroups = 64;

struct Params {
  CUtensorMap mapA;  // K-major: [M, K], box {64, 128}.   MN-major: [K, M], box {64, 64}.   kRows: [groups * cap, K]; kSum: [groups * cap, M]
  CUtensorMap mapB;  // K-major: [N, K], box {64, BN / 2}. MN-major: [K, N], box {64, 64}.  kRows: groups of them in turn; kSum: [groups * cap, N]
  __nv_bfloat16* C;
  int ldc;
  int M, N, K;         // kRows: N, K per group; kSum: M, N per group
  int tilesM, tilesN;  // tiles of 256 x BN (kRows: tilesM unused; kSum: per group)
  const uint32_t* cnt; // rows of every group (may exceed cap)
  int groups, cap;
  int* err;
};

// One tile: first rows of the operands (for an operand stored MN-major its first column) and first reduction steps, 16-step
// slices of the reduction, rows [cRow, cEnd) of C, column block.
struct Tile {
  int aRow, aK, bRow, bK, steps, cRow, cEnd, tn;
};

template <int BN, Mode MODE>
__device__ __forceinline__ Tile tileAt(const Params& p, const int* prefix, int t) {
  Tile o;
  o.aK = o.bK = 0;
  o.steps = (p.K + 15) / 16;
  if constexpr (MODE == kPlain) {
    int tm;
    gemm::bandedCoord(t, p.tilesM, p.tilesN, tm, o.tn);
    o.aRow = o.cRow = tm * 2 * BM;
    o.cEnd = p.M;
    o.bRow = o.tn * BN;
  } else if constexpr (MODE == kRows) {
    const int rb = t / p.tilesN;
    o.tn = t - rb * p.tilesN;
    int g = 0;
    while (prefix[g + 1] <= rb) g++;
    o.aRow = o.cRow = g * p.cap + (rb - prefix[g]) * 2 * BM;
    o.cEnd = g * p.cap + min((int)p.cnt[g], p.cap);
    o.bRow = o.tn * BN;
    o.bK = g;  // the caller turns the group into rows of B
  } else {
    const int per = p.tilesM * p.tilesN, g = t / per;
    int tm;
    gemm::bandedCoord(t - g * per, p.tilesM, p.tilesN, tm, o.tn);
    o.aRow = tm * 2 * BM;
    o.bRow = o.tn * BN;
    o.aK = o.bK = g * p.cap;
    o.steps = (min((int)p.cnt[g], p.cap) + 15) / 16;
    o.cRow = g * p.M + o.aRow;
    o.cEnd = (g + 1) * p.M;
  }
  return o;
}

template <int BN, bool A_MN, bool B_MN, Mode MODE, bool SWIGLU>
__device__ __forceinline__ void gemmPairCta(const Params& p, uint8_t* smemRaw) {
  using C = Cfg<BN>;
  using namespace sm100;
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~(uintptr_t)1023);
  uint8_t* smemA = smem;
  uint8_t* smemB = smem + (size_t)kStages * C::kABytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (size_t)kStages * C::kStageBytes);
  uint64_t* full = bars;                 // used in the even CTA only
  uint64_t* empty = bars + kStages;      // one set per CTA
  uint64_t* accFull = bars + 2 * kStages;   // one set per CTA
  uint64_t* accEmpty = accFull + 2;      // used in the even CTA only
  uint32_t* tmemSlot = reinterpret_cast<uint32_t*>(accEmpty + 2);
  uint8_t* epiStage = reinterpret_cast<uint8_t*>(bars) + 256;

  __shared__ int prefix[MODE == kRows ? kMaxGroups + 1 : 1];  // 256-row blocks with tokens before group g

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t cr = clusterCtaRank();  // 0: issues the MMAs; 1: its partner
  volatile int* err = p.err;

  if constexpr (MODE == kRows) {  // the counts are read side by side, then summed
    for (int g = threadIdx.x; g <= p.groups; g += kThreads) prefix[g] = g == 0 ? 0 : (min((int)p.cnt[g - 1], p.cap) + 2 * BM - 1) / (2 * BM);
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    prefetchTensorMap(&p.mapA);
    prefetchTensorMap(&p.mapB);
    for (int s = 0; s < kStages; s++) {
      mbarInit(&full[s], 1);
      mbarInit(&empty[s], 1);
    }
    for (int b = 0; b < 2; b++) {
      mbarInit(&accFull[b], 1);
      mbarInit(&accEmpty[b], 8);  // four epilogue warps in each CTA of the pair
    }
    fenceBarrierInit();
    if constexpr (MODE == kRows)
      for (int g = 0; g < p.groups; g++) prefix[g + 1] += prefix[g];
  }
  if (warp == 1) {
    tmemAllocPair(tmemSlot, C::kTmemCols);
    tmemRelinquishPair();
  }
  tcFenceBefore();
  __syncthreads();
  clusterArrive();  // the partner's barriers exist before anything arrives on them
  clusterWait();
  tcFenceAfter();
  const uint32_t tmem = *tmemSlot;

  const int numTiles = MODE == kRows ? prefix[p.groups] * p.tilesN : MODE == kSum ? p.groups * p.tilesM * p.tilesN : p.tilesM * p.tilesN;
  constexpr int kStageSteps = kSub * BK / 16;
  const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = pair; t < numTiles && ok; t += npairs) {
        const Tile o = tileAt<BN, MODE>(p, prefix, t);
        const int aRow = o.aRow + (int)cr * BM;
        const int bRow = o.bRow + (int)cr * (BN / 2) + (MODE == kRows && !B_MN ? o.bK * p.N : 0);
        const int bK = MODE == kRows ? (B_MN ? o.bK * p.K : 0) : o.bK;
        const int kIters = (o.steps + kStageSteps - 1) / kStageSteps;
        for (int k = 0; k < kIters; k++) {
          if (!mbarWait(&empty[stage], phase ^ 1, err, gemm::ERR_PRODUCER_EMPTY)) { ok = false; break; }
          const uint32_t fullAddr = mapToCta(smemAddr(&full[stage]), 0);
          if (cr == 0) mbarArriveExpectTx(&full[stage], 2 * C::kStageBytes);  // both CTAs' bytes land here
          uint8_t* sa = smemA + (size_t)stage * C::kABytes;
          uint8_t* sb = smemB + (size_t)stage * C::kBBytes;
#pragma unroll
          for (int h = 0; h < kSub; h++) {
            const int k0 = (k * kSub + h) * BK;  // a slice that starts beyond K reads zeros
            if constexpr (A_MN) {
#pragma unroll
              for (int c = 0; c < BM / 64; c++) tmaLoad2dPair(sa + h * C::kASub + c * kChunkBytes, &p.mapA, aRow + c * 64, o.aK + k0, fullAddr);
            } else {
              tmaLoad2dPair(sa + h * C::kASub, &p.mapA, k0, aRow, fullAddr);
            }
            if constexpr (B_MN) {
#pragma unroll
              for (int c = 0; c < BN / 2 / 64; c++) tmaLoad2dPair(sb + h * C::kBSub + c * kChunkBytes, &p.mapB, bRow + c * 64, bK + k0, fullAddr);
            } else {
              tmaLoad2dPair(sb + h * C::kBSub, &p.mapB, k0, bRow, fullAddr);
            }
          }
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
      }
      if (!ok && cr == 0)
        for (int s = 0; s < kStages; s++) mbarWait(&full[s], 0, err, 0, 2000u);  // let loads in flight land
    }
  } else if (warp == 1) {
    if (lane == 0 && cr == 0) {
      constexpr uint32_t idesc = instrDescMajor(2 * BM, BN, 1 /*bf16*/, A_MN ? 1u : 0u, B_MN ? 1u : 0u);
      int stage = 0;
      uint32_t phase = 0;
      int it = 0;
      bool ok = true;
      for (int t = pair; t < numTiles && ok; t += npairs) {
        const int steps = MODE == kSum ? tileAt<BN, MODE>(p, prefix, t).steps : (p.K + 15) / 16;
        if (MODE == kSum && steps == 0) continue;  // a group without rows: the epilogue writes zeros by itself
        const int kIters = (steps + kStageSteps - 1) / kStageSteps;
        const int b = it & 1;
        const uint32_t accPhase = (it >> 1) & 1;
        it++;
        if (!mbarWait(&accEmpty[b], accPhase ^ 1, err, gemm::ERR_MMA_ACC_EMPTY)) { ok = false; break; }
        tcFenceAfter();
        const uint32_t d = tmem + (uint32_t)b * BN;
        for (int k = 0; k < kIters; k++) {
          if (!mbarWait(&full[stage], phase, err, gemm::ERR_MMA_FULL)) { ok = false; break; }
          tcFenceAfter();
          const uint32_t aAddr = smemAddr(smemA + (size_t)stage * C::kABytes);
          const uint32_t bAddr = smemAddr(smemB + (size_t)stage * C::kBBytes);
#pragma unroll
          for (int h = 0; h < kSub; h++) {
#pragma unroll
            for (int kk = 0; kk < BK / 16; kk++) {
              // 16 reduction steps: 32 bytes along a K-major row, 16 rows of 128 bytes in an MN-major tile
              const uint32_t ah = aAddr + h * C::kASub, bh = bAddr + h * C::kBSub;
              const uint64_t da = A_MN ? smemDescSw128Mn(ah + kk * 2048, kChunkBytes) : smemDescSw128(ah + kk * 32);
              const uint64_t db = B_MN ? smemDescSw128Mn(bh + kk * 2048, kChunkBytes) : smemDescSw128(bh + kk * 32);
              if (MODE != kSum || k * kStageSteps + h * (BK / 16) + kk < steps) mmaF16Pair(d, da, db, idesc, (k | h | kk) != 0);
            }
          }
          mmaCommitBoth(smemAddr(&empty[stage]));  // the stage is free in both CTAs once these MMAs have read it
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
        if (ok) mmaCommitBoth(smemAddr(&accFull[b]));
      }
    }
  } else {
    const int q = warp & 3;
    int it = 0;
    bool ok = true;
    for (int t = pair; t < numTiles && ok; t += npairs) {
      const Tile o = tileAt<BN, MODE>(p, prefix, t);
      const int row0 = o.cRow + (int)cr * BM + q * 32;
      uint8_t* sw = epiStage + (size_t)q * C::kEpiBytesPerWarp;
      constexpr int kOut = SWIGLU ? BN / 2 : BN;  // output columns of a tile
      const auto rowPtr = [&](int r) -> __nv_bfloat16* { return row0 + r < o.cEnd ? p.C + (size_t)(row0 + r) * p.ldc + (size_t)o.tn * kOut : nullptr; };
      const int colLimit = (SWIGLU ? p.N / 2 : p.N) - o.tn * kOut;
      if (MODE == kSum && o.steps == 0) {
        for (int r = 0; r < 32; r++) {  // N is a multiple of 8
          __nv_bfloat16* dst = rowPtr(r);
          if (dst != nullptr && lane * 8 < min(colLimit, kOut)) reinterpret_cast<uint4*>(dst)[lane] = make_uint4(0, 0, 0, 0);
        }
        continue;
      }
      const int b = it & 1;
      const uint32_t accPhase = (it >> 1) & 1;
      it++;
      if (!mbarWait(&accFull[b], accPhase, err, gemm::ERR_EPI_ACC_FULL)) { ok = false; break; }
      tcFenceAfter();
      const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * BN);
      // Rows past the end are neither read back nor run through the activation: they are zeros as a rule, and dividing zeros takes the
      // slow path of the division (2176 x 8192 x 1024, half of the last row tile past the end: 110 us, 53 without).
      const bool live = row0 + lane < o.cEnd;
      if (row0 < o.cEnd) gemm::drainStaged(
          sw, lane, kOut, colLimit,
          [&](int c, uint32_t(&acc)[32]) {
            tmemLoad32(taddr + c * 32, acc);
            if constexpr (SWIGLU) {
              uint32_t up[32];
              tmemLoad32(taddr + BN / 2 + c * 32, up);
              tmemLoadWait();
              if (live) {
#pragma unroll
                for (int i = 0; i < 32; i++) {
                  const float g = __uint_as_float(acc[i]);
                  acc[i] = __float_as_uint(g / (1.f + __expf(-g)) * __uint_as_float(up[i]));
                }
              }
            } else {
              tmemLoadWait();
            }
          },
          rowPtr);
      tcFenceBefore();
      __syncwarp();
      if (lane == 0) mbarArriveCluster(mapToCta(smemAddr(&accEmpty[b]), 0));
    }
  }
  tcFenceBefore();
  __syncthreads();
  clusterArrive();  // no arrival may land on a CTA that has left, and no MMA may read the shared memory of one
  clusterWait();
  if (warp == 1) tmemDeallocPair(tmem, C::kTmemCols);
}

template <int BN, bool A_MN, bool B_MN, bool SWIGLU>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1) gemmPairKernel(const __grid_constant__ Params p) {
  extern __shared__ uint8_t smemRaw[];
  gemmPairCta<BN, A_MN, B_MN, kPlain, SWIGLU>(p, smemRaw);
}

}  // namespace gemm2
namespace ep {

template <bool A_MN, bool B_MN, gemm2::Mode MODE, bool SWIGLU>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(gemm2::kThreads, 1) groupedGemmKernel(const __grid_constant__ gemm2::Params p) {
  extern __shared__ uint8_t smemRaw[];
  gemm2::gemmPairCta<256, A_MN, B_MN, MODE, SWIGLU>(p, smemRaw);
}

}  // namespace ep
}  // namespace b200
