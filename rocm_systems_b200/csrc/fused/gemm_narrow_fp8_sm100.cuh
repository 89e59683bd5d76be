// Block-scaled fp8 (e4m3) GEMM for few rows of activations: the arithmetic of gemm_fp8_sm100.cuh (one fp32 scale per activation row
// and 128 channels, one per 128 x 128 weight block, each 128-deep partial product folded into fp32 registers) in the shape of
// gemm_narrow_sm100.cuh: MMA rows are output features, MMA columns are the TN tokens, K is split over the CTAs of a cluster.
//
// A tile of 128 features is one row of weight blocks, so a partial product has ONE weight scale, and the activation scale belongs to
// the column: the 128 epilogue threads (one feature each) read the products scale(token) * scale(block) of this CTA's part of K
// from shared memory, where they were put before the main loop. Interleaved gate / up weights have 64 + 64 rows per block, so a
// tile also holds both halves of 64 SwiGLU outputs.
//
// Bound by the reads of W as long as a CTA's fold of a block (TN FMAs per thread) is shorter than the load of its 16 KB.
#pragma once

#include <cuda_fp8.h>

#include "gemm_narrow_sm100.cuh"

namespace b200 {
namespace gemmn8 {

using gemmn::BF;
using gemmn::kMaxSplit;
using gemmn::kThreads;
constexpr int BK = 128;            // elements and bytes: one scale block
constexpr int kMaxBlocks = 64;     // blocks of K per CTA: the size of its scale table

template <int TN> struct Cfg {
  static constexpr uint32_t kWBytes = BF * BK;
  static constexpr uint32_t kXBytes = TN * BK;
  static constexpr uint32_t kStageBytes = kWBytes + kXBytes;
  static constexpr int kStages = TN == 16 ? 5 : TN == 32 ? 4 : 3;
  // Partial products in flight in tensor memory. Never more than there are stages: a product that is not folded yet holds its buffer,
  // so the stage barrier it is waited for on cannot complete a second time.
  static constexpr int kAccBufs = TN == 64 ? 2 : 4;
  static_assert(kAccBufs <= kStages, "see above");
  static constexpr uint32_t kTmemCols = kAccBufs * TN;
  static constexpr size_t kSmemBytes = (size_t)kStages * kStageBytes + (size_t)kMaxBlocks * TN * 4 + 1024 + 256;
  static_assert((size_t)TN * BF * 4 <= (size_t)kStages * kStageBytes, "the partial tile reuses the ring");
};

struct Params {
  CUtensorMap mapW;  // [groups * N, K] bytes, box {128, 128}
  CUtensorMap mapX;  // [rows of X, K] bytes, box {128, TN}
  const float* sX;   // scale of row r, block kb: sX[kb * sXBlock + r * sXRow]
  size_t sXBlock, sXRow;
  const float* sW;   // [groups * ceil(N / 128)][kBlocks]
  __nv_bfloat16* C;
  int ldc;
  int M, N, kBlocks;
  gemmn::Group group;
  int* err;
};

// Grid: x = split rank + S * feature tile, y = token tile, z = group; cluster (S, 1, 1).
template <int TN, bool SWIGLU>
__global__ void __launch_bounds__(kThreads, 2) gemmNarrowFp8Kernel(const __grid_constant__ Params p, int S) {
  using C = Cfg<TN>;
  using namespace sm100;
  extern __shared__ uint8_t smemRaw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~(uintptr_t)1023);
  uint8_t* smemW = smem;
  uint8_t* smemX = smem + (size_t)C::kStages * C::kWBytes;
  float* scales = reinterpret_cast<float*>(smem + (size_t)C::kStages * C::kStageBytes);  // [blocks of this CTA][TN]
  uint64_t* bars = reinterpret_cast<uint64_t*>(scales + (size_t)kMaxBlocks * TN);
  uint64_t* full = bars;
  uint64_t* done = bars + C::kStages;           // the MMAs of a stage are complete: stage free AND product ready
  uint64_t* accEmpty = bars + 2 * C::kStages;   // the epilogue warps have folded a product
  uint32_t* tmemSlot = reinterpret_cast<uint32_t*>(accEmpty + C::kAccBufs);
  float* part = reinterpret_cast<float*>(smem);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  volatile int* err = p.err;
  const int split = blockIdx.x % S, tile = blockIdx.x / S;
  const int tok0 = blockIdx.y * TN;
  const int xRow0 = (int)blockIdx.z * p.group.cap + tok0;
  const int rows = p.group.count ? min((int)p.group.count[blockIdx.z], p.group.cap) : p.M;
  if (tok0 >= rows) return;  // the same for the whole cluster
  const int tokens = min(TN, rows - tok0);
  const int kb0 = p.kBlocks * split / S, kb1 = p.kBlocks * (split + 1) / S;

  if (threadIdx.x == 0) {
    prefetchTensorMap(&p.mapW);
    prefetchTensorMap(&p.mapX);
    for (int s = 0; s < C::kStages; s++) {
      mbarInit(&full[s], 1);
      mbarInit(&done[s], 1);
    }
    for (int b = 0; b < C::kAccBufs; b++) mbarInit(&accEmpty[b], 4);
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
      const int wRow = (int)blockIdx.z * p.N + tile * BF;
      // The kernel in front may be the quantiser of X that let this one start early: it has not written W, so the ring is filled
      // with W while it finishes. (Without the launch attribute the wait returns at once.)
      const int ahead = min(C::kStages, kb1 - kb0);
      for (int i = 0; i < ahead; i++) {
        mbarArriveExpectTx(&full[i], C::kStageBytes);
        tmaLoad2d(smemW + (size_t)i * C::kWBytes, &p.mapW, (kb0 + i) * BK, wRow, &full[i]);
      }
      gridDependencyWait();
      for (int i = 0; i < ahead; i++) tmaLoad2d(smemX + (size_t)i * C::kXBytes, &p.mapX, (kb0 + i) * BK, xRow0, &full[i]);
      if (ahead == C::kStages) phase = 1;
      else stage = ahead;
      for (int kb = kb0 + ahead; kb < kb1; kb++) {
        if (!mbarWait(&done[stage], phase ^ 1, err, gemm::ERR_PRODUCER_EMPTY)) { ok = false; break; }
        mbarArriveExpectTx(&full[stage], C::kStageBytes);
        tmaLoad2d(smemW + (size_t)stage * C::kWBytes, &p.mapW, kb * BK, wRow, &full[stage]);
        tmaLoad2d(smemX + (size_t)stage * C::kXBytes, &p.mapX, kb * BK, xRow0, &full[stage]);
        if (++stage == C::kStages) { stage = 0; phase ^= 1; }
      }
      if (!ok)
        for (int s = 0; s < C::kStages; s++) mbarWait(&full[s], 0, err, 0, 2000u);  // let loads in flight land
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = instrDesc(BF, TN, 0 /*e4m3*/);
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = kb0; kb < kb1; kb++) {
        const uint32_t b = (uint32_t)(kb - kb0) % C::kAccBufs, bPhase = ((uint32_t)(kb - kb0) / C::kAccBufs) & 1;
        if (!mbarWait(&accEmpty[b], bPhase ^ 1, err, gemm::ERR_MMA_ACC_EMPTY)) break;
        if (!mbarWait(&full[stage], phase, err, gemm::ERR_MMA_FULL)) break;
        tcFenceAfter();
        const uint32_t wAddr = smemAddr(smemW + (size_t)stage * C::kWBytes);
        const uint32_t xAddr = smemAddr(smemX + (size_t)stage * C::kXBytes);
#pragma unroll
        for (int kk = 0; kk < BK / 32; kk++) mmaF8(tmem + b * TN, smemDescSw128(wAddr + kk * 32), smemDescSw128(xAddr + kk * 32), idesc, kk != 0);
        mmaCommit(&done[stage]);
        if (++stage == C::kStages) { stage = 0; phase ^= 1; }
      }
    }
    __syncwarp();
  } else {
    const int q = warp & 3, et = threadIdx.x - 64;
    {
      gridDependencyWait();
      const float* sW = p.sW + ((size_t)blockIdx.z * ((p.N + BF - 1) / BF) + tile) * p.kBlocks;
      const int nb = kb1 - kb0;
      const bool rowMajor = p.sXBlock == 1;  // neighbouring threads take what lies side by side in the table
      for (int i = et; i < nb * TN; i += 128) {
        const int t = rowMajor ? i / nb : i % TN, kb = rowMajor ? i % nb : i / TN;
        scales[kb * TN + t] = t < tokens ? p.sX[(size_t)(kb0 + kb) * p.sXBlock + (size_t)(xRow0 + t) * p.sXRow] * __ldg(sW + kb0 + kb) : 0.f;
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");
    }
    float acc[TN];
#pragma unroll
    for (int i = 0; i < TN; i++) acc[i] = 0.f;
    int stage = 0;
    uint32_t phase = 0;
    for (int kb = kb0; kb < kb1; kb++) {
      const uint32_t b = (uint32_t)(kb - kb0) % C::kAccBufs;
      if (!mbarWait(&done[stage], phase, err, gemm::ERR_EPI_ACC_FULL)) break;
      if (++stage == C::kStages) { stage = 0; phase ^= 1; }
      tcFenceAfter();
      const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + b * TN;
      const float4* sc = reinterpret_cast<const float4*>(scales + (size_t)(kb - kb0) * TN);
#pragma unroll
      for (int c = 0; c < TN; c += 16) {
        if (c < tokens) {  // columns beyond the last token hold nothing
          uint32_t x[16];
          tmemLoad16(taddr + c, x);
          tmemLoadWait();
#pragma unroll
          for (int i = 0; i < 4; i++) {
            const float4 s = sc[c / 4 + i];
            acc[c + 4 * i] = fmaf(s.x, __uint_as_float(x[4 * i]), acc[c + 4 * i]);
            acc[c + 4 * i + 1] = fmaf(s.y, __uint_as_float(x[4 * i + 1]), acc[c + 4 * i + 1]);
            acc[c + 4 * i + 2] = fmaf(s.z, __uint_as_float(x[4 * i + 2]), acc[c + 4 * i + 2]);
            acc[c + 4 * i + 3] = fmaf(s.w, __uint_as_float(x[4 * i + 3]), acc[c + 4 * i + 3]);
          }
        }
      }
      tcFenceBefore();
      __syncwarp();
      if (lane == 0) mbarArrive(&accEmpty[b]);
    }
    // The last `done` says that every MMA has read its stage: once all four warps have seen it the ring is free for the partial tile.
    asm volatile("bar.sync 1, 128;" ::: "memory");
    float* dst = part + q * 32 + lane;
#pragma unroll
    for (int i = 0; i < TN; i++) dst[i * BF] = acc[i];
    __syncwarp();
  }
  tcFenceBefore();
  if (S > 1) {
    clusterArrive();
    clusterWait();
  } else {
    __syncthreads();
  }
  constexpr int kOut = SWIGLU ? BF / 2 : BF;
  gemmn::sumSplitsAndStore<SWIGLU>(part, S, split, tokens, p.C + (size_t)xRow0 * p.ldc, p.ldc, tile * kOut, SWIGLU ? p.N / 2 : p.N);
  if (S > 1) {
    clusterArrive();  // no CTA leaves while a peer still reads its partial tile
    clusterWait();
  } else {
    __syncthreads();
  }
  if (warp == 1) tmemDealloc(tmem, C::kTmemCols);
}

}  // namespace gemmn8
}  // namespace b200
