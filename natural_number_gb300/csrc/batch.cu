// batch.cu — thousands of products of uneven lengths in one persistent launch.
//
// The host (engine.cpp) turns a batch into a work queue: every product is a
// job with a short pipeline of steps — for an NTT job: the strided forward
// passes of both operands, the fused last pass (both operands' last levels,
// block products, first inverse levels), the strided inverse passes, the CRT +
// carry scan; for a short operand (schoolbook job): one column-sum scan — and
// every step is cut into tiles (items).  Transforms of one pass (up to 4096
// words) are a fused item a prime, from limbs, and the CRT.  An unbalanced
// product may be split: the longer operand (operand 0) in pieces, each with
// its own transform, sharing the shorter operand's; the CRT + carry scan adds
// the pieces' overlapping residues.  Items are
// sorted by step, then job, then tile.  A fixed grid of CTAs (all resident)
// pulls items from an atomic head; an item of step k of job j waits until all
// items of step k-1 of job j have completed (a per-(job, step) counter).
// Because every item of step k-1 was dequeued before any item of step k,
// the wait always ends; it is bounded anyway and records an error.  Data that
// other CTAs wrote in the same launch is read around L1 (.cg).
#include <cuda_runtime.h>

#include <algorithm>
#include <array>

#include "nn_device.cuh"
#include "nn_internal.h"
#include "scan_tiles.cuh"
#include "six_tiles.cuh"

namespace nn {

namespace {

constexpr int kWaitLimit = 1 << 24;

__device__ __forceinline__ u32 ld_acquire(const u32* p) {
  u32 v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// The transform that tile g of a pass over the first operand's pieces
// belongs to, and the tile's index within it.
struct PieceTile {
  u64 piece, tile;
};
__device__ __forceinline__ PieceTile piece_tile(const BatchJob& J, u64 g, u64 tiles_per_transform) {
  if (J.pieces == 1) return {0, g};
  const u64 i = g / tiles_per_transform;
  return {i, g - i * tiles_per_transform};
}

using namespace six;

// The multipliers of the CRT by scale, and the twiddle tables.
struct BatchConst {
  SixTables t;
  SixCrt crt[kSixMaxScale + 1];
};

template <int R>
__device__ __forceinline__ void strided(u32* sm, const BatchJob& J, const BatchItem& it, const BatchConst& k, u32* res,
                                        const u64* in, u64 n, u32 tile) {
  constexpr int C = batch_col_width(R);
  const int s = J.plan.s;
  if (it.kind == kItemInv)  // the pieces' residues are added in the CRT: folded
    col_tile<R, C, kBatchThreads, true, true>(sm, res, s, J.plan.lambda0[it.pass], tile, it.prime,
                                              k.t.tab + kPrimes * k.t.cap, k.t.cap);
  else if (it.pass == 0)
    load_tile<R, C, kBatchThreads, true>(sm, in, n, res, s, tile, it.prime, k.t.tab, k.t.cap);
  else
    col_tile<R, C, kBatchThreads, false, true>(sm, res, s, J.plan.lambda0[it.pass], tile, it.prime, k.t.tab, k.t.cap);
}

// A strided pass: forward passes of operand 0 (the pieces of the longer
// operand) or 1 (the shorter), inverse passes of operand 0.
__device__ __forceinline__ void run_pass(u32* sm, const BatchJob& J, const BatchItem& it, const BatchConst& k,
                                         u32 per_transform) {
  const u64 words = (u64)kPrimes << J.plan.s;
  for (u32 q = 0; q < it.ntile; ++q) {
    if (q) __syncthreads();  // the previous tile has been read from shared memory
    PieceTile pt{0, (u64)it.tile + q};
    u32* res = J.res_b;
    const u64* in = J.b;
    u64 n = J.nb;
    if (it.operand == 0) {
      pt = piece_tile(J, pt.tile, per_transform);
      res = J.res_a + pt.piece * words;
      in = J.a + pt.piece * J.piece;
      n = min(J.piece, J.na - pt.piece * J.piece);
    }
    const u32 tile = (u32)pt.tile;
    switch (J.plan.R[it.pass]) {
      case 4: strided<4>(sm, J, it, k, res, in, n, tile); break;
      case 5: strided<5>(sm, J, it, k, res, in, n, tile); break;
      case 6: strided<6>(sm, J, it, k, res, in, n, tile); break;
      case 7: strided<7>(sm, J, it, k, res, in, n, tile); break;
      case 8: strided<8>(sm, J, it, k, res, in, n, tile); break;
      case 9: strided<9>(sm, J, it, k, res, in, n, tile); break;
    }
  }
}

template <int R, int LGM>
__device__ __forceinline__ void fused(u32* sm, const BatchJob& J, const BatchItem& it, const BatchConst& k, u32* res,
                                      u32 tile, int mode) {
  u32* b = J.square ? nullptr : J.res_b;
  fused_tile<R, LGM, kBatchThreads, 4, false, true>(sm, res, 0, b, 0, res, J.plan.s, tile, it.prime, k.t.tab,
                                                 k.t.tab + kPrimes * k.t.cap, k.t.cap, J.plan.reduce_in(), false, mode);
}
template <int R>
__device__ __forceinline__ void small(u32* sm, const BatchJob& J, const BatchItem& it, const BatchConst& k, u32* res,
                                      const u64* a, u64 na) {
  const u64* b = J.square ? nullptr : J.b;
  fused_tile<R, 3, kBatchThreads, 4, true, true>(sm, a, na, b, J.nb, res, J.plan.s, 0, it.prime, k.t.tab,
                                              k.t.tab + kPrimes * k.t.cap, k.t.cap, false, false);
}

// The contiguous last pass, tile by tile; transforms of one pass run it from
// limbs, a piece an index.
__device__ __forceinline__ void run_fused(u32* sm, const BatchJob& J, const BatchItem& it, const BatchConst& k) {
  const SixPlan& pl = J.plan;
  const u64 words = (u64)kPrimes << pl.s;
  const int R = pl.R[pl.n - 1];
  const u32 per = (u32)((1ull << pl.s) >> (R + pl.lgm));
  const int mode = it.kind == kItemRow ? kForward : J.rows ? kProduct : kAll;
  for (u32 q = 0; q < it.ntile; ++q) {
    if (q) __syncthreads();
    if (pl.n == 1) {
      const u64 piece = (u64)it.tile + q;
      u32* res = J.res_a + piece * words;
      const u64* a = J.a + piece * J.piece;
      const u64 na = min(J.piece, J.na - piece * J.piece);
      switch (R) {
        case 1: small<1>(sm, J, it, k, res, a, na); break;
        case 2: small<2>(sm, J, it, k, res, a, na); break;
        case 3: small<3>(sm, J, it, k, res, a, na); break;
        case 4: small<4>(sm, J, it, k, res, a, na); break;
        case 5: small<5>(sm, J, it, k, res, a, na); break;
        case 6: small<6>(sm, J, it, k, res, a, na); break;
        case 7: small<7>(sm, J, it, k, res, a, na); break;
        case 8: small<8>(sm, J, it, k, res, a, na); break;
        case 9: small<9>(sm, J, it, k, res, a, na); break;
      }
      continue;
    }
    const PieceTile pt = it.operand == 0 ? piece_tile(J, (u64)it.tile + q, per) : PieceTile{0, (u64)it.tile + q};
    u32* res = it.operand == 0 ? J.res_a + pt.piece * words : J.res_b;
    const u32 tile = (u32)pt.tile;
    switch (pl.lgm) {
      case 4: fused<8, 4>(sm, J, it, k, res, tile, mode); continue;
      case 5: fused<7, 5>(sm, J, it, k, res, tile, mode); continue;
      case 6: fused<6, 6>(sm, J, it, k, res, tile, mode); continue;
      case 7: fused<5, 7>(sm, J, it, k, res, tile, mode); continue;
      case 8: fused<4, 8>(sm, J, it, k, res, tile, mode); continue;
      case 9: fused<4, 9>(sm, J, it, k, res, tile, mode); continue;
    }
    switch (R) {
      case 5: fused<5, 3>(sm, J, it, k, res, tile, mode); break;
      case 6: fused<6, 3>(sm, J, it, k, res, tile, mode); break;
      case 7: fused<7, 3>(sm, J, it, k, res, tile, mode); break;
      case 8: fused<8, 3>(sm, J, it, k, res, tile, mode); break;
      case 9: fused<9, 3>(sm, J, it, k, res, tile, mode); break;
    }
  }
}

// Six CTAs of 128 threads an SM (80 registers a thread, two padded tiles of
// 4096 words of shared memory).
__global__ void __launch_bounds__(kBatchThreads, 6) batch_kernel(const BatchJob* __restrict__ jobs,
                                                    const BatchItem* __restrict__ items, u32 n_items,
                                                    const u32* __restrict__ need, u32* done, u32* head, u32* flags,
                                                    u32* err, const __grid_constant__ BatchConst k) {
  extern __shared__ __align__(16) u64 sm[];
  u32* const sm32 = reinterpret_cast<u32*>(sm);
  __shared__ u32 s_item;
  // Thread 0 claims the next item while the current one runs, so the queue
  // atomic's latency is hidden.  Items are claimed in queue order and depend
  // only on earlier ones, so the earliest unfinished item is always being
  // worked on: a claimed-but-waiting item never blocks its own dependencies.
  u32 next = 0;
  if (threadIdx.x == 0) next = atomicAdd(head, 1u);
  for (;;) {
    if (threadIdx.x == 0) s_item = next;
    __syncthreads();
    const u32 idx = s_item;
    if (idx >= n_items) break;
    if (threadIdx.x == 0) next = atomicAdd(head, 1u);
    const BatchItem it = items[idx];
    const BatchJob& J = jobs[it.job];
    if (threadIdx.x == 0 && it.step > 0) {
      const u32 c = J.ctr_base + it.step - 1;
      const u32 want = need[c];
      int spins = 0;
      while (ld_acquire(&done[c]) < want) {
        if (++spins > kWaitLimit) {
          atomicExch(err, 2u);
          break;
        }
        __nanosleep(64);
      }
      __threadfence();
    }
    __syncthreads();
    switch (it.kind) {
      case kItemFwd:
      case kItemInv: {
        const u32 R = J.plan.R[it.pass];
        run_pass(sm32, J, it, k, (u32)((1ull << J.plan.s) / ((u64)batch_col_width((int)R) << R)));
        break;
      }
      case kItemRow:
      case kItemFused:
        run_fused(sm32, J, it, k);
        break;
      case kItemCrt: {
        const u64 size = J.na + J.nb, L = 1ull << J.plan.s;
        const SixCrt crt = k.crt[J.plan.s];
        const PieceCrtProducer<true> prod{J.res_a, L, J.piece, J.pieces, J.nb, size - 1, crt};
        scan_tile<PieceCrtProducer<true>, true, kBatchThreads>(prod, it.tile, size, J.out, size, nullptr,
                                                               flags + J.flag_base, err);
        break;
      }
      case kItemColumn: {
        const u64 size = J.na + J.nb;
        column_tile_sums<kBatchThreads, kBatchScanTile>(sm, ColumnProducer{J.a, J.na, J.b, J.nb}, it.tile);
        __syncthreads();
        const SmemSumsProducer<kBatchScanTile> prod{sm, (u64)it.tile * kBatchScanTile - kScanE, size};
        scan_tile<SmemSumsProducer<kBatchScanTile>, true, kBatchThreads>(prod, it.tile, size, J.out, size, nullptr,
                                                                         flags + J.flag_base, err);
        break;
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      atomicAdd(&done[J.ctr_base + it.step], 1u);
    }
  }
}

}  // namespace

u32 batch_pass_tiles(const SixPlan& pl, int k) {
  const u64 L = 1ull << pl.s;
  if (k == pl.n - 1) return (u32)(L >> (pl.R[k] + pl.lgm));
  return (u32)(L / ((u64)batch_col_width(pl.R[k]) << pl.R[k]));
}
size_t batch_pass_smem(const SixPlan& pl, int k, bool square) {
  const int R = pl.R[k];
  if (k == pl.n - 1) {
    const size_t rows = (size_t)1 << R, C = (size_t)1 << pl.lgm;
    return (square ? 4 : 8) * (rows * C + (C < 32 ? (rows + 7) / 8 * C : 0));
  }
  return 4 * (R == 9 ? tile_words32<16>(9) : ((size_t)batch_col_width(R) << R));
}

cudaError_t batch_configure(int* blocks_per_sm, size_t smem) {
  cudaError_t e = cudaFuncSetAttribute(batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, batch_kernel, kBatchThreads, smem);
}

cudaError_t batch_launch(const BatchJob* jobs, const BatchItem* items, u32 n_items, const u32* need, u32* done,
                         u32* head, u32* flags, u32* err, const SixTables& t, int grid, size_t smem, cudaStream_t st) {
  // Recorded into a CUDA graph by the caller, which accounts for the launch
  // at each replay.
  BatchConst k;
  k.t = t;
  static const auto crt = [] {
    std::array<SixCrt, kSixMaxScale + 1> c{};
    for (int s = kSixMinScale; s <= kSixMaxScale; ++s) c[s] = six_crt(s);
    return c;
  }();
  std::copy(crt.begin(), crt.end(), k.crt);
  batch_kernel<<<grid, kBatchThreads, smem, st>>>(jobs, items, n_items, need, done, head, flags, err, k);
  return cudaGetLastError();
}

}  // namespace nn
