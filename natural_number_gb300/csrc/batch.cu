// batch.cu — thousands of products of uneven lengths as a handful of launches.
//
// The host (engine.cpp) sorts a batch's work by what it is: every product is a
// job with a short pipeline of steps — for an NTT job: the first pass of both
// operands, strided passes, the fused last pass (both operands' last levels,
// block products, first inverse levels), the strided inverse passes, the CRT +
// carry scan; transforms of one pass (up to 4096 words) are one step from
// limbs, and the CRT; a short operand makes a schoolbook job of one column-sum
// scan.  A launch takes one kind of step at one tile shape for all jobs that
// have it, a CTA an item (a few consecutive tiles of one job and prime), so
// every kernel is the single product's with its registers, shared memory and
// threads.  Launches of one phase are independent of each other (the host
// forks them in the batch's CUDA graph); phases follow each other in stream
// order.  An unbalanced product may be split: the longer operand (operand 0)
// in pieces, each with its own transform, sharing the shorter operand's; the
// CRT + carry scan adds the pieces' overlapping residues.
//
// One persistent kernel that runs every kind of item from a queue, waiting on
// per-step counters, measured slower: its tile shapes either took 1.2 MB of
// code with spilled registers or 160 bytes of saved registers a thread and
// call, at five CTAs an SM for the largest shape's shared memory (4096 uneven
// products: 26 to 28 ms; FMA-heavy pipe 44 % busy).
#include <cuda_runtime.h>

#include "nn_device.cuh"
#include "nn_internal.h"
#include "scan_tiles.cuh"
#include "six_tiles.cuh"

namespace nn {

namespace {

using namespace six;

// The transform that tile g of a pass over the first operand's pieces
// belongs to, and the tile's index within it.
struct PieceTile {
  u64 piece;
  u32 tile;
};
__device__ __forceinline__ PieceTile piece_tile(const BatchJob& J, u64 g, u32 tiles_per_transform) {
  if (J.pieces == 1) return {0, (u32)g};
  const u64 i = g / tiles_per_transform;
  return {i, (u32)(g - i * tiles_per_transform)};
}

template <int R>
__global__ void __launch_bounds__(col_threads(R), col_blocks(R))
    batch_load_kernel(const BatchJob* __restrict__ jobs, const BatchItem* __restrict__ items, const SixTables t) {
  extern __shared__ __align__(16) u32 sm6[];
  const BatchItem it = items[blockIdx.x];
  const BatchJob& J = jobs[it.job];
  const int s = J.plan.s;
  const u32 per = (u32)((1ull << s) / ((u64)col_width(R) << R));
  for (u32 q = 0; q < it.ntile; ++q) {
    if (q) __syncthreads();  // the previous tile has been read from shared memory
    const u64* in = J.b;
    u64 n = J.nb;
    u32* res = J.res_b;
    u32 tile = it.tile + q;
    if (it.operand == 0) {
      const PieceTile pt = piece_tile(J, tile, per);
      tile = pt.tile;
      in = J.a + pt.piece * J.piece;
      n = min(J.piece, J.na - pt.piece * J.piece);
      res = J.res_a + (pt.piece * kPrimes << s);
    }
    load_tile<R, col_width(R), col_threads(R)>(sm6, in, n, res, s, tile, it.prime, t.tab, t.cap, J.plan.k8);
  }
}

// Strided pass `pass` of the plans, forward of either operand or inverse.
template <int R, bool INV>
__global__ void __launch_bounds__(col_threads(R), col_blocks(R))
    batch_col_kernel(const BatchJob* __restrict__ jobs, const BatchItem* __restrict__ items, const SixTables t, int pass) {
  extern __shared__ __align__(16) u32 sm6[];
  const BatchItem it = items[blockIdx.x];
  const BatchJob& J = jobs[it.job];
  const int s = J.plan.s;
  const u32 per = (u32)((1ull << s) / ((u64)col_width(R) << R));
  for (u32 q = 0; q < it.ntile; ++q) {
    if (q) __syncthreads();
    u32* res = J.res_b;
    u32 tile = it.tile + q;
    if (it.operand == 0) {
      const PieceTile pt = piece_tile(J, tile, per);
      tile = pt.tile;
      res = J.res_a + (pt.piece * kPrimes << s);
    }
    const bool last = INV && pass == 0;
    col_tile<R, col_width(R), col_threads(R), INV>(sm6, res, s, J.plan.lambda0[pass], tile, it.prime,
                                                           t.tab + (INV ? kPrimes * t.cap : 0), t.cap, last,
                                                           J.plan.scale[it.prime], last ? J.plan.k8 : 8);
  }
}

// The contiguous last pass, tile by tile (MODE: six_tiles.cuh).
template <int R, int LGM, int MODE>
__global__ void __launch_bounds__(fused_threads(R, LGM, 4), fused_blocks(R, LGM, 4))
    batch_fused_kernel(const BatchJob* __restrict__ jobs, const BatchItem* __restrict__ items, const SixTables t) {
  extern __shared__ __align__(16) u32 sm6[];
  const BatchItem it = items[blockIdx.x];
  const BatchJob& J = jobs[it.job];
  const int s = J.plan.s;
  const u32 per = (u32)((1ull << s) >> (R + LGM));
  const u32* b = !J.square ? J.res_b : MODE == kProduct ? J.res_a : nullptr;
  for (u32 q = 0; q < it.ntile; ++q) {
    if (q) __syncthreads();
    u32* res = J.res_b;
    u32 tile = it.tile + q;
    if (it.operand == 0) {
      const PieceTile pt = piece_tile(J, tile, per);
      tile = pt.tile;
      res = J.res_a + (pt.piece * kPrimes << s);
    }
    fused_tile<R, LGM, fused_threads(R, LGM, 4), 4, MODE, false>(sm6, res, 0, b, 0, res, s, tile, it.prime, t.tab,
                                                                 t.tab + kPrimes * t.cap, t.cap, J.plan.reduce_in(),
                                                                 false, int2{}, 8);
  }
}

// One-pass transforms from limbs: a's pieces with b (kAll), with b's finished
// words (kReady), or b's forward levels (kForward).
// Columns a thread: a warp or more of busy threads.
constexpr int small_columns(int R) { return R <= 6 ? 1 : R == 7 ? 2 : 4; }
template <int R, int MODE>
__global__ void __launch_bounds__(fused_threads(R, 3, small_columns(R)), fused_blocks(R, 3, small_columns(R)))
    batch_small_kernel(const BatchJob* __restrict__ jobs, const BatchItem* __restrict__ items, const SixTables t) {
  extern __shared__ __align__(16) u32 sm6[];
  constexpr int V = small_columns(R);
  const BatchItem it = items[blockIdx.x];
  const BatchJob& J = jobs[it.job];
  const int s = J.plan.s;
  for (u32 q = 0; q < it.ntile; ++q) {  // a piece an index
    if (q) __syncthreads();
    const u64 piece = it.tile + q;
    const u64* a = MODE == kForward ? J.b : J.a + piece * J.piece;
    const u64 na = MODE == kForward ? J.nb : min(J.piece, J.na - piece * J.piece);
    const void* b = MODE == kReady ? static_cast<const void*>(J.res_b) : J.square ? nullptr : J.b;
    u32* out = MODE == kForward ? J.res_b : J.res_a + (piece * kPrimes << s);
    fused_tile<R, 3, fused_threads(R, 3, V), V, MODE, true>(sm6, a, na, b, J.nb, out, s, 0, it.prime, t.tab,
                                                            t.tab + kPrimes * t.cap, t.cap, false, true,
                                                            J.plan.scale[it.prime], J.plan.k8);
  }
}

// The next item of a carry scan's launch: items start in order, so a tile's
// predecessors are running or done when it looks back.
__device__ __forceinline__ u32 next_item(u32* ticket) {
  __shared__ u32 s_item;
  if (threadIdx.x == 0) s_item = atomicAdd(ticket, 1u);
  __syncthreads();
  return s_item;
}

// A product's carry scan, tile by tile with carry-in 0; what a tile does with a
// carry goes to its flag, and batch_carry_kernel adds the carries after.
template <bool PIECES>
__global__ void __launch_bounds__(kScanThreads, 3)
    batch_crt_kernel(const BatchJob* __restrict__ jobs, const BatchItem* __restrict__ items, u32* flags) {
  const BatchItem it = items[blockIdx.x];
  const BatchJob& J = jobs[it.job];
  const u64 size = J.na + J.nb, L = 1ull << J.plan.s;
  if constexpr (PIECES) {
    const PieceCrtProducer prod{J.res_a, L, J.piece, J.pieces, J.nb, size - 1};
    scan_tile<PieceCrtProducer, kScanRecord>(prod, it.tile, size, J.out, size, nullptr, flags + J.flag_base, nullptr);
  } else {
    const SixCrtProducer prod{J.res_a, L, size - 1};
    scan_tile<SixCrtProducer, kScanRecord>(prod, it.tile, size, J.out, size, nullptr, flags + J.flag_base, nullptr);
  }
}

// One warp a tile of those scans.  The carry into it is the generate bit of the
// nearest earlier tile of its product that does not propagate (0 when all do);
// it turns the tile's leading limbs of all ones into zeros and adds 1 to the
// next, 32 limbs a step.
__global__ void __launch_bounds__(256) batch_carry_kernel(const BatchJob* __restrict__ jobs,
                                                          const BatchItem* __restrict__ items, u32 count,
                                                          const u32* flags) {
  const u32 i = (blockIdx.x * 256 + threadIdx.x) / 32, lane = threadIdx.x & 31;
  if (i >= count) return;  // whole warps leave together
  const BatchItem it = items[i];
  const BatchJob& J = jobs[it.job];
  const u32* f = flags + J.flag_base;
  u32 cin = 0;
  for (u32 before = it.tile; before > 0; before -= min(before, 32u)) {
    const u32 v = lane < before ? f[before - 1 - lane] : 0;
    const u32 ends = __ballot_sync(0xffffffffu, !(v & 2)), generates = __ballot_sync(0xffffffffu, v & 1);
    if (ends) {
      cin = generates >> (__ffs(ends) - 1) & 1;
      break;
    }
  }
  if (!cin) return;
  const u64 size = J.na + J.nb, end = min(size, (u64)(it.tile + 1) * kScanTile);
  for (u64 k = (u64)it.tile * kScanTile; k < end; k += 32) {
    const u64 x = k + lane < end ? J.out[k + lane] : 0;
    const u32 below = __ballot_sync(0xffffffffu, x != ~0ull);
    const u32 first = below ? __ffs(below) - 1 : 32;
    if (lane <= first && k + lane < end) J.out[k + lane] = lane < first ? 0 : x + 1;
    if (first < 32) break;
  }
}

__global__ void __launch_bounds__(kBatchSumThreads, 3)
    batch_columns_kernel(const BatchJob* __restrict__ jobs, const BatchItem* __restrict__ items, u32* ticket,
                         u32* flags, u32* err) {
  __shared__ u64 sums[3 * (kBatchSumTile + kScanE)];
  const BatchItem it = items[next_item(ticket)];
  const BatchJob& J = jobs[it.job];
  const u64 size = J.na + J.nb;
  column_tile_sums<kBatchSumThreads, kBatchSumTile>(sums, ColumnProducer{J.a, J.na, J.b, J.nb}, it.tile);
  __syncthreads();
  typedef SmemSumsProducer<kBatchSumTile> Prod;
  scan_tile<Prod, kScanLookback, kBatchSumThreads, kBatchSumTile>(Prod{sums, (u64)it.tile * kBatchSumTile - kScanE, size}, it.tile, size, J.out,
                                          size, nullptr, flags + J.flag_base, err);
}

struct Launch {
  const BatchSegment& g;
  const BatchJob* jobs;
  const BatchItem* items;
  const SixTables& t;
  cudaStream_t st;

  template <int R>
  cudaError_t strided() const {
    constexpr int smem = col_smem(R), threads = col_threads(R);
    static DeviceOnce once[3];
    const cudaError_t e = g.kind == kBatchLoad  ? allow_smem<smem>(once[0], batch_load_kernel<R>)
                          : g.kind == kBatchCol ? allow_smem<smem>(once[1], batch_col_kernel<R, false>)
                                                : allow_smem<smem>(once[2], batch_col_kernel<R, true>);
    if (e != cudaSuccess) return e;
    if (g.kind == kBatchLoad)
      batch_load_kernel<R><<<g.count, threads, smem, st>>>(jobs, items, t);
    else if (g.kind == kBatchCol)
      batch_col_kernel<R, false><<<g.count, threads, smem, st>>>(jobs, items, t, g.pass);
    else
      batch_col_kernel<R, true><<<g.count, threads, smem, st>>>(jobs, items, t, g.pass);
    return cudaGetLastError();
  }
  template <int R, int LGM, int MODE>
  cudaError_t contiguous_mode() const {
    constexpr int smem = fused_tiles(LGM, MODE) * (int)tile_words32<1 << LGM, true>(R) * 4;
    static DeviceOnce once;
    if (const cudaError_t e = allow_smem<smem>(once, batch_fused_kernel<R, LGM, MODE>); e != cudaSuccess) return e;
    batch_fused_kernel<R, LGM, MODE><<<g.count, fused_threads(R, LGM, 4), smem, st>>>(jobs, items, t);
    return cudaGetLastError();
  }
  template <int R, int LGM>
  cudaError_t contiguous() const {
    if (g.kind == kBatchRow) return contiguous_mode<R, LGM, kForward>();
    switch (g.pass) {
      case kBatchRowsB: return contiguous_mode<R, LGM, kReady>();
      case kBatchRowsAll: return contiguous_mode<R, LGM, kProduct>();
    }
    return contiguous_mode<R, LGM, kAll>();
  }
  template <int R, int MODE>
  cudaError_t small_mode() const {
    constexpr int smem = fused_tiles(3, MODE) * (int)tile_words32<8, true>(R) * 4;
    static_assert(smem <= 48 * 1024);
    batch_small_kernel<R, MODE><<<g.count, fused_threads(R, 3, small_columns(R)), smem, st>>>(jobs, items, t);
    return cudaGetLastError();
  }
  template <int R>
  cudaError_t small() const {
    if (g.kind == kBatchSmallRow) return small_mode<R, kForward>();
    return g.pass == kBatchRowsB ? small_mode<R, kReady>() : small_mode<R, kAll>();
  }

  // Two launches: with the lookback (a ticket before a tile's first load, a wait
  // for the tile before it) 4096 products of 64 to 2^18 limbs, 123484 tiles,
  // took 15.6 ms instead of 14.5.
  template <bool PIECES>
  cudaError_t crt(u32* flags) const {
    batch_crt_kernel<PIECES><<<g.count, kScanThreads, 0, st>>>(jobs, items, flags);
    batch_carry_kernel<<<(g.count + 7) / 8, 256, 0, st>>>(jobs, items, g.count, flags);
    return cudaGetLastError();
  }

  cudaError_t operator()(u32* ticket, u32* flags, u32* err) const {
    switch (g.kind) {
      case kBatchLoad:
      case kBatchCol:
      case kBatchInvCol:
        switch (g.R) {
          case 4: return strided<4>();
          case 5: return strided<5>();
          case 6: return strided<6>();
          case 7: return strided<7>();
          case 8: return strided<8>();
          case 9: return strided<9>();
        }
        break;
      case kBatchRow:
      case kBatchFused:
        switch (g.lgm) {
          case 4: return contiguous<8, 4>();
          case 5: return contiguous<7, 5>();
          case 6: return contiguous<6, 6>();
          case 7: return contiguous<5, 7>();
          case 8: return contiguous<4, 8>();
          case 9: return contiguous<4, 9>();
        }
        switch (g.R) {
          case 5: return contiguous<5, 3>();
          case 6: return contiguous<6, 3>();
          case 7: return contiguous<7, 3>();
          case 8: return contiguous<8, 3>();
          case 9: return contiguous<9, 3>();
        }
        break;
      case kBatchSmallRow:
      case kBatchSmall:
        switch (g.R) {
          case 1: return small<1>();
          case 2: return small<2>();
          case 3: return small<3>();
          case 4: return small<4>();
          case 5: return small<5>();
          case 6: return small<6>();
          case 7: return small<7>();
          case 8: return small<8>();
          case 9: return small<9>();
        }
        break;
      case kBatchCrt:
        return crt<false>(flags);
      case kBatchPieceCrt:
        return crt<true>(flags);
      case kBatchColumns:
        batch_columns_kernel<<<g.count, kBatchSumThreads, 0, st>>>(jobs, items, ticket, flags, err);
        return cudaGetLastError();
    }
    return cudaErrorInvalidValue;
  }
};

}  // namespace

u32 batch_pass_tiles(const SixPlan& pl, int k) {
  const u64 L = 1ull << pl.s;
  u64 tiles = k == pl.n - 1 ? L >> (pl.R[k] + pl.lgm) : L / ((u64)col_width(pl.R[k]) << pl.R[k]);
  if (k > 0) tiles = tiles / 8 * pl.k8;  // past the first pass, the blocks of the first k8 eighths
  return (u32)tiles;
}

cudaError_t batch_launch_segment(const BatchSegment& seg, const BatchJob* jobs, const BatchItem* items, u32* ticket,
                                 u32* flags, u32* err, const SixTables& t, cudaStream_t st) {
  return Launch{seg, jobs, items + seg.first, t, st}(ticket, flags, err);
}

}  // namespace nn
