// carry.cu — multiword carry propagation on sm_103a: CRT recombination fused
// with a carry scan, plus the same scan driving the schoolbook base case and
// shifted multiword adds.
//
// Each position k contributes a three-word value x_k (< 2^186) at limb k; the
// output is sum_k x_k * B^k, B = 2^64 (asmCRT, asmLinux.asm:1369-1450, does
// this serially with a two-word running carry).  Thread t of a tile owns E
// consecutive positions and forms S_t = sum_e x_{k0+e} B^e = lo_t + H_t B^E
// with a zero carry-in (H_t: two words).  Adding the neighbour's H_{t-1} into
// lo_t leaves an E-limb value u_t plus a one-bit generate g_t; the remaining
// carries are one bit each (propagate p_t = u_t is all ones; g_t and p_t are
// exclusive), resolved by warp ballots inside a tile.
//
// Between tiles the per-call scans take two launches and never wait:
//  1. every tile runs with carry-in 0, writes its limbs and records its
//     one-bit generate and propagate (no tile waits for another);
//  2. each CTA takes the carry into its range of tiles from the nearest tile
//     before it that does not propagate, resolves the carries inside its range
//     with ballots, and adds a tile's carry-in of 1 at its first limb, where
//     it ripples only while limbs wrap to zero.
// The shortest are one cluster, whose CTAs exchange their bits.  No scan leaves
// anything behind for the next one.  The batches' base case and the
// allocation-free entry point take the decoupled lookback instead (scan_tile
// with kScanLookback: one launch, each tile's carry-in from its predecessors'
// status words, cleared before the launch), whose waits are bounded and record
// an error instead of hanging.
#include <cuda_runtime.h>

#include <algorithm>
#include <functional>

#include "nn_device.cuh"
#include "nn_internal.h"
#include "scan_tiles.cuh"

namespace nn {

NN_DEFINE_PRIME_UPLOADER(upload_primes_carry)

namespace {

// Step 1: tile tile_base + blockIdx.x with carry-in 0; flags[tile] receives
// its generate (bit 0) and propagate (bit 1) bits.
template <class Prod, int NT>
__global__ void __launch_bounds__(NT, 768 / NT) scan_kernel(Prod prod, u64 total, u64* out, u64 out_limit, u64* side,
                                                            u32* flags, u64 tile_base) {
  grid_begin();
  scan_tile<Prod, kScanRecord, NT>(prod, tile_base + blockIdx.x, total, out, out_limit, side, flags, nullptr);
}

// Step 2: 32 tiles a CTA.  The carry into the range is the generate bit of the
// nearest earlier tile that does not propagate (0 when all do): the CTA looks
// 256 tiles further back at a time, for random limbs once.  Earlier ranges of
// the same scan are complete (stream order).  One ballot gives every tile of
// the range its carry-in: lane t of warp 0 adds tile t's at its first limb.
// Where that limb wraps to zero, a warp carries on, 32 limbs a step (a product
// next to a power of 2^64, as a reciprocal's with its operand, starts tiles
// with up to 2047 limbs of all ones: one lane's walk took 14 us a launch, 8 so);
// a tile that propagates holds ones only and becomes zeros, by the whole CTA (a
// difference of nearly equal operands has long runs of such tiles).
constexpr int kFixTiles = 32;
template <u64 TILE>
__global__ void __launch_bounds__(256) carry_fix_kernel(const u32* flags, u64 t0, u64 t1, u64 total, u64* out,
                                                        u64 out_limit, u64* side) {
  grid_begin();
  __shared__ u32 s_first, s_cin, s_ones, s_wrapped;
  const u64 c0 = t0 + (u64)blockIdx.x * kFixTiles;
  const int tid = threadIdx.x;
  u32 cin = 0;
  for (u64 back = c0; back > 0;) {  // the same for every thread
    const u32 f = (u64)tid < back ? flags[back - 1 - tid] : 0;  // before tile 0: a kill
    __syncthreads();
    if (tid == 0) s_first = 256;
    __syncthreads();
    if (!((f >> 1) & 1)) atomicMin(&s_first, (u32)tid);
    __syncthreads();
    const u32 first = s_first;
    if (first < 256) {
      if ((u32)tid == first) s_cin = f & 1;
      __syncthreads();
      cin = s_cin;
      break;
    }
    back = back > 256 ? back - 256 : 0;
  }
  auto limb = [&](u64 k) { return k < out_limit ? out + k : side + (k - out_limit); };
  if (tid < 32) {
    const u64 t = c0 + tid;
    const u32 f = t < t1 ? flags[t] : 0;
    const u32 G = __ballot_sync(0xffffffffu, f & 1), GP = __ballot_sync(0xffffffffu, f & 3);
    const u32 in = (u32)((u64)G + GP + cin) ^ G ^ GP;  // the carry into each lane's tile
    const u32 ones = in & GP & ~G;
    const bool add = t < t1 && (((in & ~ones) >> tid) & 1);
    const u32 wrapped = __ballot_sync(0xffffffffu, add && ++*limb(t * TILE) == 0);
    if (tid == 0) {
      s_ones = ones;
      s_wrapped = wrapped;
    }
  }
  __syncthreads();
  const u32 lane = tid & 31;
  for (u32 left = s_wrapped, i = 0; left; left &= left - 1, ++i) {  // a warp a tile
    if (i % 8 != (u32)tid / 32) continue;
    const u64 t = c0 + __ffs(left) - 1, end = min((t + 1) * TILE, total);
    for (u64 k = t * TILE + 1; k < end; k += 32) {
      const u64 x = k + lane < end ? *limb(k + lane) : 0;
      const u32 below = __ballot_sync(0xffffffffu, x != ~0ull);
      const u32 first = below ? __ffs(below) - 1 : 32;
      if (lane <= first && k + lane < end) *limb(k + lane) = lane < first ? 0 : x + 1;
      if (first < 32) break;
    }
  }
  for (u32 ones = s_ones; ones; ones &= ones - 1) {
    const u64 t = c0 + __ffs(ones) - 1, end = min((t + 1) * TILE, total);
    for (u64 k = t * TILE + tid; k < end; k += 256) *limb(k) = 0;
  }
}

// Adds side[0] + side[1]*B into out[0..L) and wraps the final carry around to
// limb 0 (ntt_info.h:238-242): the result is the product mod B^L - 1.
__global__ void __launch_bounds__(1024) wrap_fix_kernel(u64* out, u64 L, const u64* side) {
  grid_begin();
  __shared__ int s_carry;
  __shared__ unsigned long long s_first;
  const int tid = threadIdx.x;
  if (tid == 0) {
    const u64 c0 = side[0], c1 = side[1];
    const u64 v0 = out[0] + c0;
    const u64 cy = v0 < c0;
    u64 t = out[1] + c1;
    u64 cy2 = t < c1;
    const u64 v1 = t + cy;
    cy2 += v1 < cy;
    out[0] = v0;
    out[1] = v1;
    s_carry = (int)cy2;
    s_first = ~0ull;
  }
  __syncthreads();
  if (!s_carry) return;
  for (u64 base = 2; base < L; base += blockDim.x) {
    const u64 i = base + tid;
    const bool stop = i < L && out[i] != ~0ull;
    if (stop) atomicMin(&s_first, (unsigned long long)i);
    __syncthreads();
    const u64 first = s_first;
    if (first != ~0ull) {
      if (i < first && i < L) out[i] = 0;
      __syncthreads();
      if (tid == 0) out[first] += 1;
      return;
    }
    if (i < L) out[i] = 0;
    __syncthreads();
  }
  if (tid == 0) {  // carry left limb L-1: end-around into limb 0
    for (u64 i = 0; i < L; ++i)
      if (++out[i] != 0) break;
  }
}

// out[0..n] = in[0..n) << cl and out[0..n) = in[0..n) >> cl, 1 <= cl <= 63
// (asmShl / asmShr, asm.h:31-33); out does not overlap in.
__global__ void shl_bits_kernel(u64* out, const u64* in, u64 n, unsigned cl) {
  grid_begin();
  for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i <= n; i += (u64)gridDim.x * blockDim.x)
    out[i] = (i < n ? in[i] << cl : 0) | (i > 0 ? in[i - 1] >> (64 - cl) : 0);
}
__global__ void shr_bits_kernel(u64* out, const u64* in, u64 n, unsigned cl) {
  grid_begin();
  for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x)
    out[i] = (in[i] >> cl) | (i + 1 < n ? in[i + 1] << (64 - cl) : 0);
}

// The lookback's bounded wait on a status word that nothing sets: after
// `limit` polls it gives up and records the error, as a scan tile does.
__global__ void wait_probe_kernel(const u32* flag, u32* err, int limit) {
  if (threadIdx.x == 0 && wait_flag(flag, limit) == 0) atomicExch(err, 1u);
}

// Scans of up to 2^17 positions run in tiles of 512, so that more SMs share
// them (a thread's eight values are a serial chain): products of 2^16
// coefficients 18.9 us, 19.3 in tiles of 2048, of 2^17 24.4 and 24.7, of 2^18
// 29.9 and 29.3.  Up to eight such tiles are one cluster (kScanCluster): 9.6 us
// for 1500 x 1201 limbs, 10.2 in two launches; sixteen, 15.9 and 15.4 us.  In
// one launch with the lookback, 2^16 coefficients took 21.0 us, 2^18 33.3, 2^21
// 178 instead of 167.5 (sums alike: a division of 2800007 by 1400003 limbs 2.50
// ms with its sums so, 2.40 without).
constexpr int kScanSmall = 64;  // threads
constexpr u64 kClusterTiles = 8, kSmallTiles = 256;
template <class Prod>
__global__ void __launch_bounds__(kScanSmall) scan_cluster_kernel(Prod prod, u64 total, u64* out, u64 out_limit,
                                                                  u64* side) {
  grid_begin();
  scan_tile<Prod, kScanCluster, kScanSmall>(prod, blockIdx.x, total, out, out_limit, side, nullptr, nullptr);
  cluster_sync();
}

// Base-case products of up to sixteen tiles of 64 positions: one cluster.  The
// shorter operand and the window of the longer one that a tile needs come
// into shared memory, padded with zeros; sixteen lanes share four columns,
// each a run of the longer operand's limbs (of odd length, so that the lanes
// hit different banks): a step reads one limb of either operand and feeds
// four independent sums.  383 x 383 limbs: 14.4 us with one term a step and
// the status words of the lookback in global memory.
constexpr int kSchoolClusterCtas = 16;
constexpr u64 kSchoolClusterTile = 64, kSchoolShorter = 384;
__global__ void __launch_bounds__(256) school_cluster_kernel(ColumnProducer prod, u64 total, u64* out) {
  grid_begin();
  constexpr u64 TILE = kSchoolClusterTile;
  constexpr int kLanes = 16;
  __shared__ u64 sums[3 * (TILE + kScanE)];
  __shared__ u64 window[TILE + kSchoolShorter], shorter[kSchoolShorter + 8];
  const int tid = threadIdx.x, nb = (int)prod.nb;
  const long long k0 = (long long)blockIdx.x * TILE, a0 = max(0ll, k0 - nb + 1);
  const long long end = min((long long)prod.na, k0 + (long long)TILE);
  for (long long i = a0 + tid; i < end; i += 256) window[i - a0] = prod.a[i];
  for (int i = tid; i < nb + 8; i += 256) shorter[i] = i >= 4 && i < nb + 4 ? prod.b[i - 4] : 0;
  __syncthreads();
  const int g = tid / kLanes, lane = tid % kLanes;
  const long long k = k0 + 4 * g, lo = max(0ll, k - nb + 1), hi = min((long long)prod.na - 1, k + 3);
  const int len = hi >= lo ? (int)(hi - lo + 1) : 0, run = ((len + kLanes - 1) / kLanes) | 1;
  const int from = min(lane * run, len), to = min(from + run, len);
  W3 acc[4] = {};
  const u64* wa = window + (lo - a0);
  const u64* sb = shorter + 4 + (k - lo);  // term t: a[lo + t] with b[k + q - lo - t], q < 4
  u64 b0 = 0, b1 = 0, b2 = 0, b3 = 0;
  if (from < to) {
    b0 = sb[-from];
    b1 = sb[1 - from];
    b2 = sb[2 - from];
    b3 = sb[3 - from];
  }
  for (int t = from; t < to; ++t) {
    const u64 x = wa[t];
    mac(acc[0], x, b0);
    mac(acc[1], x, b1);
    mac(acc[2], x, b2);
    mac(acc[3], x, b3);
    b3 = b2;
    b2 = b1;
    b1 = b0;
    b0 = sb[-t - 1];
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
#pragma unroll
    for (int d = kLanes / 2; d >= 1; d >>= 1) {
      const W3 o{__shfl_down_sync(0xffffffffu, acc[q].w0, d, kLanes), __shfl_down_sync(0xffffffffu, acc[q].w1, d, kLanes),
                 __shfl_down_sync(0xffffffffu, acc[q].w2, d, kLanes)};
      acc[q] = add_w3(acc[q], o);
    }
    if (lane == 0) {
      const u64 i = kScanE + 4 * g + q;
      sums[i] = acc[q].w0;
      sums[TILE + kScanE + i] = acc[q].w1;
      sums[2 * (TILE + kScanE) + i] = acc[q].w2;
    }
  }
  __syncthreads();
  typedef SmemSumsProducer<TILE> Sums;
  scan_tile<Sums, kScanCluster, 256, TILE>(Sums{sums, (u64)k0 - kScanE, total}, blockIdx.x, total, out, total, nullptr,
                                           nullptr, nullptr);
  cluster_sync();
}

// Longer base-case products: each CTA forms its tile's column sums in shared
// memory, eight lanes a position, and runs the scan's first step on them.
// A tile forms the sums of the eight positions before it too, so that its CTA's
// 32 groups of lanes have no part of a round idle at 56 and 248 positions (64 and
// 256: three rounds for 72, nine for 264; 4000 x 4000 limbs 77 us, 60 so).  Small
// tiles spread a short product over the GPU: the column sums are the work.  Of a
// long operand times a short one, up to kSchoolFew limbs beyond kSchoolLong, a
// thread forms the sums of eight positions by itself (run_scan).  Measured, us,
// tiles of 56 / 248 positions / run_scan: 8000 x 383 limbs 14 / 26 / 269, 40000 x
// 383 26 / 38 / 271, 65000 x 383 39 / 39 / 271, 131072 x 1 19 / 15 / 15, x 31 24 /
// 21 / 28, 196000 x 1 - / 20 / 15, 262144 x 31 - / 33 / 28, x 40 - / 28 / 34, x 383
// - / 115 / 272, 2^20 x 31 - / 110 / 81, x 40 - / 94 / 101, x 383 - / 433 / 890.
// run_scan takes an eighth of the tiles' words, too: what is captured keeps to it
// where more would have to be allocated.
constexpr u64 kSchoolTile = 56, kSchoolWideTile = 248;
constexpr u64 kSchoolShort = kSchoolTile << 10, kSchoolLong = 3 << 16, kSchoolFew = 39;
template <u64 TILE>
__global__ void __launch_bounds__(256) school_kernel(ColumnProducer prod, u64 total, u64* out, u32* flags) {
  grid_begin();
  __shared__ u64 sums[3 * (TILE + kScanE)];
  const u64 tile = blockIdx.x;
  column_tile_sums<256, TILE>(sums, prod, tile);
  __syncthreads();
  typedef SmemSumsProducer<TILE> Sums;
  scan_tile<Sums, kScanRecord, 256, TILE>(Sums{sums, tile * TILE - kScanE, total}, tile, total, out, total, nullptr,
                                          flags, nullptr);
}

// One warp a job: lane i adds limb base + i of x and y; the block's carries
// are those of the integer sum G + (G | P) + carry-in over the lanes' generate
// and propagate bits (the same identity as the scan's warp step).  A
// difference adds the complement of y with a carry-in of 1.
__global__ void __launch_bounds__(256) add_batch_kernel(const AddJob* __restrict__ jobs, u64 m) {
  grid_begin();
  const u64 j = ((u64)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const u32 lane = threadIdx.x & 31;
  if (j >= m) return;  // whole warps leave together
  const AddJob J = jobs[j];
  const u64 flip = J.sub ? ~0ull : 0;
  u32 carry = J.sub ? 1 : 0;
  // four 32-limb steps' loads issued together, then their carries in order
  constexpr int kSteps = 4;
  for (u64 base = 0; base < J.nout; base += 32 * kSteps) {
    u64 a[kSteps], b[kSteps];
#pragma unroll
    for (int q = 0; q < kSteps; ++q) {
      const u64 k = base + 32 * q + lane;
      a[q] = k < J.nx ? J.x[k] : 0;
      b[q] = (k < J.ny ? J.y[k] : 0) ^ flip;
    }
#pragma unroll
    for (int q = 0; q < kSteps; ++q) {
      if (base + 32 * q >= J.nout) break;  // the same for every lane
      const u64 k = base + 32 * q + lane;
      const u64 sum = a[q] + b[q];
      const u32 G = __ballot_sync(0xffffffffu, sum < a[q]),
                GP = __ballot_sync(0xffffffffu, sum < a[q] || sum == ~0ull);
      const u64 t = (u64)G + GP + carry;
      const u32 cin = (((u32)t ^ G ^ GP) >> lane) & 1;
      if (k < J.nout) J.out[k] = sum + cin;
      carry = (u32)(t >> 32);
    }
  }
}
// The same with one CTA a job, 1024 limbs a step: the ballots of each 32 limbs
// give what that chunk does with a carry, and the 32 chunks' carries come from
// ballots over those.
__global__ void __launch_bounds__(256) add_batch_long_kernel(const AddJob* __restrict__ jobs) {
  grid_begin();
  constexpr int kSteps = 4;
  __shared__ u32 s_g[2][32], s_gp[2][32];  // by chunk; two sets, so that one barrier a step does
  const AddJob J = jobs[blockIdx.x];
  const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const u64 flip = J.sub ? ~0ull : 0;
  u32 carry = J.sub ? 1 : 0, set = 0;
  for (u64 base = 0; base < J.nout; base += 256 * kSteps, set ^= 1) {
    u64 sum[kSteps];
    u32 G[kSteps], GP[kSteps];
    u64 a[kSteps], b[kSteps];
#pragma unroll
    for (int q = 0; q < kSteps; ++q) {
      const u64 k = base + 256 * q + threadIdx.x;
      a[q] = k < J.nx ? J.x[k] : 0;
      b[q] = (k < J.ny ? J.y[k] : 0) ^ flip;
    }
#pragma unroll
    for (int q = 0; q < kSteps; ++q) {
      sum[q] = a[q] + b[q];
      G[q] = __ballot_sync(0xffffffffu, sum[q] < a[q]);
      GP[q] = __ballot_sync(0xffffffffu, sum[q] < a[q] || sum[q] == ~0ull);
      if (lane == 0) {
        s_g[set][8 * q + warp] = (u32)(((u64)G[q] + GP[q]) >> 32);
        s_gp[set][8 * q + warp] = (u32)(((u64)G[q] + GP[q] + 1) >> 32);
      }
    }
    __syncthreads();
    const u32 CG = __ballot_sync(0xffffffffu, s_g[set][lane]), CGP = __ballot_sync(0xffffffffu, s_gp[set][lane]);
    const u64 t = (u64)CG + CGP + carry;
    const u32 chunk_in = (u32)t ^ CG ^ CGP;
#pragma unroll
    for (int q = 0; q < kSteps; ++q) {
      const u64 k = base + 256 * q + threadIdx.x;
      const u32 in = (u32)((u64)G[q] + GP[q] + (chunk_in >> (8 * q + warp) & 1)) ^ G[q] ^ GP[q];
      if (k < J.nout) J.out[k] = sum[q] + (in >> lane & 1);
    }
    carry = (u32)(t >> 32);
  }
}

// Step 2 over tiles [t0, t1) of TILE positions.
template <u64 TILE>
cudaError_t carry_fix(u64 t0, u64 t1, u64 total, u64* out, u64 out_limit, Scan& sc, cudaStream_t st) {
  launch_begin("scan_carry_fix", st);
  const cudaError_t e = launch_next(carry_fix_kernel<TILE>, (unsigned)((t1 - t0 + kFixTiles - 1) / kFixTiles), 256, 0, 0,
                                    st, sc.flags, t0, t1, total, out, out_limit, sc.side);
  launch_end(st);
  return e;
}

// Tiles [tile_begin, tile_end) of the scan (all of them by default).  The
// ranges of one scan go in order on one stream (each range's carry-in comes
// from the words of the tiles before it).
template <class Prod>
cudaError_t run_scan(const Prod& prod, u64 total, u64* out, u64 out_limit, Scan& sc, cudaStream_t st,
                     const char* name, u64 tile_begin = 0, u64 tile_end = ~0ull) {
  const u64 tiles = scan_tiles(total);
  tile_end = std::min(tile_end, tiles);
  cudaError_t e = scan_reserve(sc, tiles);
  if (e != cudaSuccess || tile_end <= tile_begin) return e;
  // the short ones, whole: column sums come here only beyond them (school_mul)
  if constexpr (Prod::kBulk) {
    const bool whole = tile_begin == 0 && tile_end == tiles;
    constexpr u64 kSmallTile = kScanSmall * kScanE;
    const u64 small = (total + kSmallTile - 1) / kSmallTile;
    if (whole && small <= kClusterTiles) {
      launch_begin(name, st);
      e = launch_next(scan_cluster_kernel<Prod>, (unsigned)small, kScanSmall, 0, (unsigned)small, st, prod, total, out,
                      out_limit, sc.side);
      launch_end(st);
      return e;
    }
    if (whole && small <= kSmallTiles) {
      launch_begin(name, st);
      e = launch_next(scan_kernel<Prod, kScanSmall>, (unsigned)small, kScanSmall, 0, 0, st, prod, total, out, out_limit,
                      sc.side, sc.flags, 0);
      launch_end(st);
      return e == cudaSuccess ? carry_fix<kSmallTile>(0, small, total, out, out_limit, sc, st) : e;
    }
  }
  launch_begin(name, st);
  e = launch_next(scan_kernel<Prod, kScanThreads>, (unsigned)(tile_end - tile_begin), kScanThreads, 0, 0, st, prod, total,
                  out, out_limit, sc.side, sc.flags, tile_begin);
  launch_end(st);
  return e == cudaSuccess ? carry_fix<kScanTile>(tile_begin, tile_end, total, out, out_limit, sc, st) : e;
}

template <u64 TILE>
cudaError_t launch_school(const ColumnProducer& prod, u64 total, u64* out, Scan& sc, cudaStream_t st) {
  const u64 tiles = (total + TILE - 1) / TILE;
  cudaError_t e = scan_reserve(sc, tiles);
  if (e != cudaSuccess) return e;
  launch_begin("school_tiles", st);
  e = launch_next(school_kernel<TILE>, (unsigned)tiles, 256, 0, 0, st, prod, total, out, sc.flags);
  launch_end(st);
  return e == cudaSuccess ? carry_fix<TILE>(0, tiles, total, out, total, sc, st) : e;
}

}  // namespace

u64 scan_tiles(u64 positions) { return positions ? (positions + kScanTile - 1) / kScanTile : 1; }

// Carry bits for that many tiles.  A replaced buffer stays until the context
// goes: a captured graph, or work on another stream, may still use it; the
// replaced ones together are smaller than the live one.
cudaError_t scan_reserve(Scan& sc, u64 tiles) {
  if (!sc.err) {
    u32* words = nullptr;
    cudaError_t e = cudaMalloc((void**)&words, 2 * sizeof(u32) + 4 * sizeof(u64));
    if (e != cudaSuccess) return e;
    e = cudaMemset(words, 0, 2 * sizeof(u32) + 4 * sizeof(u64));
    // the context's streams do not wait for the legacy one
    if (e == cudaSuccess) e = cudaStreamSynchronize(cudaStreamLegacy);
    if (e != cudaSuccess) {
      cudaFree(words);
      return e;
    }
    sc.err = words;
    sc.probe = words + 1;
    sc.side = reinterpret_cast<u64*>(words + 2);
  }
  if (sc.max_tiles >= tiles) return cudaSuccess;
  u64 cap = sc.max_tiles ? sc.max_tiles : 1024;
  while (cap < tiles) cap *= 2;
  u32* flags = nullptr;
  const cudaError_t e = cudaMalloc((void**)&flags, cap * sizeof(u32));
  if (e != cudaSuccess) return e;
  if (sc.flags) sc.replaced.push_back(sc.flags);
  sc.flags = flags;
  sc.max_tiles = cap;
  sc.held_tiles += cap;
  return cudaSuccess;
}

void scan_free(Scan& sc) {
  for (u32* p : sc.replaced) cudaFree(p);
  if (sc.flags) cudaFree(sc.flags);
  if (sc.err) cudaFree(sc.err);
  sc = Scan{};
}

cudaError_t ntt_save(const u64* res, int s, u64* out, u64 size, Scan& sc, u64* written, cudaStream_t st) {
  const u64 L = 1ull << s;
  cudaError_t e = scan_reserve(sc, 1);
  if (e != cudaSuccess) return e;
  if (size - 1 > L) {  // wrap mode
    e = run_scan(CrtProducer{res, L, L}, L + 2, out, L, sc, st, "crt_carry_scan");
    if (e != cudaSuccess) return e;
    launch_begin("wrap_fix", st);
    e = launch_next(wrap_fix_kernel, 1, 1024, 0, 0, st, out, L, sc.side);
    launch_end(st);
    *written = L;
    return e;
  }
  *written = size;
  return run_scan(CrtProducer{res, L, size - 1}, size, out, size, sc, st, "crt_carry_scan");
}

namespace {
// Coefficient k of the six-prime residues modulo each 62-bit prime: its three
// words by Horner's rule, b[i] = 2^64 mod p_i with its Shoup companion.
struct TwoTo64 {
  u64 w[3], s[3];
};
// HALVES: out is res itself; a word's halves go where two of its coefficient's
// residues were.
template <bool HALVES>
__global__ void __launch_bounds__(256) six_to_three_kernel(const u32* res, u64 L, u64* out, const TwoTo64 b) {
  grid_begin();
  const u64 k = (u64)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= L) return;
  const W3 v = SixCrtProducer{res, L, L}(k);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const u64 p = g_primes.p[i], m = g_primes.m64[i];
    const u32 ch = g_primes.c_hi[i];
    u64 r = limb_mod(v.w2, m, p, ch);
    r = reduce2p(shoup_mul(r, b.w[i], b.s[i], p, ch) + limb_mod(v.w1, m, p, ch), p);
    r = reduce2p(shoup_mul(r, b.w[i], b.s[i], p, ch) + limb_mod(v.w0, m, p, ch), p);
    if (HALVES) {
      u32* half = reinterpret_cast<u32*>(out) + 2 * i * L + k;
      half[0] = (u32)r;
      half[L] = (u32)(r >> 32);
    } else {
      out[i * L + k] = r;
    }
  }
}
// One of the two steps that bring the halves together, a plane of 2^bits of them
// (all low ones, then all high ones) a blockIdx.y: half j belongs at j rotated
// left by one bit, which is the reversal of its bits and then that of all but the
// lowest.  Either is its own inverse, so it goes by swaps, in place.
__global__ void __launch_bounds__(256) swap_halves_kernel(u32* x, int bits, bool all) {
  grid_begin();
  const u32 j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >> bits) return;
  const u32 q = all ? __brev(j) >> (32 - bits) : (j & 1) | (__brev(j >> 1) >> (33 - bits)) << 1;
  if (j >= q) return;
  x += (u64)blockIdx.y << bits;
  const u32 t = x[j];
  x[j] = x[q];
  x[q] = t;
}
}  // namespace

cudaError_t six_to_three(const u32* res, int s, u64* out, cudaStream_t st) {
  u64 p[3];
  primes_host(p);
  TwoTo64 b;
  for (int i = 0; i < 3; ++i) {
    b.w[i] = (u64)(((unsigned __int128)1 << 64) % p[i]);
    b.s[i] = (u64)(((unsigned __int128)b.w[i] << 64) / p[i]) + 1;
  }
  const u64 L = 1ull << s;
  const bool in_place = static_cast<const void*>(res) == out;
  launch_begin("six_to_three", st);
  cudaError_t e = launch_next(in_place ? six_to_three_kernel<true> : six_to_three_kernel<false>,
                              (unsigned)((L + 255) / 256), 256, 0, 0, st, res, L, out, b);
  launch_end(st);
  for (int step = 0; in_place && step < 2 && e == cudaSuccess; ++step) {
    launch_begin("swap_halves", st);
    e = launch_next(swap_halves_kernel, dim3((unsigned)((2 * L + 255) / 256), 3), 256, 0, 0, st,
                    reinterpret_cast<u32*>(out), s + 1, step == 0);
    launch_end(st);
  }
  return e;
}

cudaError_t six_save_words(const u32* res, int s, u64* out, u64 size, Scan& sc, u64* written, cudaStream_t st) {
  const u64 L = 1ull << s;
  cudaError_t e = scan_reserve(sc, 1);
  if (e != cudaSuccess) return e;
  if (size - 1 <= L) {
    *written = size;
    return run_scan(SixCrtProducer{res, L, size - 1}, size, out, size, sc, st, "six_crt_scan");
  }
  e = run_scan(SixCrtProducer{res, L, L}, L + 2, out, L, sc, st, "six_crt_scan");
  if (e != cudaSuccess) return e;
  launch_begin("wrap_fix", st);
  e = launch_next(wrap_fix_kernel, 1, 1024, 0, 0, st, out, L, sc.side);
  launch_end(st);
  *written = L;
  return e;
}

cudaError_t six_save(const SixOperands& op, const SixPlan& pl, u64* out, Scan& sc, cudaStream_t st, int chunks,
                     const std::function<cudaError_t(u64, u64)>& done) {
  const u64 L = 1ull << pl.s, nb = op.b ? op.nb : op.na, size = op.na + nb;
  const u64 tiles = scan_tiles(size);
  cudaError_t e = scan_reserve(sc, tiles);
  for (int k = 0; k < chunks && e == cudaSuccess; ++k) {
    const u64 t0 = tiles * k / chunks, t1 = tiles * (k + 1) / chunks;
    if (t1 == t0) continue;
    if (op.pieces == 1)
      e = run_scan(SixCrtProducer{op.ra, L, size - 1}, size, out, size, sc, st, "six_crt_scan", t0, t1);
    else
      e = run_scan(PieceCrtProducer{op.ra, L, op.piece, op.pieces, nb, size - 1}, size, out, size, sc, st,
                   "six_crt_scan", t0, t1);
    if (e == cudaSuccess && done) e = done(t0 * kScanTile, std::min(size, t1 * kScanTile));
  }
  return e;
}

// The decimal split's seven launches for 200003 limbs (jobs of 480 to 14000
// limbs): 0.35 ms with a warp a job, 0.16 ms with a CTA.  Up to 512 limbs a
// warp's few steps are as fast, and many jobs share a CTA.
cudaError_t add_batch(const AddJob* d_jobs, u64 m, u64 longest, cudaStream_t st) {
  if (m == 0) return cudaSuccess;
  launch_begin("add_batch", st);
  const cudaError_t e = longest > 512
                            ? launch_next(add_batch_long_kernel, (unsigned)m, 256, 0, 0, st, d_jobs)
                            : launch_next(add_batch_kernel, (unsigned)((m * 32 + 255) / 256), 256, 0, 0, st, d_jobs, m);
  launch_end(st);
  return e;
}

bool school_whole(u64 na, u64 nb) {
  return na + nb <= kSchoolClusterTile * kSchoolClusterCtas && std::min(na, nb) <= kSchoolShorter;
}
cudaError_t school_mul(const u64* a, u64 na, const u64* b, u64 nb, u64* out, Scan& sc, cudaStream_t st) {
  const u64 total = na + nb;
  const ColumnProducer prod = na >= nb ? ColumnProducer{a, na, b, nb} : ColumnProducer{b, nb, a, na};
  if (school_whole(na, nb)) {
    static DeviceOnce once;  // clusters of more than eight CTAs want asking
    cudaError_t e = kernel_attribute(once, school_cluster_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    const unsigned tiles = (unsigned)((total + kSchoolClusterTile - 1) / kSchoolClusterTile);
    launch_begin("school_tiles", st);
    e = launch_next(school_cluster_kernel, tiles, 256, 0, tiles, st, prod, total, out);
    launch_end(st);
    return e;
  }
  if (total <= kSchoolShort) return launch_school<kSchoolTile>(prod, total, out, sc, st);
  const u64 tiles = (total + kSchoolWideTile - 1) / kSchoolWideTile;
  if (total <= kSchoolLong || (prod.nb > kSchoolFew && tiles <= 0x7fffffff)) {
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (tiles <= sc.max_tiles ||
        (cudaStreamIsCapturing(st, &capture) == cudaSuccess && capture == cudaStreamCaptureStatusNone))
      return launch_school<kSchoolWideTile>(prod, total, out, sc, st);
  }
  return run_scan(prod, total, out, total, sc, st, "school_column_scan");
}

cudaError_t add_shifted(const u64* x, u64 nx, const u64* y, u64 ny, u64 shift, u64* out, u64 n, Scan& sc,
                        cudaStream_t st) {
  cudaError_t e = scan_reserve(sc, 1);
  if (e != cudaSuccess) return e;
  return run_scan(AddProducer{x, nx, y, ny, shift}, n, out, n, sc, st, "add_scan");
}

cudaError_t lin_combine(u64* out, u64 n_out, const u64* x, u64 nx, u64 xs, const u64* y, u64 ny, u64 ys, bool sub,
                        int cin, Scan& sc, cudaStream_t st, const u64* flip) {
  cudaError_t e = scan_reserve(sc, 1);
  if (e != cudaSuccess) return e;
  return run_scan(LinProducer{x, nx, xs, y, ny, ys, n_out, sub ? 1 : 0, cin, flip}, n_out + 1, out, n_out + 1, sc,
                  st, sub ? "sub_scan" : "add_scan");
}

cudaError_t shl_bits(u64* out, const u64* in, u64 n, unsigned cl, cudaStream_t st) {
  if (cl == 0) {
    cudaError_t e = cudaMemcpyAsync(out, in, n * 8, cudaMemcpyDeviceToDevice, st);
    return e == cudaSuccess ? cudaMemsetAsync(out + n, 0, 8, st) : e;
  }
  const unsigned blocks = (unsigned)std::min<u64>((n + 1 + 255) / 256, 152 * 16);
  launch_begin("shift_bits", st);
  const cudaError_t e = launch_next(shl_bits_kernel, blocks, 256, 0, 0, st, out, in, n, cl);
  launch_end(st);
  return e;
}

cudaError_t shr_bits(u64* out, const u64* in, u64 n, unsigned cl, cudaStream_t st) {
  if (cl == 0) return cudaMemcpyAsync(out, in, n * 8, cudaMemcpyDeviceToDevice, st);
  const unsigned blocks = (unsigned)std::min<u64>((n + 255) / 256, 152 * 16);
  launch_begin("shift_bits", st);
  const cudaError_t e = launch_next(shr_bits_kernel, blocks, 256, 0, 0, st, out, in, n, cl);
  launch_end(st);
  return e;
}

cudaError_t wait_probe(Scan& sc, int limit, cudaStream_t st) {
  cudaError_t e = scan_reserve(sc, 1);
  if (e != cudaSuccess) return e;
  launch_begin("wait_probe", st);
  wait_probe_kernel<<<1, 32, 0, st>>>(sc.probe, sc.err, limit);
  launch_end(st);
  return cudaGetLastError();
}

}  // namespace nn
