// six.cu — the product pipeline over six 32-bit primes on sm_103a: twiddle
// tables, the tiled passes and their launches (six_tiles.cuh has the
// arithmetic and the tiles).
//
// A transform of scale s runs T = min(s - 3, 22) levels: strided passes of up
// to 9 levels (tiles of 2^R rows x 128 bytes), then one pass over contiguous
// tiles of 4096 words, which takes both operands through their last levels,
// multiplies them block by block and runs the first inverse levels, so
// neither operand's finished transform goes through memory:
//   scale  4-12  1 pass   limbs -> product residues
//   scale 13-21  2 passes load, fused, inverse
//   scale 22-31  3 passes load, strided, fused, inverse strided, inverse
// Both operands' strided passes share a launch (and the pieces of a split
// operand do).  Groups of at most three levels run in registers (eight rows of
// four columns a thread); the first group of a pass reads global memory
// directly and the last one writes it, so a pass of eight levels crosses
// shared memory twice.
#include <cuda_runtime.h>

#include <algorithm>

#include "nn_device.cuh"
#include "nn_internal.h"
#include "six_tiles.cuh"

namespace nn {

namespace {

using namespace six;
typedef unsigned __int128 h128;

u64 h_pow(u64 b, u64 e, u64 p) {
  u64 r = 1;
  for (b %= p; e; e >>= 1, b = b * b % p)
    if (e & 1) r = r * b % p;
  return r;
}
i32 h_center(u64 w, u64 p) { return (i32)(w > p / 2 ? (i64)w - (i64)p : (i64)w); }
i32 h_companion(i32 w, u64 p) {  // round(w 2^32 / p)
  const i64 n = (i64)w * (1ll << 32), h = (i64)p / 2;
  return (i32)((n + (n < 0 ? -h : h)) / (i64)p);
}
// An element of order 2^22 modulo each p.
u64 h_root(u64 p) {
  for (u64 a = 2;; ++a) {
    const u64 g = h_pow(a, (p - 1) >> kRootLog, p);
    if (h_pow(g, 1ull << (kRootLog - 1), p) == p - 1) return g;
  }
}

// rho_t and its inverse for every prime: the factors of the table entries.
struct Factors {
  int2 f[2][kPrimes][kRootLog - 1];  // (w, companion)
};
Factors make_factors() {
  Factors F;
  for (int i = 0; i < kPrimes; ++i) {
    const u64 p = prime_of(i), g = h_root(p);
    for (int t = 0; t < kRootLog - 1; ++t) {  // rho_t has order 2^(t+2)
      const u64 r = h_pow(g, 1ull << (kRootLog - 2 - t), p);
      const i32 w = h_center(r, p), v = h_center(h_pow(r, p - 2, p), p);
      F.f[0][i][t] = make_int2(w, h_companion(w, p));
      F.f[1][i][t] = make_int2(v, h_companion(v, p));
    }
  }
  return F;
}

// 2^(32 steps - t) / (M / p_i) modulo each prime, by t.
struct ScaleTable {
  int2 f[kRootLog + 2][kPrimes];
};
ScaleTable make_scales(int steps) {
  ScaleTable S;
  for (int i = 0; i < kPrimes; ++i) {
    const u64 p = prime_of(i);
    u64 m = 1;
    for (int j = 0; j < kPrimes; ++j)
      if (j != i) m = m * (prime_of(j) % p) % p;
    const u64 inv = h_pow(m, p - 2, p);
    for (int t = 0; t < kRootLog + 2; ++t) {
      const i32 w = h_center(h_pow(2, 32 * steps - t, p) * inv % p, p);
      S.f[t][i] = make_int2(w, h_companion(w, p));
    }
  }
  return S;
}

// W[b] = the product of rho_t over the bits t of b (and of the inverses in
// the second direction), centred, with its companion.  One launch writes
// every entry of the 12 tables; an entry is at most 21 products.
__global__ void __launch_bounds__(256) six_table_kernel(int2* tab, u64 cap, const Factors F) {
  const u64 b = (u64)blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= cap) return;
  const int dir = blockIdx.y / kPrimes, prime = blockIdx.y % kPrimes;
  const i32 p = c_primes[prime].p;
  i32 w = 1;
  for (int t = 0; t < kRootLog - 1; ++t)
    if ((b >> t) & 1) w = mul_mod(w, F.f[dir][prime][t].x, F.f[dir][prime][t].y, p);
  const i32 h = p >> 1;
  if (w > h) w -= p;
  if (w < -h) w += p;
  const i64 n = (i64)w << 32;
  tab[blockIdx.y * cap + b] = make_int2(w, (i32)((n + (n < 0 ? -(i64)h : (i64)h)) / p));
}

// First pass of up to two operands, the first in pieces: CTA (6 tile + prime,
// y): piece y of a, or b for y = pieces.  The CTAs of one tile's six primes
// run together, so its limbs cross HBM about once.
template <int R>
__global__ void __launch_bounds__(col_threads(R), col_blocks(R))
    six_load_kernel(SixOperands op, int s, const int2* __restrict__ tab, u64 cap, u32 tile0, int k8) {
  grid_begin();
  extern __shared__ __align__(16) u32 sm6[];
  const int prime = (int)(blockIdx.x % kPrimes);
  const u32 tile = tile0 + blockIdx.x / kPrimes;
  if (blockIdx.y < op.pieces) {
    const u64 at0 = blockIdx.y * op.piece;
    load_tile<R, col_width(R), col_threads(R)>(sm6, op.a + at0, min(op.piece, op.na - at0),
                                        op.ra + ((u64)blockIdx.y * kPrimes << s), s, tile, prime, tab, cap, k8);
  } else {
    load_tile<R, col_width(R), col_threads(R)>(sm6, op.b, op.nb, op.rb, s, tile, prime, tab, cap, k8);
  }
}

template <int R, bool INV>
__global__ void __launch_bounds__(col_threads(R), col_blocks(R))
    six_col_kernel(u32* ra, u32* rb, u32 pieces, const SixPlan pl, int lambda0, const int2* __restrict__ tab, u64 cap) {
  grid_begin();
  extern __shared__ __align__(16) u32 sm6[];
  u32* res = blockIdx.z < pieces ? ra + ((u64)blockIdx.z * kPrimes << pl.s) : rb;
  const bool last = INV && lambda0 == 0;
  col_tile<R, col_width(R), col_threads(R), INV>(sm6, res, pl.s, lambda0, blockIdx.x, blockIdx.y, tab, cap, last,
                                                           pl.scale[blockIdx.y], last ? pl.k8 : 8);
}

// op.ra's pieces (or, FIRST, the limbs op.a) with op.rb (op.b), into `out`;
// modes kForward and kInverse: op.ra alone.
template <int R, int LGM, int V, int MODE, bool FIRST, bool PAIR>
__global__ void __launch_bounds__(fused_threads(R, LGM, V) * (PAIR ? 2 : 1), PAIR ? 1 : fused_blocks(R, LGM, V))
    six_fused_kernel(SixOperands op, u32* out, const SixPlan pl, const int2* __restrict__ tab, u64 cap) {
  grid_begin();
  extern __shared__ __align__(16) u32 sm6[];
  constexpr int NT = fused_threads(R, LGM, V);
  const u64 piece = ((u64)blockIdx.z * kPrimes) << pl.s, at0 = blockIdx.z * op.piece;
  const void* a = FIRST ? static_cast<const void*>(op.a + at0) : op.ra + piece;
  const void* b = FIRST && MODE == kAll ? static_cast<const void*>(op.b) : op.rb;
  const bool last = pl.n == 1;
  fused_tile<R, LGM, NT, V, MODE, FIRST, PAIR>(sm6, a, min(op.piece, op.na - at0), b, op.nb, out + piece, pl.s, blockIdx.x,
                                         blockIdx.y, tab, tab + kPrimes * cap, cap, pl.reduce_in(), last,
                                         pl.scale[blockIdx.y], last ? pl.k8 : 8);
}

template <int R>
cudaError_t launch_load(const SixOperands& op, int s, int k8, const SixTables& t, u32 tile0, u32 tile1,
                        cudaStream_t st) {
  constexpr int smem = col_smem(R);
  static DeviceOnce once;
  if (const cudaError_t e = allow_smem<smem>(once, six_load_kernel<R>); e != cudaSuccess) return e;
  const u32 tiles = (u32)((1ull << s) / ((u64)col_width(R) << R));
  tile1 = std::min(tile1, tiles);
  const dim3 grid(kPrimes * (tile1 - tile0), op.pieces + (op.b ? 1 : 0));
  launch_begin("six_load_col_pass", st);
  const cudaError_t e = launch_next(six_load_kernel<R>, grid, col_threads(R), smem, 0, st, op, s, t.tab, t.cap, tile0, k8);
  launch_end(st);
  return e;
}
template <int R, bool INV>
cudaError_t launch_col(u32* ra, u32* rb, u32 pieces, const SixPlan& pl, int lambda0, const SixTables& t,
                       cudaStream_t st) {
  constexpr int smem = col_smem(R);
  static DeviceOnce once;
  if (const cudaError_t e = allow_smem<smem>(once, six_col_kernel<R, INV>); e != cudaSuccess) return e;
  // past the first pass, only the blocks of the first k8 eighths
  const u64 tiles = (1ull << pl.s) / ((u64)col_width(R) << R);
  const dim3 grid((unsigned)(lambda0 ? tiles / 8 * pl.k8 : tiles), kPrimes, pieces + (rb ? 1 : 0));
  launch_begin(INV ? (lambda0 == 0 ? "six_inv_last_col_pass" : "six_inv_col_pass") : "six_fwd_col_pass", st);
  const cudaError_t e = launch_next(six_col_kernel<R, INV>, grid, col_threads(R), smem, 0, st, ra, rb, pieces, pl,
                                    lambda0, t.tab + (INV ? kPrimes * t.cap : 0), t.cap);
  launch_end(st);
  return e;
}
template <int R, int LGM, int V, int MODE, bool FIRST, bool PAIR = false>
cudaError_t launch_fused_v(const SixOperands& op, u32* out, const SixPlan& pl, const SixTables& t, cudaStream_t st) {
  constexpr int tile = (int)tile_words32<1 << LGM, true>(R) * 4, smem = fused_tiles(LGM, MODE) * tile + (PAIR ? (16 << (R - 1)) : 0);
  static DeviceOnce once;
  if (const cudaError_t e = allow_smem<smem>(once, six_fused_kernel<R, LGM, V, MODE, FIRST, PAIR>); e != cudaSuccess)
    return e;
  const u32 tiles = (u32)((1ull << pl.s) >> (R + LGM));
  const dim3 grid(pl.n == 1 ? 1u : tiles / 8 * pl.k8, kPrimes, op.pieces);
  launch_begin(MODE == kForward ? "six_fwd_row_pass" : MODE == kInverse ? "six_inv_row_pass" : FIRST ? "six_small_pass" : "six_fused_row_pass", st);
  const cudaError_t e =
      launch_next(six_fused_kernel<R, LGM, V, MODE, FIRST, PAIR>, grid, fused_threads(R, LGM, V) * (PAIR ? 2 : 1),
                  MODE == kAll && !op.b ? tile : smem, 0, st, op, out, pl, t.tab, t.cap);
  launch_end(st);
  return e;
}
// A few one-pass products: an operand a half of the CTA (six CTAs a piece:
// up to 96 fill under one wave).  Columns a thread: as few as keep the grid
// within one wave of the GPU's 152 x 768 threads, so a short product uses as
// many of them as it can (a limit of 1024 threads: 18.7 instead of 17.7 us for
// the pass at scale 18).
template <int R, int LGM, int MODE, bool FIRST>
cudaError_t launch_fused(const SixOperands& op, u32* out, const SixPlan& pl, const SixTables& t, cudaStream_t st) {
  if constexpr (FIRST && MODE == kAll && R >= 5)
    if (op.b && op.pieces <= 16) return launch_fused_v<R, LGM, 1, MODE, FIRST, true>(op, out, pl, t, st);
  if constexpr (LGM == 3)
    if (((u64)kPrimes * op.pieces << pl.s) / 64 * pl.k8 <= 152 * 768)
      return launch_fused_v<R, LGM, 1, MODE, FIRST>(op, out, pl, t, st);
  return launch_fused_v<R, LGM, 4, MODE, FIRST>(op, out, pl, t, st);
}

cudaError_t load_pass(const SixOperands& op, int s, int k8, int R, const SixTables& t, u32 t0, u32 t1,
                      cudaStream_t st) {
  switch (R) {
    case 4: return launch_load<4>(op, s, k8, t, t0, t1, st);
    case 5: return launch_load<5>(op, s, k8, t, t0, t1, st);
    case 6: return launch_load<6>(op, s, k8, t, t0, t1, st);
    case 7: return launch_load<7>(op, s, k8, t, t0, t1, st);
    case 8: return launch_load<8>(op, s, k8, t, t0, t1, st);
    case 9: return launch_load<9>(op, s, k8, t, t0, t1, st);
  }
  return cudaErrorInvalidValue;
}
template <bool INV>
cudaError_t col_pass(u32* ra, u32* rb, u32 pieces, const SixPlan& pl, int k, const SixTables& t, cudaStream_t st) {
  const int lambda0 = pl.lambda0[k];
  switch (pl.R[k]) {
    case 4: return launch_col<4, INV>(ra, rb, pieces, pl, lambda0, t, st);
    case 5: return launch_col<5, INV>(ra, rb, pieces, pl, lambda0, t, st);
    case 6: return launch_col<6, INV>(ra, rb, pieces, pl, lambda0, t, st);
    case 7: return launch_col<7, INV>(ra, rb, pieces, pl, lambda0, t, st);
    case 8: return launch_col<8, INV>(ra, rb, pieces, pl, lambda0, t, st);
    case 9: return launch_col<9, INV>(ra, rb, pieces, pl, lambda0, t, st);
  }
  return cudaErrorInvalidValue;
}
// FIRST: from limbs, the plan's only pass.
template <int MODE, bool FIRST>
cudaError_t fused_pass(const SixOperands& op, u32* out, const SixPlan& pl, const SixTables& t, cudaStream_t st) {
  const int R = pl.R[pl.n - 1];
  if constexpr (!FIRST) {
    switch (pl.lgm) {
      case 4: return launch_fused<8, 4, MODE, false>(op, out, pl, t, st);
      case 5: return launch_fused<7, 5, MODE, false>(op, out, pl, t, st);
      case 6: return launch_fused<6, 6, MODE, false>(op, out, pl, t, st);
      case 7: return launch_fused<5, 7, MODE, false>(op, out, pl, t, st);
      case 8: return launch_fused<4, 8, MODE, false>(op, out, pl, t, st);
      case 9: return launch_fused<4, 9, MODE, false>(op, out, pl, t, st);
    }
  }
  if constexpr (FIRST || MODE == kProduct || MODE == kInverse) {
    switch (R) {
      case 1: return launch_fused<1, 3, MODE, FIRST>(op, out, pl, t, st);
      case 2: return launch_fused<2, 3, MODE, FIRST>(op, out, pl, t, st);
      case 3: return launch_fused<3, 3, MODE, FIRST>(op, out, pl, t, st);
      case 4: return launch_fused<4, 3, MODE, FIRST>(op, out, pl, t, st);
    }
  }
  switch (R) {
    case 5: return launch_fused<5, 3, MODE, FIRST>(op, out, pl, t, st);
    case 6: return launch_fused<6, 3, MODE, FIRST>(op, out, pl, t, st);
    case 7: return launch_fused<7, 3, MODE, FIRST>(op, out, pl, t, st);
    case 8: return launch_fused<8, 3, MODE, FIRST>(op, out, pl, t, st);
    case 9: return launch_fused<9, 3, MODE, FIRST>(op, out, pl, t, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace

SixPlan six_plan(int s, u64 length, int row_levels) {
  SixPlan pl{};
  pl.s = s;
  const int T = std::min(s - 3, kRootLog);
  pl.lgm = s - T;
  const int row_max = std::max(12 - pl.lgm, 4);  // contiguous tiles of 4096 words (8192 at scale 31)
  pl.n = T <= row_max ? 1 : T <= row_max + 9 ? 2 : 3;
  // The contiguous tile as long as the strided passes keep four levels (two
  // passes: batched products of 2^14 limbs 0.084 ns a limb with 9 levels there,
  // 0.126 with 6) or six (three passes: 2^24 x 2^24 limbs 2.80 ms with 6 + 7 +
  // 9 levels, 2.86 with 7 + 7 + 8; at 2^21 7 levels and 9 read 348 and 355 us).
  int row = T;
  if (pl.n == 2) row = std::min(9, T - 4);
  if (pl.n == 3) row = pl.lgm > 3 ? row_max : std::min(9, T - 12);
  if (pl.n == 2 && row_levels >= 5 && row_levels <= 9 && T - row_levels >= 4 && T - row_levels <= 9) row = row_levels;
  for (int k = 0, left = T - row; k + 1 < pl.n; ++k) {
    pl.R[k] = left / (pl.n - 1 - k);
    pl.lambda0[k + 1] = pl.lambda0[k] + pl.R[k];
    left -= pl.R[k];
  }
  pl.R[pl.n - 1] = row;
  const u64 eighth = (1ull << s) / 8;
  pl.k8 = pl.R[0] >= 3 ? (int)std::clamp<u64>((length + eighth - 1) / eighth, 5, 8) : 8;
  // The product residues are the coefficients times 2^T (the inverse's sums;
  // 2^(T+1) of a truncated transform) and 2^-96 (the Montgomery steps of the
  // two operands' limbs and of the blocks' products).
  static const ScaleTable scales = make_scales(3);
  std::copy_n(scales.f[T + (pl.k8 < 8)], kPrimes, pl.scale);
  return pl;
}

SixPlan six_inverse_plan(int s) {
  SixPlan pl = six_plan(s, 1ull << s);
  // the inverse's sums, and the one Montgomery step of the operand's limbs
  static const ScaleTable scales = make_scales(1);
  std::copy_n(scales.f[std::min(s - 3, kRootLog)], kPrimes, pl.scale);
  return pl;
}

cudaError_t six_tables_ensure(SixTables& t, int s, cudaStream_t st, std::vector<u64*>* retired) {
  const u64 need = std::max<u64>(8, 1ull << (std::min(std::max(s, kSixMinScale) - 3, kRootLog) - 1));
  if (t.cap >= need) return cudaSuccess;
  // from the size of one-pass transforms at once, then doubling: a handful of
  // growths in a context's life
  const u64 cap = std::max<u64>(need, 1 << 12);
  int2* tab = nullptr;
  cudaError_t e = cudaMallocAsync((void**)&tab, 2 * kPrimes * cap * sizeof(int2), st);
  if (e != cudaSuccess) return e;
  static const Factors F = make_factors();
  launch_begin("six_table", st);
  six_table_kernel<<<dim3((unsigned)((cap + 255) / 256), 2 * kPrimes), 256, 0, st>>>(tab, cap, F);
  launch_end(st);
  e = cudaGetLastError();
  // other streams of the context read the table from the next launch on
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) {
    cudaFreeAsync(tab, st);
    return e;
  }
  if (t.tab) {
    if (retired)
      retired->push_back(reinterpret_cast<u64*>(t.tab));
    else
      cudaFreeAsync(t.tab, st);
  }
  t.tab = tab;
  t.cap = cap;
  return cudaSuccess;
}

void six_tables_free(SixTables& t) {
  if (t.tab) cudaFree(t.tab);
  t = SixTables{};
}

u32 six_first_pass_tiles(const SixPlan& pl) {
  return pl.n == 1 ? 0 : (u32)((1ull << pl.s) / ((u64)col_width(pl.R[0]) << pl.R[0]));
}
u32 six_first_pass_columns(const SixPlan& pl) { return (u32)col_width(pl.R[0]); }

cudaError_t six_load(const SixOperands& op, const SixPlan& pl, const SixTables& t, cudaStream_t st, u32 tile0,
                     u32 tile1) {
  return pl.n == 1 ? cudaSuccess : load_pass(op, pl.s, pl.k8, pl.R[0], t, tile0, tile1, st);
}

namespace {
cudaError_t forward_cols(const SixOperands& op, const SixPlan& pl, const SixTables& t, cudaStream_t st) {
  cudaError_t e = cudaSuccess;
  for (int k = 1; k + 1 < pl.n && e == cudaSuccess; ++k)
    e = col_pass<false>(op.ra, op.b ? op.rb : nullptr, op.pieces, pl, k, t, st);
  return e;
}
cudaError_t inverse_cols(u32* res, u32 pieces, const SixPlan& pl, const SixTables& t, cudaStream_t st) {
  cudaError_t e = cudaSuccess;
  for (int k = pl.n - 2; k >= 0 && e == cudaSuccess; --k) e = col_pass<true>(res, nullptr, pieces, pl, k, t, st);
  return e;
}
}  // namespace

cudaError_t six_finish(const SixOperands& op, const SixPlan& pl, const SixTables& t, cudaStream_t st) {
  cudaError_t e = forward_cols(op, pl, t, st);
  if (e == cudaSuccess) {
    if (six_ready(op, pl)) {  // the shorter operand's last levels once, not once a piece
      const SixOperands b{op.b, op.nb, op.nb, 1, nullptr, 0, op.rb, nullptr};
      e = pl.n == 1 ? fused_pass<kForward, true>(b, op.rb, pl, t, st) : fused_pass<kForward, false>(b, op.rb, pl, t, st);
      if (e == cudaSuccess)
        e = pl.n == 1 ? fused_pass<kReady, true>(op, op.ra, pl, t, st) : fused_pass<kReady, false>(op, op.ra, pl, t, st);
    } else {
      e = pl.n == 1 ? fused_pass<kAll, true>(op, op.ra, pl, t, st) : fused_pass<kAll, false>(op, op.ra, pl, t, st);
    }
  }
  return e == cudaSuccess ? inverse_cols(op.ra, op.pieces, pl, t, st) : e;
}

cudaError_t six_forward(const u64* limbs, u64 n, u32* res, const SixPlan& pl, const SixTables& t, cudaStream_t st) {
  const SixOperands op{limbs, n, n, 1, nullptr, 0, res, nullptr};
  cudaError_t e = six_load(op, pl, t, st);
  if (e == cudaSuccess) e = forward_cols(op, pl, t, st);
  if (e != cudaSuccess) return e;
  return pl.n == 1 ? fused_pass<kForward, true>(op, res, pl, t, st) : fused_pass<kForward, false>(op, res, pl, t, st);
}

cudaError_t six_pointwise(u32* dst, const u32* a, const u32* b, const SixPlan& pl, const SixTables& t, cudaStream_t st) {
  const SixOperands op{nullptr, 0, 0, 1, nullptr, 0, const_cast<u32*>(a), const_cast<u32*>(b)};
  const cudaError_t e = fused_pass<kProduct, false>(op, dst, pl, t, st);
  return e == cudaSuccess ? inverse_cols(dst, 1, pl, t, st) : e;
}

cudaError_t six_inverse(u32* dst, const u32* a, const SixPlan& pl, const SixTables& t, cudaStream_t st) {
  const SixOperands op{nullptr, 0, 0, 1, nullptr, 0, const_cast<u32*>(a), nullptr};
  const cudaError_t e = fused_pass<kInverse, false>(op, dst, pl, t, st);
  return e == cudaSuccess ? inverse_cols(dst, 1, pl, t, st) : e;
}

}  // namespace nn
