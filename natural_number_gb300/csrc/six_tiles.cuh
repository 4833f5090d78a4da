// six_tiles.cuh — tile-level device code of the six-prime 32-bit NTT, shared
// by the per-call kernels (six.cu) and the batches' (batch.cu).
//
// A product of limbs is a convolution of 64-bit digits whose coefficients
// stay below min(n_a, n_b) * 2^128.  It is computed modulo six primes
// p = m * 2^22 + 1 just below 2^27.4 (product 2^162) instead of three 62-bit
// ones: the same 24 bytes a coefficient, but a butterfly is one
// multiply-high and two multiply-adds of 32 bits (8 cycles of the multiply
// pipe a warp and scheduler on GB300, 8.9 measured in a register-only loop,
// so 53 for the six primes) where a 64-bit Shoup butterfly takes 46 a prime,
// 137 for the three.
//
// Residues are signed 32-bit words, lazy: |x| < 2^31, at least 12.8 p.  With
// a twiddle pair (w, wp = round(w 2^32 / p)), |w| < p/2, the product y w - q p
// with q = round(y wp / 2^32) is at most (1/2 + |y| / 2^33) p in magnitude, so
//  - a forward butterfly (x, y) -> (x + w y, x - w y) adds at most
//    p (1/2 + |y|/2^33): from |x| <= p, 18 levels stay below 12.1 p (and a
//    transform of more levels reduces its values once on the way);
//  - an inverse butterfly (x, y) -> (x + y, (x - y) w) doubles its sums: a
//    group of three levels takes values of at most 1.5 p to sums of at most
//    12 p; the first two of its eight outputs (one for shorter groups) are
//    then reduced and the others are below 1.5 p again.
//
// The transform is the CRT tree of x^L - 1: block b at any level is taken
// modulo x^h - c_b and splits with w = W[b] = sqrt(c_b) into x^(h/2) - w (child
// 2b) and x^(h/2) + w (child 2b + 1); W[b] is the product of rho_t over the
// bits t of b, rho_t a primitive 2^(t+2)-th root, so one table serves every
// level and length.  The tree stops at blocks of m = 2^lgm coefficients
// (m = 8 up to L = 2^25; 2^22 is the order of the roots), which are multiplied
// directly modulo x^m - c_b: at m = 8 the eight multiply-adds a coefficient
// cost less than the three levels they replace.
#pragma once

#include <cstdint>
#include <type_traits>

#include "nn_device.cuh"

namespace nn {
namespace six {

typedef int i32;

constexpr int kPrimes = 6;
constexpr int kRootLog = 22;    // 2^22 divides every p - 1
constexpr u32 kMul[kPrimes] = {25, 27, 33, 37, 39, 40};  // p = m * 2^22 + 1

struct Prime {
  i32 p;
  u32 pinv;  // p^-1 mod 2^32 = 1 - m 2^22
  i32 u;     // round(2^32 / p)
  u32 c32;   // 2^32 mod p
  i32 r, rp; // the same centred, and its companion round(r 2^32 / p)
};
constexpr u32 prime_of(int i) { return kMul[i] << 22 | 1; }
constexpr Prime make_prime(int i) {
  const u64 p = prime_of(i), two32 = 1ull << 32;
  // 2^32 mod p as a factor of products wants its companion in 32 signed bits: centred
  const u64 c = two32 % p;
  const i64 cc = c > p / 2 ? (i64)c - (i64)p : (i64)c, n = cc * (i64)two32, h = (i64)p / 2;
  return Prime{(i32)p, (u32)(1u - (kMul[i] << 22)), (i32)((two32 + p / 2) / p), (u32)c, (i32)cc,
               (i32)((n + (n < 0 ? -h : h)) / (i64)p)};
}
static __constant__ Prime c_primes[kPrimes] = {make_prime(0), make_prime(1), make_prime(2),
                                               make_prime(3), make_prime(4), make_prime(5)};

// round(y * wp / 2^32)
__device__ __forceinline__ i32 mulhi_round(i32 y, i32 wp) {
  return (i32)(((i64)y * wp + 0x80000000ll) >> 32);
}
// y * w mod p, at most (1/2 + |y|/2^33) p in magnitude.
__device__ __forceinline__ i32 mul_mod(i32 y, i32 w, i32 wp, i32 p) {
  return (i32)((u32)y * (u32)w - (u32)mulhi_round(y, wp) * (u32)p);
}
// Any word to at most 0.75 p in magnitude.
__device__ __forceinline__ i32 reduce(i32 x, const Prime& P) {
  return (i32)((u32)x - (u32)mulhi_round(x, P.u) * (u32)P.p);
}
// x, y -> x + w y, x - w y: the product enters the first sum as its
// multiply-adds' addend, the second is 2 x minus the first.
__device__ __forceinline__ void fwd_bfly(i32& x, i32& y, i32 w, i32 wp, i32 p) {
  const u32 q = (u32)mulhi_round(y, wp);
  const u32 s = (u32)y * (u32)w + (u32)x - q * (u32)p;
  y = (i32)(2u * (u32)x - s);
  x = (i32)s;
}
__device__ __forceinline__ void inv_bfly(i32& x, i32& y, i32 w, i32 wp, i32 p) {
  const i32 d = (i32)((u32)x - (u32)y);
  x = (i32)((u32)x + (u32)y);
  y = mul_mod(d, w, wp, p);
}
// limb * 2^-32 mod p, below p in magnitude (Montgomery step on hi * 2^32 mod
// p * + lo, which is below 2^32 p).
__device__ __forceinline__ i32 limb_residue(u64 limb, const Prime& P) {
  const u64 t = (u64)(u32)(limb >> 32) * P.c32 + (u32)limb;
  const u32 m = (u32)t * P.pinv;
  return (i32)((u32)(t >> 32) - __umulhi(m, (u32)P.p));
}
// c * 2^-32 mod p, at most |c| / 2^32 + p/2 in magnitude.
__device__ __forceinline__ i32 mont(i64 c, const Prime& P) {
  const i32 m = (i32)((u32)c * P.pinv);
  return (i32)((u32)(c >> 32) - (u32)__mulhi(m, P.p));
}

// V neighbouring words: one 16-, 8- or 4-byte access.
template <int V>
struct alignas(4 * V) Words {
  i32 v[V];
};
template <int V>
__device__ __forceinline__ Words<V> ldv(const void* p) {
  Words<V> w;
  if constexpr (V == 4) {
    const int4 t = *reinterpret_cast<const int4*>(p);
    w.v[0] = t.x, w.v[1] = t.y, w.v[2] = t.z, w.v[3] = t.w;
  } else if constexpr (V == 2) {
    const int2 t = *reinterpret_cast<const int2*>(p);
    w.v[0] = t.x, w.v[1] = t.y;
  } else {
    w.v[0] = *reinterpret_cast<const i32*>(p);
  }
  return w;
}
template <int V>
__device__ __forceinline__ void stv(void* p, const Words<V>& w) {
  if constexpr (V == 4)
    *reinterpret_cast<int4*>(p) = make_int4(w.v[0], w.v[1], w.v[2], w.v[3]);
  else if constexpr (V == 2)
    *reinterpret_cast<int2*>(p) = make_int2(w.v[0], w.v[1]);
  else
    *reinterpret_cast<i32*>(p) = w.v[0];
}

// A unit: 2^K rows of V neighbouring columns in registers.  V = 4 has the
// fewest shared-memory instructions and twiddle loads a butterfly; V = 1 and 2
// spread a short transform over four and two times the threads, where the
// GPU would otherwise be mostly idle.
template <int K, int V>
struct Unit {
  i32 x[1 << K][V];
  __device__ __forceinline__ void set(int m, const Words<V>& w) {
#pragma unroll
    for (int c = 0; c < V; ++c) x[m][c] = w.v[c];
  }
  __device__ __forceinline__ Words<V> get(int m) const {
    Words<V> w;
#pragma unroll
    for (int c = 0; c < V; ++c) w.v[c] = x[m][c];
    return w;
  }
};

// A table of roots in global memory (read-only cache), or the part of it that
// a tile needs, copied to shared memory.
struct GlobalRoots {
  const int2* p;
  __device__ __forceinline__ int2 one(u32 b) const { return __ldg(p + b); }
  __device__ __forceinline__ int4 pair(u64 b) const { return __ldg(reinterpret_cast<const int4*>(p + b)); }
};
struct SharedRoots {
  const int2* p;
  __device__ __forceinline__ int2 one(u32 b) const { return p[b]; }
  __device__ __forceinline__ int4 pair(u64 b) const { return *reinterpret_cast<const int4*>(p + b); }
};

// The twiddle pairs of local level lv of a unit whose block index at the
// unit's first level is b: W[b 2^lv + g], g < 2^lv.
template <int LV, class Roots>
__device__ __forceinline__ void twiddles(int2 (&w)[1 << LV], const Roots& tw, u32 b) {
  if constexpr (LV == 0) {
    w[0] = tw.one(b);
  } else {
#pragma unroll
    for (int g = 0; g < (1 << LV); g += 2) {
      const int4 v = tw.pair(((u64)b << LV) + g);
      w[g] = make_int2(v.x, v.y);
      w[g + 1] = make_int2(v.z, v.w);
    }
  }
}

template <int K, int V, int LV, class Roots>
__device__ __forceinline__ void fwd_level(Unit<K, V>& u, const Roots& tw, u32 b, i32 p) {
  int2 w[1 << LV];
  twiddles<LV>(w, tw, b);
  constexpr int half = (1 << K) >> (LV + 1);
#pragma unroll
  for (int g = 0; g < (1 << LV); ++g)
#pragma unroll
    for (int m = 0; m < half; ++m)
#pragma unroll
      for (int c = 0; c < V; ++c)
        fwd_bfly(u.x[g * 2 * half + m][c], u.x[g * 2 * half + m + half][c], w[g].x, w[g].y, p);
}
// Levels [LV0, K) of a unit.
template <int K, int LV = 0, int V, class Roots>
__device__ __forceinline__ void fwd_levels(Unit<K, V>& u, const Roots& tw, u32 b, i32 p) {
  if constexpr (LV < K) {
    fwd_level<K, V, LV>(u, tw, b, p);
    fwd_levels<K, LV + 1>(u, tw, b, p);
  }
}

template <int K, int V, int LV, class Roots>
__device__ __forceinline__ void inv_level(Unit<K, V>& u, const Roots& tw, u32 b, i32 p) {
  int2 w[1 << LV];
  twiddles<LV>(w, tw, b);
  constexpr int half = (1 << K) >> (LV + 1);
#pragma unroll
  for (int g = 0; g < (1 << LV); ++g)
#pragma unroll
    for (int m = 0; m < half; ++m)
#pragma unroll
      for (int c = 0; c < V; ++c)
        inv_bfly(u.x[g * 2 * half + m][c], u.x[g * 2 * half + m + half][c], w[g].x, w[g].y, p);
}
template <int K, int LV = K - 1, int V, class Roots>
__device__ __forceinline__ void inv_levels(Unit<K, V>& u, const Roots& tw, u32 b, i32 p) {
  if constexpr (LV >= 0) {
    inv_level<K, V, LV>(u, tw, b, p);
    inv_levels<K, LV - 1>(u, tw, b, p);
  }
}
// The outputs of an inverse group above 1.5 p: row 0, and row 1 of three levels.
template <int K, int V>
__device__ __forceinline__ void inv_fold(Unit<K, V>& u, const Prime& P) {
#pragma unroll
  for (int m = 0; m < (K == 3 ? 2 : 1); ++m)
#pragma unroll
    for (int c = 0; c < V; ++c) u.x[m][c] = reduce(u.x[m][c], P);
}

// Truncated transforms.  A product of at most k/8 L coefficients, k = 5, 6, 7,
// is determined by its residues in the first k of the eight blocks at depth
// 3: the passes then leave the others out, and only the last inverse group
// (levels 2, 1, 0 of eight rows y_b, b < k known) differs.  With X the eighth
// of the transform, P = sum_{j<k} a_j X^j, i = W[1], w = W[2], h = W[3] = i w
// (w^2 = i, h^2 = -i, h^3 = w), the first four rows give 4 u = 4 P mod X^4 - 1,
// the next two 2 v = 2 P mod X^2 - i, the seventh P(h); eliminating gives
//  k = 5: 4 (a0 - a4) = 4 y4 - w 4u1 - i 4u2 - h 4u3
//  k = 6: 4 (a_j - a_(j+4)) = 2 2v_j - i 4u_(j+2), j = 0, 1
//  k = 7: E = 4 (a1 - a5) = 2 2v1 - i 4u3, F = 4 y6 - h E - w 4u3,
//         8 (a0 - a4) = 2 2v0 + F, 8 (a2 - a6) = -i (2 2v0 - F).
// Rows 0 .. k-1 receive 16 a_j, twice what the full group's sums give: the
// transform's scale takes that into account.
template <int V, class Roots>
__device__ __forceinline__ void inv_truncated(Unit<3, V>& u, int k8, const Roots& itw, const Roots& ftw,
                                              const Prime& P) {
  const i32 p = P.p;
  const int2 i1 = ftw.one(1), w1 = ftw.one(2), h1 = ftw.one(3), ii = itw.one(1), wi = itw.one(2);
#pragma unroll
  for (int c = 0; c < V; ++c) {
    const i32 y0 = u.x[0][c], y1 = u.x[1][c], y2 = u.x[2][c], y3 = u.x[3][c], y4 = u.x[4][c], y5 = u.x[5][c];
    const i32 s0 = y0 + y1, d0 = y0 - y1, s1 = y2 + y3, d1 = mul_mod(y2 - y3, ii.x, ii.y, p);
    const i32 u0 = reduce(s0 + s1, P), u2 = reduce(s0 - s1, P), u1 = reduce(d0 + d1, P), u3 = reduce(d0 - d1, P);
    if (k8 == 5) {
      const i32 d = 4 * reduce(y4, P) - mul_mod(u1, w1.x, w1.y, p) - mul_mod(u2, i1.x, i1.y, p) -
                    mul_mod(u3, h1.x, h1.y, p);
      u.x[0][c] = 2 * (u0 + d);
      u.x[4][c] = 2 * (u0 - d);
      u.x[1][c] = 4 * u1;
      u.x[2][c] = 4 * u2;
      u.x[3][c] = 4 * u3;
    } else {
      const i32 v0 = reduce(y4 + y5, P), v1 = mul_mod(y4 - y5, wi.x, wi.y, p);
      const i32 e = 2 * v1 - mul_mod(u3, i1.x, i1.y, p);
      u.x[1][c] = 2 * (u1 + e);
      u.x[5][c] = 2 * (u1 - e);
      u.x[3][c] = 4 * u3;
      if (k8 == 6) {
        const i32 d = 2 * v0 - mul_mod(u2, i1.x, i1.y, p);
        u.x[0][c] = 2 * (u0 + d);
        u.x[4][c] = 2 * (u0 - d);
        u.x[2][c] = 4 * u2;
      } else {
        const i32 f = 4 * reduce(u.x[6][c], P) - mul_mod(e, h1.x, h1.y, p) - mul_mod(u3, w1.x, w1.y, p);
        const i32 g = mul_mod(2 * v0 - f, i1.x, i1.y, p);
        u.x[0][c] = 2 * u0 + 2 * v0 + f;
        u.x[4][c] = 2 * u0 - 2 * v0 - f;
        u.x[2][c] = 2 * u2 - g;
        u.x[6][c] = 2 * u2 + g;
      }
    }
  }
}

// Levels of a tile of R levels go in groups of at most three, one
// shared-memory exchange between groups: groups_of(R) of them, the longer
// ones first (forward order; the first one three levels from R = 3 on, for
// the truncated transforms).
constexpr int groups_of(int R) { return (R + 2) / 3; }
constexpr int group_size(int R, int g) {
  if (R == 4) return g == 0 ? 3 : 1;
  int left = R, k = 0;
  for (int i = 0; i <= g; ++i) {
    const int n = groups_of(R) - i;
    k = (left + n - 1) / n;
    left -= k;
  }
  return k;
}
constexpr int group_start(int R, int g) {
  int l = 0;
  for (int i = 0; i < g; ++i) l += group_size(R, i);
  return l;
}

// Word of (row, column) in a tile of C columns.  Strided tiles (32 columns or
// more) are dense: a 128-byte row takes every bank once.  Contiguous tiles
// (LEAF) are laid out for the units of the deepest group and for the block
// products, where lanes read the same word of neighbouring rows: rows of 8
// words with a row's length after every eight, longer rows with an eighth of
// their length (at least 16 bytes) after each.  A unit's rows are 2^nsub apart
// and their offsets from the first are the same for every unit.
template <int C, bool LEAF>
__device__ __forceinline__ constexpr u32 at(u32 row) {
  if (!LEAF) return row * C;
  if (C == 8) return row * C + (row >> 3) * C;
  return row * (C + (C == 16 ? 4 : C / 8));
}
template <int C, bool LEAF>
constexpr u32 tile_words32(int R) {
  const u32 rows = 1u << R;
  if (!LEAF) return rows * C;
  if (C == 8) return rows * C + (rows + 7) / 8 * C;
  return rows * (C + (C == 16 ? 4 : C / 8));
}
// Columns of a strided tile: 32 (128 bytes), more where few rows would leave
// the CTA with few units.
constexpr int col_width(int R) { return R >= 7 ? 32 : 4096 >> R; }

// ---- launch shapes ----

constexpr int at_least_warp(int threads) { return threads < 32 ? 32 : threads; }
// Threads of a strided pass's CTA: one unit of eight rows x four columns each.
constexpr int col_threads(int R) { return at_least_warp((col_width(R) / 4) << (R - 3)); }
constexpr int col_smem(int R) { return groups_of(R) > 1 ? (int)tile_words32<32, false>(R) * (col_width(R) / 32) * 4 : 0; }
// Registers: 64 a thread; tiles of up to 2^8 rows as many CTAs as that allows.
constexpr int col_blocks(int R) { return 1024 / col_threads(R) < 16 ? 1024 / col_threads(R) : 16; }

// One unit of eight rows x V columns a thread.
constexpr int fused_threads(int R, int LGM, int V) { return at_least_warp((1 << (R + LGM)) / (8 * V)); }
// Two tiles of 4096 words in shared memory let six CTAs share an SM: 768
// threads (80 registers) of four columns each, more of fewer columns; 640
// with the sums of longer blocks' products (96 registers).
constexpr int fused_blocks(int R, int LGM, int V) { 
  const int n = (LGM > 3 ? 640 : V == 4 ? 768 : 1024) / fused_threads(R, LGM, V);
  return n < 24 ? n : 24;
}

// Forward levels [0, R) of one tile of C columns x 2^R rows, block index ksb
// at its first level.  load(row, col) gives the V words from (row, col), store
// puts V finished words; between groups the words go
// through sm; thread tid of NT.  HALF: the rows from 2^(R-1) are zero, so level 0 copies.
// START: a reduction of the loaded words; LAST: one of the stored words.
// k8 < 8: only the rows of the first k8 eighths are finished and stored.
template <int R, int C, bool LEAF, int NT, int V, bool START, bool LAST, class Load, class Store, class Roots>
__device__ __forceinline__ void forward_tile(u32 tid, u32* sm, const Load& load, const Store& store, bool half_zero,
                                             const Roots& tw, u32 ksb, const Prime& P, bool start_red,
                                             int k8 = 8) {
  constexpr int G = groups_of(R);
  auto group = [&](auto gc) {
    constexpr int g = decltype(gc)::value;
    constexpr int K = group_size(R, g), l = group_start(R, g), nsub = R - l - K;
    constexpr u32 units = (u32)(C / V) << (R - K);
    if (g > 0) __syncthreads();
    const u32 todo = g == 0 ? units : units / 8 * k8;
    const int keep = g == 0 && K == 3 ? k8 : 8;
#pragma unroll 1
    for (u32 i = tid; i < todo; i += NT) {
      const u32 col = (i % (C / V)) * V, v = i / (C / V);
      const u32 rb = v >> nsub, row0 = (rb << (nsub + K)) + (v & ((1u << nsub) - 1));
      Unit<K, V> u;
      const u32 b = (ksb << l) + rb;
      u32* sp = sm + at<C, LEAF>(row0) + col;
      if constexpr (g == 0) {
        if (half_zero) {
#pragma unroll
          for (int m = 0; m < (1 << K) / 2; ++m) {
            u.set(m, load(row0 + ((u32)m << nsub), col));
            u.set(m + (1 << K) / 2, u.get(m));
          }
          fwd_levels<K, 1>(u, tw, b, P.p);
        } else {
#pragma unroll
          for (int m = 0; m < (1 << K); ++m) u.set(m, load(row0 + ((u32)m << nsub), col));
          if (START) {
            if (start_red) {
#pragma unroll
              for (int m = 0; m < (1 << K); ++m)
#pragma unroll
                for (int c = 0; c < V; ++c) u.x[m][c] = reduce(u.x[m][c], P);
            }
          }
          fwd_levels<K>(u, tw, b, P.p);
        }
      } else {
#pragma unroll
        for (int m = 0; m < (1 << K); ++m) u.set(m, ldv<V>(sp + at<C, LEAF>((u32)m << nsub)));
        fwd_levels<K>(u, tw, b, P.p);
      }
      if constexpr (g + 1 == G) {
#pragma unroll
        for (int m = 0; m < (1 << K); ++m) {
          if (LAST) {
#pragma unroll
            for (int c = 0; c < V; ++c) u.x[m][c] = reduce(u.x[m][c], P);
          }
          if (m < 5 || m < keep) store(row0 + ((u32)m << nsub), col, u.get(m));
        }
      } else {
#pragma unroll
        for (int m = 0; m < (1 << K); ++m)
          if (m < 5 || m < keep) stv<V>(sp + at<C, LEAF>((u32)m << nsub), u.get(m));
      }
    }
  };
  group(std::integral_constant<int, 0>{});
  if constexpr (G > 1) group(std::integral_constant<int, 1>{});
  if constexpr (G > 2) group(std::integral_constant<int, 2>{});
}

// Inverse levels R-1 .. 0 of one tile; the groups in the opposite order.
// last: the transform's last pass; its outputs are multiplied by the scale,
// which also makes them 0.75 p at most (k8 < 8, with the forward table ftw: a
// truncated transform's).
template <int R, int C, bool LEAF, int NT, int V, class Load, class Store, class Roots>
__device__ __forceinline__ void inverse_tile(u32 tid, u32* sm, const Load& load, const Store& store,
                                             const Roots& tw, u32 ksb, const Prime& P, bool last,
                                             int2 scale, int k8, const Roots& ftw) {
  constexpr int G = groups_of(R);
  auto group = [&](auto gc) {
    constexpr int g = decltype(gc)::value;
    constexpr int K = group_size(R, g), l = group_start(R, g), nsub = R - l - K;
    constexpr u32 units = (u32)(C / V) << (R - K);
    if (g + 1 < G) __syncthreads();
    const u32 todo = g == 0 ? units : units / 8 * k8;
    const int keep = g == 0 && K == 3 ? k8 : 8;
#pragma unroll 1
    for (u32 i = tid; i < todo; i += NT) {
      const u32 col = (i % (C / V)) * V, v = i / (C / V);
      const u32 rb = v >> nsub, row0 = (rb << (nsub + K)) + (v & ((1u << nsub) - 1));
      Unit<K, V> u;
      const u32 b = (ksb << l) + rb;
      u32* sp = sm + at<C, LEAF>(row0) + col;
#pragma unroll
      for (int m = 0; m < (1 << K); ++m) {
        if (m >= 5 && m >= keep) continue;
        if constexpr (g + 1 == G)
          u.set(m, load(row0 + ((u32)m << nsub), col));
        else
          u.set(m, ldv<V>(sp + at<C, LEAF>((u32)m << nsub)));
      }
      if (g == 0 && K == 3 && keep < 8) {
        if constexpr (g == 0 && K == 3) inv_truncated(u, keep, tw, ftw, P);
      } else {
        inv_levels<K>(u, tw, b, P.p);
      }
      if (g == 0 && last) {
#pragma unroll
        for (int m = 0; m < (1 << K); ++m)
#pragma unroll
          for (int c = 0; c < V; ++c)
            if (m < 5 || m < keep) u.x[m][c] = mul_mod(u.x[m][c], scale.x, scale.y, P.p);
      } else {
        inv_fold<K>(u, P);
      }
#pragma unroll
      for (int m = 0; m < (1 << K); ++m) {
        if (m >= 5 && m >= keep) continue;
        if constexpr (g == 0)
          store(row0 + ((u32)m << nsub), col, u.get(m));
        else
          stv<V>(sp + at<C, LEAF>((u32)m << nsub), u.get(m));
      }
    }
  };
  if constexpr (G > 2) group(std::integral_constant<int, 2>{});
  if constexpr (G > 1) group(std::integral_constant<int, 1>{});
  group(std::integral_constant<int, 0>{});
}

// V limbs from position pos as residues (zero at and beyond n).
template <int V>
__device__ __forceinline__ Words<V> limb_words(const u64* __restrict__ in, u64 n, u64 pos, bool vec, const Prime& P) {
  u64 x[V];
#pragma unroll
  for (int c = 0; c < V; ++c) x[c] = 0;
  if (V > 1 && vec && pos + V <= n) {
#pragma unroll
    for (int c = 0; c + 1 < V; c += 2) {
      const ulonglong2 t = __ldg(reinterpret_cast<const ulonglong2*>(in + pos + c));
      x[c] = t.x;
      x[c + 1] = t.y;
    }
  } else {
#pragma unroll
    for (int c = 0; c < V; ++c)
      if (pos + c < n) x[c] = __ldg(in + pos + c);
  }
  Words<V> w;
#pragma unroll
  for (int c = 0; c < V; ++c) w.v[c] = limb_residue(x[c], P);
  return w;
}

// The first pass of one operand: levels [0, R) from its limbs, columns
// [tile * C, tile * C + C) of every row of 2^(s-R).
template <int R, int C, int NT>
__device__ __forceinline__ void load_tile(u32* sm, const u64* __restrict__ in, u64 n, u32* res, int s, u32 tile,
                                          int prime, const int2* __restrict__ tab, u64 cap, int k8) {
  const Prime P = c_primes[prime];
  const int lg_s = s - R;
  u32* out = res + ((u64)prime << s) + (u64)tile * C;
  const bool vec = (reinterpret_cast<uintptr_t>(in) & 15) == 0;
  const u64 col0 = (u64)tile * C;
  forward_tile<R, C, false, NT, 4, false, false>(
      threadIdx.x, sm, [&](u32 row, u32 col) { return limb_words<4>(in, n, ((u64)row << lg_s) + col0 + col, vec, P); },
      [&](u32 row, u32 col, const Words<4>& w) { stv(out + ((u64)row << lg_s) + col, w); }, n <= (1ull << (s - 1)),
      GlobalRoots{tab + prime * cap}, 0, P, false, k8);
}

// Levels [lambda0, lambda0 + R) of residues in place: forward or inverse (tab:
// the inverse table, which follows the forward one).  k8: of the whole
// transform, for its last inverse pass only.
template <int R, int C, int NT, bool INV>
__device__ __forceinline__ void col_tile(u32* sm, u32* res, int s, int lambda0, u32 tile, int prime,
                                         const int2* __restrict__ tab, u64 cap, bool last = false,
                                         int2 scale = int2{}, int k8 = 8) {
  const Prime P = c_primes[prime];
  const int lg_s = s - lambda0 - R;
  const u32 per = (u32)((1ull << lg_s) / C);  // tiles a block
  const u32 ksb = tile / per;
  u32* g = res + ((u64)prime << s) + ((u64)ksb << (lg_s + R)) + (u64)(tile % per) * C;
  const GlobalRoots tw{tab + prime * cap};
  auto ld = [&](u32 row, u32 col) { return ldv<4>(g + ((u64)row << lg_s) + col); };
  auto st = [&](u32 row, u32 col, const Words<4>& w) { stv(g + ((u64)row << lg_s) + col, w); };
  if constexpr (INV)
    inverse_tile<R, C, false, NT, 4>(threadIdx.x, sm, ld, st, tw, ksb, P, last, scale, k8,
                                     GlobalRoots{tw.p - kPrimes * cap});
  else
    forward_tile<R, C, false, NT, 4, false, false>(threadIdx.x, sm, ld, st, false, tw, ksb, P, false);
}

// Products of polynomials of 8 coefficients by Karatsuba's method three levels
// deep: 27 multiply-adds instead of 64, at four cycles of the multiply pipe
// each.  Digit k (base 3) of a point's index takes the coefficients with bit k
// of their index clear (0), set (1) or both, added (2).  Sums over several
// products add up point by point and are interpolated once; 64-bit wrap-around
// on the way is harmless, since the coefficients themselves fit.
template <int N>
__device__ __forceinline__ void kara_points(const i32 (&x)[N], i32* e) {
  if constexpr (N == 1) {
    e[0] = x[0];
  } else {
    i32 lo[N / 2], hi[N / 2], both[N / 2];
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
      lo[i] = x[i];
      hi[i] = x[i + N / 2];
      both[i] = x[i] + x[i + N / 2];
    }
    constexpr int T = N == 8 ? 9 : N == 4 ? 3 : 1;
    kara_points<N / 2>(lo, e);
    kara_points<N / 2>(hi, e + T);
    kara_points<N / 2>(both, e + 2 * T);
  }
}
// The 2 N - 1 coefficients from the points' products.
template <int N>
__device__ __forceinline__ void kara_interpolate(const i64* u, i64 (&t)[2 * N - 1]) {
  if constexpr (N == 1) {
    t[0] = u[0];
  } else {
    constexpr int T = N == 8 ? 9 : N == 4 ? 3 : 1, H = N / 2;
    i64 lo[N - 1], hi[N - 1], both[N - 1];
    kara_interpolate<H>(u, lo);
    kara_interpolate<H>(u + T, hi);
    kara_interpolate<H>(u + 2 * T, both);
#pragma unroll
    for (int i = 0; i < 2 * N - 1; ++i) t[i] = (i < N - 1 ? lo[i] : 0) + (i >= N ? hi[i - N] : 0);
#pragma unroll
    for (int i = 0; i < N - 1; ++i) t[i + H] += both[i] - lo[i] - hi[i];
  }
}
// (sum t_i z^i) 2^-32 modulo z^8 - c, cr = c 2^32 mod p: the upper seven
// coefficients come down through a Montgomery step each and one multiply-add.
__device__ __forceinline__ void fold8(i64 (&t)[15], i32 cr, i32 (&o)[8], const Prime& P) {
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    if (j < 7) t[j] += (i64)mont(t[j + 8], P) * cr;
    o[j] = mont(t[j], P);
  }
}
// The constant c_b of block b, times 2^32: the roots' table holds it for even
// b, its negative for odd b.
template <class Roots>
__device__ __forceinline__ i32 block_constant(const Roots& tw, u32 b, const Prime& P) {
  const i32 c = tw.one(b >> 1).x;
  const i32 r = mul_mod(c, P.r, P.rp, P.p);
  return b & 1 ? -r : r;
}

// Products of the blocks of 8 coefficients of a tile: block row r of A times
// that of B modulo x^8 - c, times 2^-32, into sa.  A and B in shared memory (ga,
// gb nullptr), or finished words in global memory, where a thread's block is
// one 32-byte sector.  Words at most 0.75 p in magnitude: the sums of eight
// products, with the folded part, stay below 2^58.
template <int R, int NT, bool GA, bool GB, class Roots>
__device__ __forceinline__ void leaf_products8(u32* sa, const u32* sb, const u32* ga, const u32* gb, const Roots& tw,
                                               u32 ksb, const Prime& P, u32 rows) {
#pragma unroll 1
  for (u32 r = threadIdx.x; r < rows; r += NT) {
    const i32 cr = block_constant(tw, (ksb << R) + r, P);
    u32* pa = sa + at<8, true>(r);
    i64 u[27], t[15];
    {
      i32 x[8], ea[27], eb[27];
      auto words = [&](const u32* q) {
        const Words<4> w0 = ldv<4>(q), w1 = ldv<4>(q + 4);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          x[i] = w0.v[i];
          x[i + 4] = w1.v[i];
        }
      };
      words(GA ? ga + 8 * r : pa);
      kara_points(x, ea);
      words(GB ? gb + 8 * r : sb + at<8, true>(r));
      kara_points(x, eb);
#pragma unroll
      for (int i = 0; i < 27; ++i) u[i] = (i64)ea[i] * eb[i];
    }
    kara_interpolate<8>(u, t);
    i32 o[8];
    fold8(t, cr, o, P);
    stv(pa, Words<4>{{o[0], o[1], o[2], o[3]}});
    stv(pa + 4, Words<4>{{o[4], o[5], o[6], o[7]}});
  }
}

// The same for blocks of m = 8 G coefficients (transforms above 2^25), seen as
// polynomials of degree below G in x over Z_p[z] / (z^8 - c), z = x^G (word
// g + G i is the z^i coefficient of x^g): a thread forms one x^g of one block
// from G products of 8 coefficients each, with z b in the place of b where
// the power of x wraps.  One level of Karatsuba's method, 48 multiply-adds a
// product: its 21 sums leave room for five CTAs an SM, where the 27 sums of
// three levels take 114 registers (2^25 x 2^25 limbs: fused pass 3.02 ms at four
// CTAs, 2.73 so, 3.03 with 64 multiply-adds; 2^27 x 2^27: 19.2, 17.0, 17.5).  Results are written after every thread of the CTA has read the
// round's blocks.
template <int R, int LGM, int NT, class Roots>
__device__ __forceinline__ void leaf_products(u32* sa, const u32* sb, const Roots& tw, u32 ksb,
                                              const Prime& P) {
  constexpr int C = 1 << LGM, G = C / 8;
  constexpr u32 items = (u32)G << R;
  constexpr u32 rounds = (items + NT - 1) / NT;
#pragma unroll 1
  for (u32 it = 0; it < rounds; ++it) {
    const u32 q = it * NT + threadIdx.x;  // whole blocks a round: items of a block lie in one round
    const bool on = q < items;
    const u32 r = on ? q / G : 0, g = q % G, blk = (ksb << R) + r;
    int2 c = tw.one(blk >> 1);
    if (blk & 1) c = make_int2(-c.x, -c.y);
    i64 lo[7], hi[7], mid[7];  // products of the lower halves, the upper ones, the sums of both
#pragma unroll
    for (int i = 0; i < 7; ++i) lo[i] = hi[i] = mid[i] = 0;
    u32* pa = sa + at<C, true>(r);
    const u32* pb = sb + at<C, true>(r);
#pragma unroll 1
    for (int h = 0; h < G; ++h) {
      const u32 k = (g - h) % G;
      const bool wrap = (u32)h > g;
      i32 x[8], y[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        x[i] = (i32)pa[h + G * i];
        y[i] = (i32)pb[k + G * i];
      }
      const i32 top = mul_mod(y[7], c.x, c.y, P.p);
#pragma unroll
      for (int i = 7; i > 0; --i) y[i] = wrap ? y[i - 1] : y[i];
      y[0] = wrap ? top : y[0];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          lo[i + j] += (i64)x[i] * y[j];
          hi[i + j] += (i64)x[i + 4] * y[j + 4];
          mid[i + j] += (i64)(x[i] + x[i + 4]) * (y[j] + y[j + 4]);
        }
    }
    __syncthreads();  // these blocks have been read
    if (on) {
      i64 t[15];
      i32 o[8];
#pragma unroll
      for (int i = 0; i < 15; ++i) t[i] = (i < 7 ? lo[i] : 0) + (i >= 8 ? hi[i - 8] : 0);
#pragma unroll
      for (int i = 0; i < 7; ++i) t[i + 4] += mid[i] - lo[i] - hi[i];
      fold8(t, block_constant(tw, blk, P), o, P);
#pragma unroll
      for (int i = 0; i < 8; ++i) pa[g + G * i] = (u32)reduce(o[i], P);
    }
  }
}

// The last pass: tile `tile` (block index at the pass's first level, 2^R blocks
// of 2^LGM coefficients) of the operands forward, the blocks' products, and the
// first inverse levels, to out.
//  kAll: both operands forward (b nullptr: a square)
//  kReady: a forward; b's forward levels are done (FinishedWords)
//  kProduct: those of both are done
//  kForward: a's forward levels only, to out
//  kInverse: a's are done, and it is taken back alone, without a product
// Operands are residues after the strided passes, or, FIRST (transforms of one
// pass), limbs (na, nb of them); finished ones are words of at most 0.75 p.
// last: no strided inverse pass follows (scale, k8 as in inverse_tile).
// PAIR (FIRST, kAll): twice the threads, half of them an operand, and the
// 2^(R-1) roots of either direction that a one-pass transform needs copied to
// shared memory while the limbs are on their way: a lone short product waits
// on memory a third as often.
enum : int { kAll = 0, kReady = 1, kProduct = 2, kForward = 3, kInverse = 4 };
// Shared-memory tiles of a mode: finished operands are read from global memory
// where a block is a sector (LGM = 3).
constexpr int fused_tiles(int LGM, int mode) {
  return mode == kAll || (LGM > 3 && mode != kForward && mode != kInverse) ? 2 : 1;
}
template <int R, int LGM, int NT, int V, int MODE, bool FIRST, bool PAIR = false>
__device__ __forceinline__ void fused_tile(u32* sm, const void* a, u64 na, const void* b, u64 nb, u32* out, int s,
                                           u32 tile, int prime, const int2* __restrict__ tab,
                                           const int2* __restrict__ itab, u64 cap, bool reduce_in, bool last,
                                           int2 scale, int k8) {
  constexpr int C = 1 << LGM;
  constexpr u32 W = tile_words32<C, true>(R);
  const Prime P = c_primes[prime];
  const int2* const tw0 = tab + prime * cap;
  const int2* const itw0 = itab + prime * cap;
  const u64 off = ((u64)prime << s) + ((u64)tile << (R + LGM));
  u32* sa = sm;
  u32* sb = MODE == kAll && !b ? sm : sm + W;
  constexpr u32 kRoots = 1u << (R - 1);
  int2* const sroots = reinterpret_cast<int2*>(sm + 2 * W);
  typedef std::conditional_t<PAIR, SharedRoots, GlobalRoots> Roots;
  const Roots tw{PAIR ? sroots : tw0}, itw{PAIR ? sroots + kRoots : itw0};
  const u32 tid = PAIR ? threadIdx.x % NT : threadIdx.x;
  if constexpr (PAIR) {
    for (u32 i = threadIdx.x; i < 2 * kRoots; i += 2 * NT)
      sroots[i] = __ldg(i < kRoots ? tw0 + i : itw0 + (i - kRoots));
    __syncthreads();
  }
  auto to = [&](u32* t) { return [t](u32 row, u32 col, const Words<V>& w) { stv(t + at<C, true>(row) + col, w); }; };
  auto forward = [&](const void* src, u64 n, u32* t) {
    if constexpr (FIRST) {
      const u64* in = static_cast<const u64*>(src);
      const bool vec = (reinterpret_cast<uintptr_t>(in) & 15) == 0;
      forward_tile<R, C, true, NT, V, false, true>(
          tid, t, [&](u32 row, u32 col) { return limb_words<V>(in, n, (u64)row * C + col, vec, P); }, to(t),
          n <= (1ull << (s - 1)), tw, 0, P, false, k8);
    } else {
      const u32* in = static_cast<const u32*>(src) + off;
      forward_tile<R, C, true, NT, V, true, true>(
          tid, t, [&](u32 row, u32 col) { return ldv<V>(in + row * C + col); }, to(t), false, tw, tile, P, reduce_in);
    }
  };
  auto copy_in = [&](const void* src, u32* t) {
    const u32* in = static_cast<const u32*>(src) + off;
    for (u32 i = 4 * threadIdx.x; i < ((u32)C << R); i += 4 * NT) stv(t + at<C, true>(i / C) + i % C, ldv<4>(in + i));
  };
  if constexpr (PAIR) {
    const bool second = threadIdx.x >= NT;
    forward(second ? b : a, second ? nb : na, second ? sb : sa);
  } else if constexpr (MODE == kAll) {
    // one copy of the code for both operands
    const int operands = b ? 2 : 1;
#pragma unroll 1
    for (int op = 0; op < operands; ++op) forward(op ? b : a, op ? nb : na, op ? sb : sa);
  } else if constexpr (MODE != kProduct && MODE != kInverse) {
    forward(a, na, sa);
  } else if constexpr (LGM > 3 || MODE == kInverse) {
    copy_in(a, sa);
  }
  if constexpr (LGM > 3 && (MODE == kReady || MODE == kProduct)) copy_in(b, sb);
  __syncthreads();
  if constexpr (MODE == kForward) {
    u32* back = out + off;
    for (u32 i = 4 * threadIdx.x; i < ((u32)C << R); i += 4 * NT) stv(back + i, ldv<4>(sa + at<C, true>(i / C) + i % C));
  } else {
    if constexpr (MODE == kInverse) {
      // the words as they are
    } else if constexpr (LGM == 3)
      leaf_products8<R, PAIR ? 2 * NT : NT, MODE == kProduct, MODE != kAll>(sa, sb, static_cast<const u32*>(a) + off,
                                                            static_cast<const u32*>(b) + off, tw, tile, P,
                                                            FIRST && R >= 3 ? (u32)k8 << (R - 3) : 1u << R);
    else
      leaf_products<R, LGM, NT>(sa, sb, tw, tile, P);
    __syncthreads();
    u32* dst = out + off;
    inverse_tile<R, C, true, PAIR ? 2 * NT : NT, V>(
        threadIdx.x, sa, [&](u32 row, u32 col) { return ldv<V>(sa + at<C, true>(row) + col); },
        [&](u32 row, u32 col, const Words<V>& w) { stv(dst + row * C + col, w); }, itw, tile, P, last, scale, k8, tw);
  }
}

}  // namespace six
}  // namespace nn
