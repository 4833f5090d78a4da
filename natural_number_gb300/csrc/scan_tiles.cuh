// scan_tiles.cuh — tile-level device code of the multiword carry scan and its
// value producers, shared by the per-call kernels (carry.cu) and the batches'
// (batch.cu).  See carry.cu for the scheme.
#pragma once

#include "nn_device.cuh"
#include "nn_internal.h"
#include "six_tiles.cuh"

namespace nn {

constexpr u32 kFlagAggregate = 1, kFlagInclusive = 2;
constexpr int kSpinLimit = 1 << 22;

struct W3 {
  u64 w0, w1, w2;
};

// Multiword sums as carry chains (add.cc / addc, mad.lo.cc / madc): the carry
// travels in the condition code instead of a compare and a select per word.
// A chain lives inside one asm statement, the only place the code survives.

// a + b mod 2^192.
__device__ __forceinline__ W3 add_w3(W3 a, W3 b) {
  W3 r;
  asm("add.cc.u64 %0, %3, %6;\n\t"
      "addc.cc.u64 %1, %4, %7;\n\t"
      "addc.u64 %2, %5, %8;"
      : "=l"(r.w0), "=l"(r.w1), "=l"(r.w2)
      : "l"(a.w0), "l"(a.w1), "l"(a.w2), "l"(b.w0), "l"(b.w1), "l"(b.w2));
  return r;
}

// acc += x * y as one carry chain.
__device__ __forceinline__ void mac(W3& acc, u64 x, u64 y) {
  asm("mad.lo.cc.u64 %0, %3, %4, %0;\n\t"
      "madc.hi.cc.u64 %1, %3, %4, %1;\n\t"
      "addc.u64 %2, %2, 0;"
      : "+l"(acc.w0), "+l"(acc.w1), "+l"(acc.w2)
      : "l"(x), "l"(y));
}

// y[0..8) += a0 + a1 * 2^64 (a carry rippling through all eight words);
// returns the carry out of the top word.
__device__ __forceinline__ u64 add_ripple8(u64 (&y)[8], u64 a0, u64 a1) {
  u64 c;
  asm("add.cc.u64 %0, %0, %9;\n\t"
      "addc.cc.u64 %1, %1, %10;\n\t"
      "addc.cc.u64 %2, %2, 0;\n\t"
      "addc.cc.u64 %3, %3, 0;\n\t"
      "addc.cc.u64 %4, %4, 0;\n\t"
      "addc.cc.u64 %5, %5, 0;\n\t"
      "addc.cc.u64 %6, %6, 0;\n\t"
      "addc.cc.u64 %7, %7, 0;\n\t"
      "addc.u64 %8, 0, 0;"
      : "+l"(y[0]), "+l"(y[1]), "+l"(y[2]), "+l"(y[3]), "+l"(y[4]), "+l"(y[5]), "+l"(y[6]), "+l"(y[7]), "=l"(c)
      : "l"(a0), "l"(a1));
  return c;
}

// Garner: x = r0 + p0*u + p0*p1*v with u = (r1-r0)/p0 mod p1 and
// v = ((r2-r0)/p0 - u)/p1 mod p2; residues in [0,p) after the inverse.
struct CrtProducer {
  const u64* res;
  u64 L;
  u64 count;
  static constexpr bool kBulk = true;
  __device__ __forceinline__ W3 operator()(u64 k) const {
    if (k >= count) return W3{0, 0, 0};
    return garner(res[k], res[L + k], res[2 * L + k]);
  }
  // Eight consecutive positions from k0 (a multiple of 8) with 16-byte loads.
  __device__ __forceinline__ void bulk(u64 k0, W3 (&x)[kScanE]) const {
    if (k0 + kScanE > count) {
#pragma unroll
      for (int e = 0; e < kScanE; ++e) x[e] = (*this)(k0 + e);
      return;
    }
    u64 r[3][kScanE];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int e = 0; e < kScanE; e += 2) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(res + (u64)i * L + k0 + e);
        r[i][e] = v.x;
        r[i][e + 1] = v.y;
      }
#pragma unroll
    for (int e = 0; e < kScanE; ++e) x[e] = garner(r[0][e], r[1][e], r[2][e]);
  }
  __device__ __forceinline__ W3 garner(u64 x0, u64 x1, u64 x2) const {
    const PrimeSet& P = g_primes;
    constexpr u64 p0 = PrimeC<0>::p, p1 = PrimeC<1>::p, p2 = PrimeC<2>::p;
    const u64 d1 = x1 >= x0 ? x1 - x0 : x1 + p1 - x0;
    const u64 u = shoup_mul_c<1>(d1, P.inv01, P.inv01s);
    const u64 d2 = x2 >= x0 ? x2 - x0 : x2 + p2 - x0;
    const u64 t2 = shoup_mul_c<2>(d2, P.inv02, P.inv02s);
    const u64 e2 = t2 >= u ? t2 - u : t2 + p2 - u;
    const u64 v = shoup_mul_c<2>(e2, P.inv12, P.inv12s);
    // x0 + p0*u + (p01_lo + p01_hi*2^64)*v as one carry chain
    W3 r;
    asm("mad.lo.cc.u64 %0, %3, %4, %5;\n\t"
        "madc.hi.u64 %1, %3, %4, 0;\n\t"
        "mad.lo.cc.u64 %0, %6, %8, %0;\n\t"
        "madc.hi.cc.u64 %1, %6, %8, %1;\n\t"
        "madc.hi.u64 %2, %7, %8, 0;\n\t"
        "mad.lo.cc.u64 %1, %7, %8, %1;\n\t"
        "addc.u64 %2, %2, 0;"
        : "=l"(r.w0), "=l"(r.w1), "=l"(r.w2)
        : "l"(p0), "l"(u), "l"(x0), "l"(P.p01_lo), "l"(P.p01_hi), "l"(v));
    return r;
  }
};

// CRT of the six-prime residues (six_tiles.cuh), which the last inverse pass
// leaves multiplied by (M/p_i)^-1: with t_i any representative in (0, 4p), the
// coefficient is sum t_i (M/p_i) - q M for q = floor(sum t_i / p_i): it is
// below 2^160 (two overlapping pieces, up to 2^31 limbs each), under a quarter
// of M = 2^162.25, so a sum of 15-bit fractions tells q.  Column j of the sum
// adds the t_i times word j of M/p_i in 64 bits without carries (six terms
// below 2^61.2), then one pass propagates them; q M enters as q times 2^192 - M.
// 36 wide multiply-adds, none dependent on another before the columns, where
// Garner's mixed radix has fifteen dependent modular products.
struct SixWords {
  u32 w[6];
};
constexpr SixWords six_times(SixWords a, u32 b) {
  u64 c = 0;
  for (int i = 0; i < 6; ++i) {
    c += (u64)a.w[i] * b;
    a.w[i] = (u32)c;
    c >>= 32;
  }
  return a;
}
constexpr SixWords six_modulus_without(int skip) {  // the product of the primes but one (6: all)
  SixWords m{{1, 0, 0, 0, 0, 0}};
  for (int i = 0; i < six::kPrimes; ++i)
    if (i != skip) m = six_times(m, six::prime_of(i));
  return m;
}
constexpr SixWords six_negated(SixWords a) {
  u64 c = 1;
  for (int i = 0; i < 6; ++i) {
    c += (u32)~a.w[i];
    a.w[i] = (u32)c;
    c >>= 32;
  }
  return a;
}
template <int I>
__device__ __forceinline__ void six_crt_term(int y, u64 (&col)[6], u32& frac) {
  constexpr u32 p = six::prime_of(I);
  constexpr SixWords m = six_modulus_without(I);
  constexpr u32 f = (u32)(((1ull << 39) + p / 2) / p);
  const u32 t = (u32)y + 2 * p;  // |y| <= 1.5 p: two pieces' residues may have been added
  frac += (t >> 12) * f;  // t / p in units of 2^-27, within 2^-10
#pragma unroll
  for (int j = 0; j < 5; ++j) col[j] += (u64)t * m.w[j];
}
__device__ __forceinline__ W3 six_garner(const int (&y)[six::kPrimes]) {
  static_assert(six::kPrimes == 6);
  constexpr SixWords neg = six_negated(six_modulus_without(six::kPrimes));
  u64 col[6] = {0, 0, 0, 0, 0, 0};
  u32 frac = 1u << 24;  // an eighth: the coefficient's own fraction is below a quarter
  six_crt_term<0>(y[0], col, frac);
  six_crt_term<1>(y[1], col, frac);
  six_crt_term<2>(y[2], col, frac);
  six_crt_term<3>(y[3], col, frac);
  six_crt_term<4>(y[4], col, frac);
  six_crt_term<5>(y[5], col, frac);
  const u32 q = frac >> 27;
  u32 w[6];
  u64 c = 0;
#pragma unroll
  for (int j = 0; j < 6; ++j) {
    c += col[j] + (u64)q * neg.w[j];
    w[j] = (u32)c;
    c >>= 32;
  }
  return W3{(u64)w[1] << 32 | w[0], (u64)w[3] << 32 | w[2], (u64)w[5] << 32 | w[4]};
}
__device__ __forceinline__ void six_garner4(const int4 (&v)[six::kPrimes], W3 (&x)[kScanE], int e0) {
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    int y[six::kPrimes];
#pragma unroll
    for (int q = 0; q < six::kPrimes; ++q) y[q] = e == 0 ? v[q].x : e == 1 ? v[q].y : e == 2 ? v[q].z : v[q].w;
    x[e0 + e] = six_garner(y);
  }
}
// Zero at and beyond position count.
__device__ __forceinline__ void six_mask(W3 (&x)[kScanE], u64 k0, u64 count) {
  if (k0 + kScanE <= count) return;
#pragma unroll
  for (int e = 0; e < kScanE; ++e)
    if (k0 + e >= count) x[e] = W3{0, 0, 0};
}
// A position's six words, as loaded (fetch) and combined (finish) apart: the
// scan has the values before its tile in flight while it forms the tile's.
struct SixWordsAt {
  int y[six::kPrimes];
  bool in;
};
struct SixCrtProducer {
  const u32* res;  // [6][L]
  u64 L, count;
  static constexpr bool kBulk = true;
  typedef SixWordsAt Raw;
  __device__ __forceinline__ Raw fetch(u64 i) const {
    Raw r;
    r.in = i < count;
#pragma unroll
    for (int q = 0; q < six::kPrimes; ++q) r.y[q] = r.in ? (int)res[q * L + i] : 0;
    return r;
  }
  __device__ __forceinline__ W3 finish(const Raw& r) const { return r.in ? six_garner(r.y) : W3{0, 0, 0}; }
  __device__ __forceinline__ W3 operator()(u64 i) const { return finish(fetch(i)); }
  // Eight consecutive positions from k0 (a multiple of 8, at least one below
  // count: then all eight lie in the transform) with 16-byte loads.
  __device__ __forceinline__ void bulk(u64 k0, W3 (&x)[kScanE]) const {
    if (k0 >= count) {
#pragma unroll
      for (int e = 0; e < kScanE; ++e) x[e] = W3{0, 0, 0};
      return;
    }
#pragma unroll
    for (int e0 = 0; e0 < kScanE; e0 += 4) {
      int4 v[six::kPrimes];
#pragma unroll
      for (int q = 0; q < six::kPrimes; ++q) v[q] = *reinterpret_cast<const int4*>(res + q * L + k0 + e0);
      six_garner4(v, x, e0);
    }
    six_mask(x, k0, count);
  }
};

// A product split into pieces: the longer operand x (nx limbs) cut into P
// pieces of k limbs (the last one shorter), each multiplied by the shorter
// operand y (ny <= k + 1 limbs) through its own transform of L words, laid
// out [P][6][L].  Product coefficient j is the sum of coefficient j - i*k of
// piece i = floor(j/k) (the last piece for j beyond it) and coefficient
// j - (i-1)*k of piece i-1 when that is below k + ny - 1: at most two terms
// (k >= ny - 1), each below 2^160, so the sum fits three limbs.  k is a
// multiple of 8, so eight positions starting at a multiple of 8 lie in one
// piece.
struct PieceCrtProducer {
  const u32* res;
  u64 L, k, P, ny, count;
  static constexpr bool kBulk = true;
  typedef SixWordsAt Raw;
  __device__ __forceinline__ u64 piece_of(u64 j) const {
    const u64 i = j / k;
    return i < P ? i : P - 1;
  }
  __device__ __forceinline__ Raw fetch(u64 j) const {
    Raw w;
    w.in = j < count;
    const u64 i = w.in ? piece_of(j) : 0, r = w.in ? j - i * k : 0;
    const u32* c = res + i * six::kPrimes * L + r;
    const u32* b = c - six::kPrimes * L + k;  // the piece before, at r + k
    const bool ov = i > 0 && r + 1 < ny;
#pragma unroll
    for (int q = 0; q < six::kPrimes; ++q) {
      w.y[q] = (int)c[q * L];
      if (ov) w.y[q] += (int)b[q * L];
    }
    return w;
  }
  __device__ __forceinline__ W3 finish(const Raw& r) const { return r.in ? six_garner(r.y) : W3{0, 0, 0}; }
  __device__ __forceinline__ W3 operator()(u64 j) const { return finish(fetch(j)); }
  __device__ __forceinline__ void bulk(u64 k0, W3 (&x)[kScanE]) const {
    if (k0 >= count) {
#pragma unroll
      for (int e = 0; e < kScanE; ++e) x[e] = W3{0, 0, 0};
      return;
    }
    const u64 i = piece_of(k0), r = k0 - i * k;  // one piece for the eight positions
    const u32* c = res + i * six::kPrimes * L + r;
    const u32* b = c - six::kPrimes * L + k;
    const u64 ov = i > 0 && r + 1 < ny ? ny - 1 - r : 0;  // so many of them overlap
#pragma unroll
    for (int e0 = 0; e0 < kScanE; e0 += 4) {
      int4 v[six::kPrimes];
#pragma unroll
      for (int q = 0; q < six::kPrimes; ++q) v[q] = *reinterpret_cast<const int4*>(c + q * L + e0);
      if (ov > e0) {
#pragma unroll
        for (int q = 0; q < six::kPrimes; ++q) {
          const int4 w = *reinterpret_cast<const int4*>(b + q * L + e0);
          v[q].x += w.x;
          v[q].y += ov > e0 + 1 ? w.y : 0;
          v[q].z += ov > e0 + 2 ? w.z : 0;
          v[q].w += ov > e0 + 3 ? w.w : 0;
        }
      }
      six_garner4(v, x, e0);
    }
    six_mask(x, k0, count);
  }
};

// Column sums of a schoolbook product (asmMul1's column order, asmLinux.asm:188-278).
struct ColumnProducer {
  static constexpr bool kBulk = false;
  __device__ __forceinline__ void bulk(u64, W3 (&)[kScanE]) const {}
  const u64* a;
  u64 na;
  const u64* b;
  u64 nb;
  __device__ __forceinline__ W3 operator()(u64 k) const {
    W3 r{0, 0, 0};
    if (k + 1 >= na + nb) return r;
    const u64 lo = k >= nb ? k - nb + 1 : 0;
    const u64 hi = k < na - 1 ? k : na - 1;
    for (u64 i = lo; i <= hi; ++i) {
      const u64 x = a[i], y = b[k - i];
      const u64 pl = x * y, ph = mulhi(x, y);
      r.w0 += pl;
      const u64 c = r.w0 < pl;
      const u64 t = r.w1 + ph;
      r.w2 += t < ph;
      r.w1 = t + c;
      r.w2 += r.w1 < c;
    }
    return r;
  }
};

// The column sums of one scan tile's positions and of the kScanE positions
// before them (the scan reads those too) in shared memory, as three word
// arrays of TILE + kScanE: all NT threads at once, eight lanes a position,
// the partial sums meeting in three shuffle steps.  (With one thread forming
// its eight scan positions' sums in turn, a product of a few hundred limbs
// keeps a few dozen threads busy.)
template <u64 TILE>
struct SmemSumsProducer {
  static constexpr bool kBulk = true;
  const u64* s;
  u64 first;  // the position at s[0] (mod 2^64: tile 0's is -kScanE)
  u64 total;
  __device__ __forceinline__ W3 operator()(u64 k) const {
    if (k >= total) return W3{0, 0, 0};
    const u64 i = k - first;
    return W3{s[i], s[TILE + kScanE + i], s[2 * (TILE + kScanE) + i]};
  }
  __device__ __forceinline__ void bulk(u64 k0, W3 (&x)[kScanE]) const {
#pragma unroll
    for (int e = 0; e < kScanE; ++e) x[e] = (*this)(k0 + e);
  }
};
template <int NT, u64 TILE>
__device__ __forceinline__ void column_tile_sums(u64* sm, const ColumnProducer& J, u64 tile) {
  constexpr u32 kLanes = 8, kGroups = NT / kLanes;
  const u64 size = J.na + J.nb;
  const long long first = (long long)(tile * TILE) - kScanE;
  const u64 end = min(size, (tile + 1) * TILE);
  const u32 npos = (u32)((long long)end - first);  // at most TILE + kScanE
  const u32 g = threadIdx.x / kLanes, j = threadIdx.x % kLanes;
  const u32 rounds = (npos + kGroups - 1) / kGroups;  // the same for every thread
  for (u32 r = 0; r < rounds; ++r) {
    const u32 q = r * kGroups + g;
    const long long p = first + q;
    W3 acc{0, 0, 0};
    if (q < npos && p >= 0 && (u64)p + 1 < size) {
      const u64 k = (u64)p;
      const u64 lo = k >= J.nb ? k - J.nb + 1 : 0;
      const u64 hi = k < J.na - 1 ? k : J.na - 1;
      for (u64 i = lo + j; i <= hi; i += kLanes) {
        const u64 x = J.a[i], y = J.b[k - i];
        mac(acc, x, y);
      }
    }
#pragma unroll
    for (u32 d = kLanes / 2; d >= 1; d >>= 1) {  // every lane of the warp takes part
      const W3 o{__shfl_down_sync(0xffffffffu, acc.w0, d, kLanes), __shfl_down_sync(0xffffffffu, acc.w1, d, kLanes),
                 __shfl_down_sync(0xffffffffu, acc.w2, d, kLanes)};
      acc = add_w3(acc, o);
    }
    if (j == 0 && q < npos) {
      sm[q] = acc.w0;
      sm[TILE + kScanE + q] = acc.w1;
      sm[2 * (TILE + kScanE) + q] = acc.w2;
    }
  }
}

// Limbs of x * B^shift at positions k0 .. k0 + 7 (zero outside x), a thread's
// share of a sum: 16-byte loads from the first 16-byte boundary on.
__device__ __forceinline__ void eight_limbs(u64 (&v)[kScanE], const u64* x, u64 n, u64 shift, u64 k0) {
  if (k0 >= shift && k0 - shift + kScanE <= n) {
    const u64* p = x + (k0 - shift);
    const int odd = (int)((reinterpret_cast<uintptr_t>(p) >> 3) & 1);
    if (odd) {
      v[0] = p[0];
#pragma unroll
      for (int e = 1; e + 1 < kScanE; e += 2) {
        const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(p + e);
        v[e] = t.x;
        v[e + 1] = t.y;
      }
      v[kScanE - 1] = p[kScanE - 1];
    } else {
#pragma unroll
      for (int e = 0; e < kScanE; e += 2) {
        const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(p + e);
        v[e] = t.x;
        v[e + 1] = t.y;
      }
    }
    return;
  }
#pragma unroll
  for (int e = 0; e < kScanE; ++e) {
    const u64 k = k0 + e;
    v[e] = k >= shift && k - shift < n ? x[k - shift] : 0;
  }
}

// x[k] + y[k - shift] (two words).
struct AddProducer {
  static constexpr bool kBulk = true;
  const u64* x;
  u64 nx;
  const u64* y;
  u64 ny;
  u64 shift;
  __device__ __forceinline__ W3 operator()(u64 k) const {
    const u64 a = k < nx ? x[k] : 0;
    const u64 b = (k >= shift && k - shift < ny) ? y[k - shift] : 0;
    const u64 s = a + b;
    return W3{s, (u64)(s < a), 0};
  }
  __device__ __forceinline__ void bulk(u64 k0, W3 (&w)[kScanE]) const {
    u64 a[kScanE], b[kScanE];
    eight_limbs(a, x, nx, 0, k0);
    eight_limbs(b, y, ny, shift, k0);
#pragma unroll
    for (int e = 0; e < kScanE; ++e) {
      const u64 s = a[e] + b[e];
      w[e] = W3{s, (u64)(s < a[e]), 0};
    }
  }
};

// x*B^xs + y*B^ys (add) or, as x*B^xs + ~(y*B^ys) + cin over `count`
// positions (sub), x*B^xs - y*B^ys - (1 - cin): with the scan run over
// count + 1 positions, the extra limb receives the carry out, which for a
// subtraction is 1 exactly when no borrow occurred.  Zero beyond count.
// With `flip` set, a nonzero *flip (a limb in device memory, read by every
// thread) swaps add and subtract, so a sign known only on the device picks
// the operation without a round trip to the host.
struct LinProducer {
  static constexpr bool kBulk = true;
  const u64* x;
  u64 nx, xs;
  const u64* y;
  u64 ny, ys;
  u64 count;
  int sub, cin;
  const u64* flip;
  __device__ __forceinline__ W3 operator()(u64 k) const {
    if (k >= count) return W3{0, 0, 0};
    const u64 a = (k >= xs && k - xs < nx) ? x[k - xs] : 0;
    u64 b = (k >= ys && k - ys < ny) ? y[k - ys] : 0;
    u64 c = 0;
    if (sub ^ (flip != nullptr && __ldcg(flip) != 0)) {
      b = ~b;
      c = k == 0 ? (u64)cin : 0;
    }
    const u64 s = a + b;
    const u64 c1 = s < a;
    const u64 s2 = s + c;
    const u64 c2 = s2 < s;
    return W3{s2, c1 + c2, 0};
  }
  __device__ __forceinline__ void bulk(u64 k0, W3 (&w)[kScanE]) const {
    u64 a[kScanE], b[kScanE];
    eight_limbs(a, x, nx, xs, k0);
    eight_limbs(b, y, ny, ys, k0);
    const bool neg = sub ^ (flip != nullptr && __ldcg(flip) != 0);
#pragma unroll
    for (int e = 0; e < kScanE; ++e) {
      const u64 v = neg ? ~b[e] : b[e];
      const u64 c = neg && k0 + e == 0 ? (u64)cin : 0;
      const u64 s = a[e] + v, s2 = s + c;
      w[e] = k0 + e < count ? W3{s2, (u64)(s < a[e]) + (u64)(s2 < s), 0} : W3{0, 0, 0};
    }
  }
};

__device__ __forceinline__ u32 flag_load(const u32* f) {
  u32 v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(f) : "memory");
  return v;
}
__device__ __forceinline__ void flag_store(u32* f, u32 v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(f), "r"(v) : "memory");
}
// Polls *f until it is nonzero, at most `limit` times; 0 means the wait gave up.
__device__ __forceinline__ u32 wait_flag(const u32* f, int limit) {
  u32 v;
  int spins = 0;
  while ((v = flag_load(f)) == 0) {
    if (++spins > limit) break;
    __nanosleep(32);
  }
  return v;
}

// One tile of the scan over positions [0, total): limbs below out_limit go to
// out, the rest to side.
// kScanLookback: the tile takes its carry-in from its predecessors' status words
// (decoupled lookback); tiles of one scan must then start in increasing order
// (their predecessors already running), which the callers guarantee.
// kScanRecord: the tile takes carry-in 0 and records in flags[tile] (when given) its
// carry out for carry-in 0 (bit 0, generate) and whether a carry-in would pass
// straight through (bit 1, propagate: every limb all ones); a later step
// resolves the one-bit carries between tiles (carry.cu).
// The scan's shared scratch: one block per kernel, whatever producers its
// scan_tile instances take (a function's __shared__ variables exist once per
// CTA, while each instance of a template would get its own).
template <int NT>
struct ScanShared {
  u64 h0[NT], h1[NT];
  u32 wg[NT / 32], wp[NT / 32];
  u32 cin, bits;
  u64 x[kScanE][3];
};
template <int NT>
__device__ __forceinline__ ScanShared<NT>& scan_shared() {
  __shared__ ScanShared<NT> sh;
  return sh;
}

// How a tile learns its carry-in: later (record), by the lookback, or from the
// other tiles of its cluster.
enum : int { kScanRecord = 0, kScanLookback = 1, kScanCluster = 2 };

// All threads of all CTAs of the cluster arrive; what they wrote to shared
// memory before is visible to the others after.
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// The value at `local` in the shared memory of the cluster's CTA `rank`.
__device__ __forceinline__ u64 cluster_load64(const u64* local, u32 rank) {
  u64 v;
  asm volatile(
      "{\n\t.reg .u32 a;\n\tmapa.shared::cluster.u32 a, %1, %2;\n\tld.shared::cluster.u64 %0, [a];\n\t}"
      : "=l"(v)
      : "r"((u32)__cvta_generic_to_shared(local)), "r"(rank)
      : "memory");
  return v;
}
__device__ __forceinline__ u32 cluster_load32(const u32* local, u32 rank) {
  u32 v;
  asm volatile(
      "{\n\t.reg .u32 a;\n\tmapa.shared::cluster.u32 a, %1, %2;\n\tld.shared::cluster.u32 %0, [a];\n\t}"
      : "=r"(v)
      : "r"((u32)__cvta_generic_to_shared(local)), "r"(rank)
      : "memory");
  return v;
}

// kScanCluster: the scan's tiles are the CTAs of one cluster, tile = rank (at
// most 16).  A tile takes the overflow into its first position from the last
// thread of the tile before, and its carry-in from all earlier tiles' bits,
// both through distributed shared memory: no status words, no polling, and no
// values formed twice.  The caller ends with cluster_sync(), so that no CTA
// leaves while another reads its shared memory.
// NT: threads of the CTA.  TILE: positions of a tile, NT * kScanE at most;
// with fewer, the threads beyond them pass carries on unchanged.
template <class Prod, int MODE = kScanLookback, int NT = kScanThreads, u64 TILE = (u64)NT * kScanE>
__device__ __forceinline__ void scan_tile(const Prod& prod, u64 tile, u64 total, u64* out, u64 out_limit, u64* side,
                                          u32* flags, u32* err) {
  constexpr int E = kScanE;
  constexpr u64 kTile = TILE;
  static_assert(TILE % E == 0 && TILE <= (u64)NT * E);
  ScanShared<NT>& sh = scan_shared<NT>();
  u64* const s_h0 = sh.h0;
  u64* const s_h1 = sh.h1;
  u32* const s_wg = sh.wg;
  u32* const s_wp = sh.wp;
  u32& s_cin = sh.cin;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool on = TILE == (u64)NT * E || (u64)tid * E < TILE;
  const u64 k0 = tile * kTile + (u64)tid * E;

  u64 y[E];
  u64 c0 = 0, c1 = 0;
  W3 xs[E];
  // The E positions before this tile (below): their loads go out first.
  constexpr bool kSplit = requires { typename Prod::Raw; };
  typedef decltype([] {
    if constexpr (kSplit)
      return typename Prod::Raw{};
    else
      return W3{};
  }()) Before;
  Before before{};
  const bool preceding = MODE != kScanCluster && warp == 0 && lane < E && tile != 0;
  if constexpr (kSplit)
    if (preceding) before = prod.fetch(tile * kTile - E + lane);
  if (Prod::kBulk && on && k0 < total) {
    prod.bulk(k0, xs);
  } else {
#pragma unroll
    for (int e = 0; e < E; ++e) xs[e] = on && k0 + e < total ? prod(k0 + e) : W3{0, 0, 0};
  }
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const W3 t = add_w3(xs[e], W3{c0, c1, 0});
    y[e] = t.w0;
    c0 = t.w1;
    c1 = t.w2;
  }
  s_h0[tid] = c0;
  s_h1[tid] = c1;
  // Overflow of the E positions before this tile: lanes 0..E-1 of warp 0
  // produce one value each, thread 0 chains them.
  u64(&s_x)[E][3] = sh.x;
  if (MODE != kScanCluster && warp == 0) {
    if (preceding) {
      W3 x;
      if constexpr (kSplit)
        x = prod.finish(before);
      else
        x = prod(tile * kTile - E + lane);
      s_x[lane][0] = x.w0;
      s_x[lane][1] = x.w1;
      s_x[lane][2] = x.w2;
    }
    __syncwarp();
  }
  u64 hp0 = 0, hp1 = 0;
  if (MODE != kScanCluster && tid == 0 && tile != 0) {
    u64 d0 = 0, d1 = 0;
    for (int e = 0; e < E; ++e) {
      const W3 t = add_w3(W3{s_x[e][0], s_x[e][1], s_x[e][2]}, W3{d0, d1, 0});
      d0 = t.w1;
      d1 = t.w2;
    }
    hp0 = d0;
    hp1 = d1;
  }
  if constexpr (MODE == kScanCluster) {
    cluster_sync();
    if (tid == 0 && tile != 0) {
      hp0 = cluster_load64(s_h0 + TILE / E - 1, (u32)tile - 1);
      hp1 = cluster_load64(s_h1 + TILE / E - 1, (u32)tile - 1);
    }
  } else {
    __syncthreads();
  }
  if (tid > 0 && on) {
    hp0 = s_h0[tid - 1];
    hp1 = s_h1[tid - 1];
  }
  // u_t = lo_t + H_{t-1}; the carry out is the generate bit
  static_assert(E == 8, "the carry chains take eight limbs a thread");
  const u32 g = (u32)add_ripple8(y, hp0, hp1);
  u64 all = y[0];
#pragma unroll
  for (int e = 1; e < E; ++e) all &= y[e];
  const u32 pr = !on | ((all == ~0ull) & !g);

  const u32 G = __ballot_sync(0xffffffffu, g);
  const u32 GP = __ballot_sync(0xffffffffu, g | pr);
  if (lane == 0) {
    const u64 s0 = (u64)G + GP, s1 = (u64)G + GP + 1;
    s_wg[warp] = (u32)(s0 >> 32);
    s_wp[warp] = (u32)(s1 >> 32) & ~(u32)(s0 >> 32);
  }
  __syncthreads();
  if (tid == 0) {
    u32 c_if0 = 0, c_if1 = 1;
    for (int w = 0; w < NT / 32; ++w) {
      c_if0 = s_wg[w] | (s_wp[w] & c_if0);
      c_if1 = s_wg[w] | (s_wp[w] & c_if1);
    }
    const u32 tg = c_if0, tp = c_if1 & !c_if0;
    u32 cin = 0;
    if (MODE == kScanCluster) {
      sh.bits = tg | (tp << 1);
    } else if (MODE == kScanRecord) {
      if (flags) flags[tile] = tg | (tp << 1);
    } else if (tile > 0) {
      flag_store(&flags[tile], kFlagAggregate | (tg << 2) | (tp << 3));
      long long j = (long long)tile - 1;
      for (;;) {
        if (j < 0) {
          cin = 0;
          break;
        }
        const u32 f = wait_flag(&flags[j], kSpinLimit);
        if (f == 0) {
          atomicExch(err, 1u);
          cin = 0;
          break;
        }
        if (f & kFlagInclusive) {
          cin = (f >> 2) & 1;
          break;
        }
        if ((f >> 2) & 1) {  // predecessor generates
          cin = 1;
          break;
        }
        if (!((f >> 3) & 1)) {  // predecessor kills
          cin = 0;
          break;
        }
        --j;  // predecessor propagates: look further back
      }
    }
    if (MODE == kScanLookback) flag_store(&flags[tile], kFlagInclusive | ((tg | (tp & cin)) << 2));
    s_cin = cin;
  }
  if constexpr (MODE == kScanCluster) {
    cluster_sync();
    if (warp == 0) {
      const u32 f = (u64)lane < tile ? cluster_load32(&sh.bits, lane) : 0;
      const u32 g1 = __ballot_sync(0xffffffffu, f & 1), gp = __ballot_sync(0xffffffffu, f & 3);
      if (lane == 0) s_cin = ((g1 + gp) ^ g1 ^ gp) >> tile & 1;
    }
  }
  __syncthreads();
  u32 wc = s_cin;
  for (int w = 0; w < warp; ++w) wc = s_wg[w] | (s_wp[w] & wc);
  const u64 sum = (u64)G + GP + wc;
  const u32 cin_bits = (u32)sum ^ G ^ GP;
  add_ripple8(y, (cin_bits >> lane) & 1, 0);  // its carry out is the next thread's carry-in, counted above
  if (!on) return;
  if (k0 + E <= out_limit && k0 + E <= total && !(reinterpret_cast<uintptr_t>(out) & 15)) {
#pragma unroll
    for (int e = 0; e < E; e += 2) *reinterpret_cast<ulonglong2*>(out + k0 + e) = make_ulonglong2(y[e], y[e + 1]);
    return;
  }
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const u64 k = k0 + e;
    if (k < out_limit)
      out[k] = y[e];
    else if (k < total)
      side[k - out_limit] = y[e];
  }
}

}  // namespace nn
