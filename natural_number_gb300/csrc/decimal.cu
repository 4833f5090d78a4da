// decimal.cu — the decimal digits of many short naturals at once: the leaves
// of the split tree of _format_dec (natural.h:994-1011).
//
// The reference splits each value down to 10^18-sized leaves (_dec_split,
// natural.h:953-967; the last split is div_base by 10^18, natural.h:566-573)
// and prints each leaf as 18 zero-padded digits (the first one unpadded).
// The decimal digits of a value are unique, so a node of the tree at any
// level has exactly one digit string of its width; here one CTA takes one
// node and peels off its 18-digit groups from the low end by repeated exact
// division by 10^18, which is div_base's step applied 2^(i+1) times.
//
// A division's remainder chain runs from the top limb down, one limb after
// the other, and the next division's chain may follow one limb behind it.  So
// the CTA's lanes hold the node in segments, the top one in lane 0, and work
// as a pipeline: at step t lane L takes the remainder of division t - L from
// the lane above, divides its segment by 10^18 with it and hands its own
// remainder down.  Each division so costs its limbs' two-by-one divisions and
// nothing else (dec_groups_kernel).
//
// Layout: node k's len[k] limbs at nodes[k]; its digits go to out[k * width,
// (k + 1) * width), width = 18 * groups, most significant group first.
#include <cuda_runtime.h>

#include "nn_device.cuh"
#include "nn_internal.h"

#include <algorithm>

namespace nn {

namespace {

constexpr u64 kGroup = 1000000000000000000ull;  // 10^18 (dec_base_0)
constexpr int kNorm = 4;                        // leading zero bits of 10^18
constexpr u64 kGroupNorm = kGroup << kNorm;     // top bit set

// Division of the two-word value (u1, u0), u1 < d, by a normalised divisor d
// with its precomputed reciprocal v = floor((2^128 - 1) / d) - 2^64: the
// two-by-one division of Moller and Granlund, "Improved division by
// invariant integers" (IEEE Trans. Computers 60(2), 2011), Algorithm 4.
__device__ __forceinline__ u64 div_2by1(u64 u1, u64 u0, u64 d, u64 v, u64& r) {
  const u64 p_lo = v * u1;
  const u64 p_hi = __umul64hi(v, u1);
  u64 q0 = p_lo + u0;
  u64 q1 = p_hi + u1 + (q0 < p_lo ? 1 : 0);
  q1 += 1;
  u64 rr = u0 - q1 * d;
  if (rr > q0) {
    q1 -= 1;
    rr += d;
  }
  if (rr >= d) {
    q1 += 1;
    rr -= d;
  }
  r = rr;
  return q1;
}

// The 18 digits of x < 10^18, zero-padded, as nine 2-byte stores (o even).
__device__ __forceinline__ void put18(char* o, u64 x) {
  u32 hi = (u32)(x / 1000000000ull);
  u32 lo = (u32)(x - (u64)hi * 1000000000ull);
  unsigned char d[18];
#pragma unroll
  for (int t = 8; t >= 0; --t) {
    d[9 + t] = (unsigned char)('0' + lo % 10);
    lo /= 10;
    d[t] = (unsigned char)('0' + hi % 10);
    hi /= 10;
  }
  unsigned short* o2 = reinterpret_cast<unsigned short*>(o);
#pragma unroll
  for (int t = 0; t < 9; ++t) o2[t] = (unsigned short)(d[2 * t] | (d[2 * t + 1] << 8));
}

// One CTA a node, `blockDim.x` lanes; lane L's segment of at most `seg` limbs
// stands in shared memory from limb L * (seg | 1) on (an odd stride: lanes in
// different banks).  From lane to lane remainders go by shuffle, from warp to
// warp through a ring in shared memory that a barrier every kDecStep steps
// covers: warp w runs 32 + kDecStep steps behind the warp above, so that it
// reads a remainder at least one barrier after it was written.  The last lane
// leaves its remainders, the groups, in a ring too; once a barrier the last
// warp writes kDecStep of them as digits, a lane each.
//
// The quotients get shorter from the top: a warp whose limbs and remainders
// are all zero, and the warp above it for two barriers, leaves its divisions
// out.
//
// What bounds it: the 64-bit multiplies of the two-by-one divisions, about 300
// cycles a limb and step with three warps a scheduler.  420 nodes of 480 limbs
// (512 groups each): 0.45 ms; with one warp a node, every division split over
// its lanes by a scan of remainder maps, 1.2 ms.
constexpr int kDecStep = 16, kDecRing = 64, kDecMaxWarps = 16;
constexpr u64 kDecMaxLimbs = 8192;
// Shared memory of a node of `limbs` in the lanes of `warps`.
constexpr int dec_smem(u64 warps, u64 limbs) {
  return (int)(32 * warps * ((limbs + 32 * warps - 1) / (32 * warps) | 1) * 8);
}
__global__ void __launch_bounds__(32 * kDecMaxWarps) dec_groups_kernel(const u64* const* __restrict__ nodes,
                                                                       const u32* __restrict__ len, u32 groups, u64 v,
                                                                       char* out) {
  extern __shared__ u64 node_sm[];
  __shared__ u64 ring[kDecMaxWarps][kDecRing];
  __shared__ u32 idle[2][kDecMaxWarps];
  const int L = threadIdx.x, lane = L & 31, w = L >> 5, warps = (int)(blockDim.x >> 5);
  const u32 m = len[blockIdx.x], lanes = blockDim.x, seg = (m + lanes - 1) / lanes;
  const u32 hi = m - min(m, L * seg), n = min(hi, seg);  // limbs [hi - n, hi)
  u64* a = node_sm + (u64)L * (seg | 1);
  u64 any = 0;
  for (u32 j = 0; j < n; ++j) {
    a[j] = nodes[blockIdx.x][hi - 1 - j];  // top limb first
    any |= a[j];
  }
  char* o = out + (u64)blockIdx.x * groups * 18;
  const int lag = w * (32 + kDecStep) + lane, steps = (int)groups + (warps - 1) * (32 + kDecStep) + 31;
  u64 rn = 0;            // this lane's last remainder, times 2^kNorm
  u32 dead = 0;          // barriers since which this warp holds only zeros
  for (int t0 = 0; t0 < steps; t0 += kDecStep) {
    for (int t = t0; t < t0 + kDecStep; ++t) {
      const int g = t - lag;
      const bool on = g >= 0 && g < (int)groups;
      u64 r = __shfl_up_sync(0xffffffffu, rn, 1);
      if (lane == 0) r = w > 0 && on ? ring[w - 1][g % kDecRing] : 0;
      if (dead == 0 && on) {
        any = 0;
        for (u32 j = 0; j < n; ++j) {
          const u64 x = a[j];
          const u64 q = div_2by1(r | (x >> (64 - kNorm)), x << kNorm, kGroupNorm, v, r);
          a[j] = q;
          any |= q;
        }
        rn = r;
      }
      if (lane == 31 && on) ring[w][g % kDecRing] = rn;
    }
    const bool zero = __all_sync(0xffffffffu, any == 0 && rn == 0);
    const int parity = t0 / kDecStep & 1;
    if (lane == 0) idle[parity][w] = dead;
    __syncthreads();
    if (zero && (w == 0 || idle[parity][w - 1] >= 2)) ++dead;
    if (w == warps - 1 && lane < kDecStep) {
      const int g = t0 + lane - (warps - 1) * (32 + kDecStep) - 31;
      if (g >= 0 && g < (int)groups) put18(o + (u64)(groups - 1 - g) * 18, ring[w][g % kDecRing] >> kNorm);
    }
  }
}

// out = in >> shift bits (n_out limbs, in read as zero past n_in): block
// (x, y) covers limbs [x * 4096, x * 4096 + 4096) of job y.
__global__ void __launch_bounds__(256) shr_batch_kernel(const ShrJob* __restrict__ jobs) {
  const ShrJob J = jobs[blockIdx.y];
  const u64 ls = J.shift >> 6;
  const u32 bs = (u32)(J.shift & 63);
  for (u64 t = (u64)blockIdx.x * kShrChunk + threadIdx.x; t < J.n_out && t < (u64)(blockIdx.x + 1) * kShrChunk;
       t += blockDim.x) {
    const u64 i = t + ls;
    const u64 a = i < J.n_in ? J.in[i] : 0, b = i + 1 < J.n_in ? J.in[i + 1] : 0;
    J.out[t] = bs ? (a >> bs) | (b << (64 - bs)) : a;
  }
}

// One warp: x (nx limbs) against y (ny limbs): -1, 0 or 1.
__device__ int warp_cmp(const u64* x, u64 nx, const u64* y, u64 ny, u32 lane) {
  const u64 n = nx > ny ? nx : ny;
  for (u64 top = (n + 31) & ~31ull; top > 0; top -= 32) {
    const u64 k = top - 32 + lane;
    const u64 a = k < nx ? x[k] : 0, b = k < ny ? y[k] : 0;
    const u32 d = __ballot_sync(0xffffffffu, a != b);
    if (d) {
      const int hl = 31 - __clz(d);
      const int gt = __shfl_sync(0xffffffffu, a > b ? 1 : 0, hl);
      return gt ? 1 : -1;
    }
  }
  return 0;
}

// One warp: x (n limbs) += y (or -= y with `sub`), carries by ballots; past
// y's limbs the walk ends once no carry (borrow) is left.
__device__ void warp_addsub(u64* x, u64 n, const u64* y, u64 ny, bool sub, u32 lane) {
  const u64 flip = sub ? ~0ull : 0;
  const u32 idle = sub ? 1 : 0;  // the carry word when nothing is pending
  u32 carry = idle;
  for (u64 base = 0; base < n; base += 32) {
    if (base >= ny && carry == idle) break;
    const u64 k = base + lane;
    const u64 a = k < n ? x[k] : 0, b = (k < ny ? y[k] : 0) ^ flip;
    const u64 sum = a + b;
    const u32 G = __ballot_sync(0xffffffffu, sum < a), GP = __ballot_sync(0xffffffffu, sum < a || sum == ~0ull);
    const u64 t = (u64)G + GP + carry;
    if (k < n) x[k] = sum + ((((u32)t ^ G ^ GP) >> lane) & 1);
    carry = (u32)(t >> 32);
  }
}

// The split's correction (natural.h:962-965): while lo >= base, hi += 1 and
// lo -= base, at most kMaxFix times (an error otherwise); zero[k] = hi == 0.
constexpr int kMaxFix = 8;
__global__ void __launch_bounds__(256) dec_fix_kernel(const DecFixJob* __restrict__ jobs, u64 m, const u64* base,
                                                      u64 nb, u32* zero, u32* err) {
  const u64 k = ((u64)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const u32 lane = threadIdx.x & 31;
  if (k >= m) return;  // whole warps leave together
  const DecFixJob J = jobs[k];
  const u64 one = 1;
  int it = 0;
  for (; it < kMaxFix && warp_cmp(J.lo, J.n_lo, base, nb, lane) >= 0; ++it) {
    warp_addsub(J.lo, J.n_lo, base, nb, true, lane);
    __syncwarp();
    warp_addsub(J.hi, J.n_hi, &one, 1, false, lane);
    __syncwarp();
  }
  if (it == kMaxFix && lane == 0) atomicExch(err, 1u);
  // hi == 0: the walk ends at the first nonzero limb (within the first 32
  // limbs but for a zero or nearly zero hi)
  u32 nz = 0;
  for (u64 i0 = 0; i0 < J.n_hi && !nz; i0 += 32) {
    const u64 i = i0 + lane;
    nz = __any_sync(0xffffffffu, i < J.n_hi && J.hi[i] != 0);
  }
  if (lane == 0) zero[k] = !nz;
}

__global__ void __launch_bounds__(256) dec_need_kernel(const DecFixJob* __restrict__ jobs, u64 m, const u64* base,
                                                       u64 nb, u32* need) {
  const u64 k = ((u64)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const u32 lane = threadIdx.x & 31;
  if (k >= m) return;  // whole warps leave together
  const int c = warp_cmp(jobs[k].lo, jobs[k].n_lo, base, nb, lane);
  if (lane == 0) need[k] = c >= 0;
}

// hi += 1 for the jobs with need[k] set, one warp a job (the walk stops once
// no carry is left).
__global__ void __launch_bounds__(256) dec_inc_kernel(const DecFixJob* __restrict__ jobs, u64 m,
                                                      const u32* __restrict__ need) {
  const u64 k = ((u64)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const u32 lane = threadIdx.x & 31;
  if (k >= m || !need[k]) return;  // whole warps leave together
  const u64 one = 1;
  warp_addsub(jobs[k].hi, jobs[k].n_hi, &one, 1, false, lane);
}

}  // namespace

cudaError_t dec_groups(const u64* const* nodes, u64 stride, const u32* len, u64 n, u32 groups, char* out,
                       cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  if (stride > kDecMaxLimbs || stride % 2) return cudaErrorInvalidValue;
  const unsigned __int128 all = ~(unsigned __int128)0;
  const u64 v = (u64)(all / kGroupNorm);  // floor((2^128-1)/d) - 2^64: the 2^64 bit drops in the cast
  // four limbs a lane, up to the most warps
  const u64 warps = std::max<u64>(1, std::min<u64>(kDecMaxWarps, (stride + 127) / 128));
  const int smem = dec_smem(warps, stride);  // the longest node's; shorter ones take less
  // the most that any call wants, so that no other thread's call takes it back before this one's launch
  static DeviceOnce once;
  if (const cudaError_t e = allow_smem<dec_smem(kDecMaxWarps, kDecMaxLimbs)>(once, dec_groups_kernel); e != cudaSuccess)
    return e;
  launch_begin("dec_groups", st);
  dec_groups_kernel<<<(unsigned)n, (unsigned)(32 * warps), smem, st>>>(nodes, len, groups, v, out);
  launch_end(st);
  return cudaGetLastError();
}

cudaError_t shr_batch(const ShrJob* d_jobs, const std::vector<ShrJob>& jobs, cudaStream_t st) {
  u64 chunks = 1;
  for (const ShrJob& j : jobs) chunks = std::max<u64>(chunks, (j.n_out + kShrChunk - 1) / kShrChunk);
  for (u64 j0 = 0; j0 < jobs.size(); j0 += 65535) {  // grid y holds at most 65535 jobs
    const unsigned ny = (unsigned)std::min<u64>(65535, jobs.size() - j0);
    launch_begin("dec_shift", st);
    shr_batch_kernel<<<dim3((unsigned)chunks, ny), 256, 0, st>>>(d_jobs + j0);
    launch_end(st);
  }
  return cudaGetLastError();
}

cudaError_t dec_need(const DecFixJob* d_jobs, u64 m, const u64* base, u64 nb, u32* need, cudaStream_t st) {
  if (m == 0) return cudaSuccess;
  launch_begin("dec_need", st);
  dec_need_kernel<<<(unsigned)((m * 32 + 255) / 256), 256, 0, st>>>(d_jobs, m, base, nb, need);
  launch_end(st);
  return cudaGetLastError();
}

cudaError_t dec_inc(const DecFixJob* d_jobs, u64 m, const u32* need, cudaStream_t st) {
  if (m == 0) return cudaSuccess;
  launch_begin("dec_inc", st);
  dec_inc_kernel<<<(unsigned)((m * 32 + 255) / 256), 256, 0, st>>>(d_jobs, m, need);
  launch_end(st);
  return cudaGetLastError();
}

cudaError_t dec_fix(const DecFixJob* d_jobs, u64 m, const u64* base, u64 nb, u32* zero, u32* err, cudaStream_t st) {
  if (m == 0) return cudaSuccess;
  launch_begin("dec_fix", st);
  dec_fix_kernel<<<(unsigned)((m * 32 + 255) / 256), 256, 0, st>>>(d_jobs, m, base, nb, zero, err);
  launch_end(st);
  return cudaGetLastError();
}

}  // namespace nn
