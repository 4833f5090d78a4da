// nn_internal.h — device-side building blocks shared by the engine.
// Host C++; no CUDA types leak past this header except cudaStream_t/cudaError_t.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <functional>
#include <string>
#include <vector>

namespace nn {

typedef std::uint64_t u64;
typedef unsigned int u32;

// Host copy of the prime constants; uploaded to __constant__ memory once per device.
void primes_host(u64 p[3]);
cudaError_t upload_primes();

// Twiddle tables in the reference's layout (ntt_info.h:22-41): per prime,
// words 2k and 2k+1 hold w_k = prod_{bit t of k} root_base[t+1] and its Shoup
// companion floor(w_k * 2^64 / p) + 1.  Grow-only; a table built for scale s
// serves every smaller scale.
struct Tables {
  u64* root = nullptr;   // [3][cap] forward
  u64* iroot = nullptr;  // [3][cap] inverse
  u64 cap = 0;           // words per prime (= 2^(scale-1))
  int scale = 0;
  u32* err = nullptr;    // device error word for kernels whose bounded waits run out (the context's)
};
// Grows the tables to scale s on stream st.  The tables they replace are
// handed to `retired` when given (freed by the caller once no stream can
// still read them: kernels on other streams may hold their pointers), else
// freed in stream order on st.
cudaError_t tables_ensure(Tables& t, int s, cudaStream_t st, std::vector<u64*>* retired = nullptr);
void tables_free(Tables& t);

// One tiled pass over transform levels [lambda0, lambda0 + R) with C columns per tile.
struct Pass {
  int lambda0, R, C;
};
// r_last: levels of the contiguous (deepest) pass; r_col: most levels of a
// strided column pass.
std::vector<Pass> plan_passes(int s, int r_last = 11, int r_col = 9);
// Shared memory of a pass tile (C << R words, padded two words per 32); a
// row pass (C = 2) also stages its 2^R - 1 twiddle pairs.
inline size_t tile_smem_bytes(int C, int R) {
  const size_t n = (size_t)C << R;
  const size_t tile = ((n + n / 16 + 3) & ~(size_t)1) * 8;  // even words: the twiddles start 16-byte aligned
  return C == 2 ? tile + (((size_t)1 << R) - 1) * 16 : tile;
}

// ---- The product pipeline over six 32-bit primes (six.cu) ----

// W[b] pairs (w, round(w 2^32 / p)) of the six primes, then of the inverses:
// [2][6][cap].  Grow-only; a table for scale s serves every smaller one.
struct SixTables {
  int2* tab = nullptr;
  u64 cap = 0;
};
cudaError_t six_tables_ensure(SixTables& t, int s, cudaStream_t st, std::vector<u64*>* retired = nullptr);
void six_tables_free(SixTables& t);

constexpr int kSixMinScale = 4, kSixMaxScale = 31;
// The passes of a transform of scale s: levels R[k] from lambda0[k], the last
// pass over contiguous tiles, down to blocks of 2^lgm coefficients.
// k8 eighths of the transform are computed (5 to 8): the product has at most
// k8 / 8 * 2^s coefficients.
// The last inverse pass multiplies by scale[i] modulo prime i (with its
// companion): the inverse of the factors that the passes leave, times that of
// the other primes' product, as the CRT wants it.
struct SixPlan {
  int s, lgm, n, k8;
  int R[3], lambda0[3];
  int2 scale[6];
  // more than 18 levels: the lazy words are reduced at the last pass's start
  constexpr bool reduce_in() const { return lambda0[n - 1] + R[n - 1] > 18; }
};
// length: coefficients of the product.  row_levels: levels of the last pass of a two-pass transform, where it can
// have that many (0: as even as possible).
SixPlan six_plan(int s, u64 length, int row_levels = 0);
// The plan that takes one operand's finished transform back by itself.
SixPlan six_inverse_plan(int s);

// Operands of a product: a in `pieces` pieces of `piece` limbs (one piece of
// na limbs: not split), residues ra [pieces][6][2^s]; b (nullptr: a square),
// residues rb [6][2^s].  One-pass transforms leave rb untouched.
struct SixOperands {
  const u64* a;
  u64 na, piece;
  u32 pieces;
  const u64* b;
  u64 nb;
  u32* ra;
  u32* rb;
};
// The first pass (tiles [tile0, tile1) of it: tile j covers
// six_first_pass_columns() columns of every row of 2^(s - R[0]) limbs), and
// the rest: products of the pieces with b, as residues in ra for the CRT.
u32 six_first_pass_tiles(const SixPlan& pl);
u32 six_first_pass_columns(const SixPlan& pl);
cudaError_t six_load(const SixOperands& op, const SixPlan& pl, const SixTables& t, cudaStream_t st, u32 tile0 = 0,
                     u32 tile1 = ~0u);
cudaError_t six_finish(const SixOperands& op, const SixPlan& pl, const SixTables& t, cudaStream_t st);
// Whether six_finish takes b through its last levels by itself first (rb is
// then needed for one-pass transforms too): worth its launch when several
// pieces would repeat them.
inline bool six_ready(const SixOperands& op, const SixPlan& pl) {
  return op.b && op.pieces > 1 && ((u64)op.pieces << pl.s) >= (1ull << 18);
}
// The two halves apart, for a transform that is kept: all forward levels, and
// the product of two such transforms (dst may be either) back to residues for
// the CRT.
cudaError_t six_forward(const u64* limbs, u64 n, u32* res, const SixPlan& pl, const SixTables& t, cudaStream_t st);
cudaError_t six_pointwise(u32* dst, const u32* a, const u32* b, const SixPlan& pl, const SixTables& t, cudaStream_t st);
// A finished transform (dst may be it) back to the residues of its operand for the CRT; pl: six_inverse_plan's.
cudaError_t six_inverse(u32* dst, const u32* a, const SixPlan& pl, const SixTables& t, cudaStream_t st);
// Scratch for the carry scan.  Nothing in it outlives a scan but the error word.
struct Scan {
  u32* flags = nullptr;  // per-tile carry bits
  u32* err = nullptr;    // nonzero after a lookback wait gave up
  u32* probe = nullptr;  // a status word that nothing sets
  u64* side = nullptr;   // limbs of the scan beyond the output (the carry words)
  u64 max_tiles = 0;     // tiles that flags holds
  u64 held_tiles = 0;    // ... and the replaced ones with it
  std::vector<u32*> replaced;  // carry bits of smaller scans
};
constexpr int kScanThreads = 256;
constexpr int kScanE = 8;  // limbs per thread
constexpr u64 kScanTile = (u64)kScanThreads * kScanE;

// Batched products (batch.cu): jobs, their work items by launch, and the run.
// A pass item covers consecutive tiles worth about kBatchItemWords residues,
// so a CTA's fixed cost (its item and job) stays small beside its work.
constexpr u64 kBatchItemWords = 8192;
// Base-case items: 256 positions by 256 threads.  With 1024 positions by 128
// threads one item's column sums took 40 us, the whole of a small batch's time:
// 64 jobs of 8 to 1024 limbs 62 us, 37 so.
constexpr int kBatchSumThreads = 256;
constexpr u64 kBatchSumTile = 256;
struct BatchJob {
  const u64* a;  // NTT jobs: the longer operand (split into pieces)
  const u64* b;
  u64* out;      // na + nb limbs
  u64 na, nb;
  u32* res_a;    // [pieces][6][2^s] residues (NTT jobs)
  u32* res_b;    // [6][2^s]
  u64 piece;     // limbs of a per piece (na when not split)
  u64 pieces;
  u32 flag_base; // first carry-scan status word
  int square;    // a == b: one transform
  int rows;      // whose last forward levels run on their own (BatchRows)
  SixPlan plan;  // plan.s 0 for a schoolbook job
};
struct BatchItem {
  u32 job, tile;
  unsigned short ntile;  // consecutive tiles (pass items) of this item
  unsigned char prime, operand;
};
// Launches of a batch, in order: those of one phase are independent.
enum BatchKind : int { kBatchLoad, kBatchCol, kBatchRow, kBatchFused, kBatchInvCol, kBatchSmallRow, kBatchSmall,
                       kBatchCrt, kBatchPieceCrt, kBatchColumns };
// No operand's (both go through them in the fused pass), both operands'
// (batch_fused 0), or the shorter one's, shared by the pieces of the longer.
enum BatchRows : int { kBatchRowsNone, kBatchRowsAll, kBatchRowsB };
struct BatchSegment {
  int phase, kind;
  int pass;    // strided passes: its index in the jobs' plans; contiguous ones: BatchRows
  int R, lgm;  // levels; log2 of the block length (contiguous passes)
  u32 first, count;  // items
};
// Tiles a transform has in pass k of its plan.
u32 batch_pass_tiles(const SixPlan& pl, int k);
// tickets: a zeroed word a segment (the carry scans' tile order); flags: the
// scans' zeroed status words.
cudaError_t batch_launch_segment(const BatchSegment& seg, const BatchJob* jobs, const BatchItem* items, u32* ticket,
                                 u32* flags, u32* err, const SixTables& t, cudaStream_t st);

// Many sums at once (carry.cu): job j writes out = x + y in nout >=
// max(nx, ny) + 1 limbs, or with `sub` out = x - y mod B^nout (x >= y: the
// difference), one warp a job walking 32 limbs a step with the carries of a
// step resolved by ballots.  For jobs of up to a few 10^4 limbs; longer sums
// take lin_combine.
struct AddJob {
  const u64* x;
  u64 nx;
  const u64* y;
  u64 ny;
  u64* out;
  u64 nout;
  u64 sub = 0;
};
cudaError_t add_batch(const AddJob* d_jobs, u64 m, u64 longest, cudaStream_t st);

// Forward transform: limbs (n <= 2^s) -> residues [3][2^s] equal to
// NTT_info::load + NTT (ntt_info.h:147-198) modulo each prime; lazy values in
// [0, 4p) for p0 and p1, [0, 2p) for p2.
cudaError_t ntt_forward(const u64* limbs, u64 n, u64* res, int s, const Tables& t, cudaStream_t st,
                        const std::vector<Pass>* plan = nullptr);
// The forward passes over coefficients that are already residues [3][2^s] below p.
cudaError_t ntt_forward_residues(u64* res, int s, const Tables& t, cudaStream_t st, const std::vector<Pass>& plan);
// A forward transform's lazy values to [0, p), as ntt_inverse takes them.
cudaError_t ntt_canonical(u64* res, int s, cudaStream_t st);
// Pointwise product of degree-1 residues (ntt_info.h:224-231); dst may alias a or b.
cudaError_t ntt_pointwise(u64* dst, const u64* a, const u64* b, int s, const Tables& t, cudaStream_t st);
// Inverse transform with the final 2^-(s-1) scale (ntt_info.h:200-221); values in [0,p).
cudaError_t ntt_inverse(u64* res, int s, const Tables& t, cudaStream_t st, const std::vector<Pass>* plan = nullptr,
                        bool skip_last_pass = false);
// The forward transform of limbs without its last (contiguous) pass.
cudaError_t ntt_forward_head(const u64* limbs, u64 n, u64* res, int s, const Tables& t, cudaStream_t st,
                             const std::vector<Pass>& plan);
// The last forward pass of `res` fused with the pointwise product by `other`
// (a complete forward transform; nullptr squares) and the first inverse pass.
cudaError_t ntt_fused_last(u64* res, const u64* other, int s, const Tables& t, cudaStream_t st,
                           const std::vector<Pass>& plan);
// CRT + carry of six_finish's residues: op's product in out[0..na+nb).
// chunks > 1: in that many ranges of scan tiles, calling done(limb_begin,
// limb_end) after each range's launch (for instance to queue its copy-back).
cudaError_t six_save(const SixOperands& op, const SixPlan& pl, u64* out, Scan& sc, cudaStream_t st, int chunks = 1,
                     const std::function<cudaError_t(u64, u64)>& done = nullptr);
// The same of one transform's product residues at scale s, normal or wrap mode
// as ntt_save below.
cudaError_t six_save_words(const u32* res, int s, u64* out, u64 size, Scan& sc, u64* written, cudaStream_t st);
// The coefficients of product residues [6][2^s] reduced modulo the three
// 62-bit primes: [3][2^s], s < 31; out may be res, apart from it otherwise.
cudaError_t six_to_three(const u32* res, int s, u64* out, cudaStream_t st);
// CRT + carry into `size` limbs (normal mode) or the wrapped product mod
// B^L - 1 in L limbs when size-1 > L (ntt_info.h:237-248).  Returns the
// number of limbs written through *written (host value).
cudaError_t ntt_save(const u64* res, int s, u64* out, u64 size, Scan& sc, u64* written, cudaStream_t st);
// Schoolbook product by column sums + carry scan: out[0..na+nb), apart from the
// operands but where school_whole says that they are read before any limb is
// written.
bool school_whole(u64 na, u64 nb);
cudaError_t school_mul(const u64* a, u64 na, const u64* b, u64 nb, u64* out, Scan& sc, cudaStream_t st);
// out[0..n) = x (nx limbs) + y (ny limbs) shifted up by `shift` limbs; the
// carry out of limb n-1 is dropped.  out must not alias x or y (a tile
// re-reads the inputs just below it while its predecessor may be writing).
cudaError_t add_shifted(const u64* x, u64 nx, const u64* y, u64 ny, u64 shift, u64* out, u64 n, Scan& sc,
                        cudaStream_t st);

// out[0..n_out) = x*B^xs + y*B^ys (sub = false) or x*B^xs - y*B^ys - (1 - cin)
// modulo B^n_out (sub = true), and out[n_out] = the carry out of the top limb
// (for a subtraction with cin = 1: 1 exactly when x*B^xs >= y*B^ys).  out
// holds n_out + 1 limbs and does not alias x or y.  A nonzero *flip (device
// memory, when flip is given) swaps add and subtract.
cudaError_t lin_combine(u64* out, u64 n_out, const u64* x, u64 nx, u64 xs, const u64* y, u64 ny, u64 ys, bool sub,
                        int cin, Scan& sc, cudaStream_t st, const u64* flip = nullptr);
// out[0..n] = in << cl (n + 1 limbs) and out[0..n) = in >> cl, 0 <= cl <= 63;
// out does not overlap in.
cudaError_t shl_bits(u64* out, const u64* in, u64 n, unsigned cl, cudaStream_t st);
cudaError_t shr_bits(u64* out, const u64* in, u64 n, unsigned cl, cudaStream_t st);

// Runs the carry lookback's bounded wait on a status word nothing sets (at
// most `limit` polls); it gives up and sets sc.err, which the host reads.
cudaError_t wait_probe(Scan& sc, int limit, cudaStream_t st);

// The decimal split on the device (decimal.cu): out = in >> shift bits for
// many jobs (n_out limbs each, in read as zero past n_in); and the split's
// correction (natural.h:962-965): while lo >= base, hi += 1 and lo -= base,
// one warp a node, with zero[k] = (hi == 0) after it and *err set when a node
// needed more than 8 steps.
constexpr u64 kShrChunk = 4096;
struct ShrJob {
  const u64* in;
  u64 n_in;
  u64* out;
  u64 n_out;
  u64 shift;
};
cudaError_t shr_batch(const ShrJob* d_jobs, const std::vector<ShrJob>& jobs, cudaStream_t st);
struct DecFixJob {
  u64* lo;
  u64 n_lo;
  u64* hi;
  u64 n_hi;
};
cudaError_t dec_fix(const DecFixJob* d_jobs, u64 m, const u64* base, u64 nb, u32* zero, u32* err, cudaStream_t st);
// need[k] = (lo of job k >= base), one warp a job: the test of dec_fix's loop
// alone, for callers that correct long nodes with multiword scans.
cudaError_t dec_need(const DecFixJob* d_jobs, u64 m, const u64* base, u64 nb, u32* need, cudaStream_t st);
// hi += 1 for the jobs with need[k] set, one warp a job.
cudaError_t dec_inc(const DecFixJob* d_jobs, u64 m, const u32* need, cudaStream_t st);

// Decimal digits of n short naturals at once (decimal.cu): node k's len[k]
// limbs at nodes[k] (device pointers; len[k] <= stride, stride even and at
// most 8192); node k < 10^(18 * groups) goes to out[k * 18 * groups ...) as
// 18 * groups zero-padded digits, most significant first.
cudaError_t dec_groups(const u64* const* nodes, u64 stride, const u32* len, u64 n, u32 groups, char* out,
                       cudaStream_t st);

// Launch accounting (profile.cpp): every launch site brackets its kernel.
void launch_begin(const char* name, cudaStream_t st);
void launch_end(cudaStream_t st);
unsigned long long launch_count();
void profile_enable(bool on);
std::string profile_report();

u64 scan_tiles(u64 positions);
cudaError_t scan_reserve(Scan& sc, u64 tiles);
void scan_free(Scan& sc);

}  // namespace nn
