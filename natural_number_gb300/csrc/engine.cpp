// engine.cpp — context, device-resident transforms and the C ABI of
// include/natural_gb300.h.  Host C++ that orders the sm_103a kernels of
// ntt.cu / carry.cu on one CUDA stream; no computation happens on the host
// besides size bookkeeping and the final normalisation of host results.
#include <cuda_runtime.h>
#include <dlfcn.h>

#include <algorithm>
#include <array>
#include <bit>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <unordered_map>
#include <unordered_set>
#include <vector>

#include "../../include/natural_gb300.h"
#include "nn_internal.h"
#include "stage_ring.h"

using nn::u64;

namespace {
constexpr u64 kNttMulThreshold = 384;  // ntt_info.h:6

int ntt_scale(u64 n1, u64 n2) {  // get_NTT_scale (natural.h:384-386)
  u64 v = n1 + n2 - 2;
  return 64 - std::countl_zero(v);
}

// Page-locked staging ring for the small host tables a call uploads (batch
// plans, job tables, sum tables).  A copy from pageable memory may wait for
// the stream's earlier work before it returns, which would stop the host
// from planning the next batch while the GPU runs this one; from this ring
// the copy is queued and the call returns at once.  Regions are handed out
// in order; one is reused after the event recorded behind its copy (the
// bookkeeping: RegionRing, stage_ring.h).
struct CudaEvents {
  using event = cudaEvent_t;
  std::vector<cudaEvent_t> spare;
  bool done(cudaEvent_t e) { return cudaEventQuery(e) == cudaSuccess; }
  void wait(cudaEvent_t e) { cudaEventSynchronize(e); }
  void recycle(cudaEvent_t e) { spare.push_back(e); }
};

struct Stager {
  char* base = nullptr;
  CudaEvents ev;
  nn::RegionRing<CudaEvents> ring;

  // bytes from host memory at src to device memory at dst, queued on st.
  cudaError_t upload(void* dst, const void* src, u64 bytes, cudaStream_t st) {
    if (!bytes) return cudaSuccess;
    const u64 n = ring.granule(bytes);
    if (n > ring.cap) {  // a larger ring, once every copy from this one is done
      ring.drain(ev);
      if (base) nn_host_free(base, ring.cap);
      ring.cap = std::max<u64>(std::bit_ceil(2 * n), 16ull << 20);
      ring.head = 0;
      base = static_cast<char*>(nn_host_alloc(ring.cap));
      if (!base) {  // no page-locked memory to be had
        ring.cap = 0;
        return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
      }
    }
    char* h = base + ring.place(n, ev);
    std::memcpy(h, src, bytes);
    cudaError_t e = cudaMemcpyAsync(dst, h, bytes, cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) {
      ring.drop();
      return e;
    }
    cudaEvent_t done = nullptr;
    if (!ev.spare.empty()) {
      done = ev.spare.back();
      ev.spare.pop_back();
    } else {
      e = cudaEventCreateWithFlags(&done, cudaEventDisableTiming);
    }
    if (e == cudaSuccess) e = cudaEventRecord(done, st);
    if (e != cudaSuccess) {  // the copy is queued but no event marks its end: wait for it here
      if (done) ev.spare.push_back(done);
      cudaStreamSynchronize(st);
      ring.drop();
      return e;
    }
    ring.seal(done);
    return cudaSuccess;
  }
  void release() {
    ring.drain(ev);
    for (cudaEvent_t e : ev.spare) cudaEventDestroy(e);
    ev.spare.clear();
    if (base) nn_host_free(base, ring.cap);
    base = nullptr;
    ring.cap = ring.head = 0;
  }
};
}  // namespace

struct nn_context {
  int device = 0;
  cudaStream_t own = nullptr;
  cudaStream_t stream = nullptr;
  // host-pointer calls: the second operand's copy runs on `copy` while the
  // first operand is transformed
  cudaStream_t copy = nullptr;
  cudaEvent_t ev_first = nullptr, ev_second = nullptr, ev_chunk = nullptr, ev_in = nullptr;
  // a batch's independent launches beside each other (made by the first batch that runs)
  static constexpr int kSide = 3;
  cudaStream_t side[kSide] = {};
  cudaEvent_t ev_side = nullptr;
  u64 budget = 0;
  u64 held = 0;  // bytes of live allocations made through the context
  nn::Tables tables;   // three-prime transforms (nn_transform_*, nn_ntt_mul)
  nn::SixTables six;   // products
  nn::Scan scan;
  std::string err;
  u64* scratch[3] = {nullptr, nullptr, nullptr};  // grow-only device staging for host calls
  u64 scratch_words[3] = {0, 0, 0};
  Stager stage;  // page-locked ring for uploaded tables
  // Twiddle tables replaced by larger ones: kept until the context goes, as
  // work on another stream (set_stream, or a server's concurrent batches)
  // may still read them; together at most the size of the live tables.
  std::vector<u64*> retired_tables;
  // tunables (nn_context_set_tunable)
  int r_last = 11;            // levels of the contiguous NTT pass
  int r_col = 9;              // most levels of a strided column pass
  int r_last_at[64] = {};     // per-scale overrides (0: use r_last / r_col)
  int r_col_at[64] = {};
  int batch_r_last_at[64] = {};  // levels of a two-pass batched transform's last pass (0: six_plan's)
  std::vector<nn::Pass> passes(int s) const {
    const int rl = (s >= 0 && s < 64 && r_last_at[s]) ? r_last_at[s] : r_last;
    const int rc = (s >= 0 && s < 64 && r_col_at[s]) ? r_col_at[s] : r_col;
    return nn::plan_passes(s, rl, rc);
  }
  u64 batch_ntt_min = 384;    // batches: schoolbook when min(n_a, n_b) is below this
  u64 batch_school_balanced = 256;  // ... or below this when max(n_a, n_b) <= 2 min(n_a, n_b) (0: off)
  u64 batch_item_words = nn::kBatchItemWords;  // residues a pass item covers at least
  int batch_fused = 1;        // batches: last forward levels, products and first inverse levels in one item
  int batch_merge = 1;        // kept for callers that set it: every batch tile fills its CTA
  int batch_split = 1;        // batches: unbalanced products in pieces sharing one transform
  int batch_blocks_per_sm = 0;  // kept for callers that set it: a CTA an item
  int batch_solo_scale = 22;    // batches: products of this scale and up run one at a time (0: never)
  int batch_few = 1;            // batches of a few short products: one scale for all of them
};

struct nn_batch {
  u64 count = 0;
  std::vector<u64> na, nb;
  std::vector<nn::BatchJob> jobs;
  std::vector<nn::BatchItem> items;        // by launch
  std::vector<nn::BatchSegment> segments;  // the launches, in order
  std::vector<u64> off_a, off_b;
  std::vector<char> swap;  // NTT job whose second operand is the longer one
  std::vector<u64> solo;   // jobs run one at a time after the launches
  u64 arena_words = 0;
  nn::u32 n_flags = 0;
  nn::BatchJob* d_jobs = nullptr;
  nn::BatchItem* d_items = nullptr;
  nn::u32* d_state = nullptr;  // a ticket counter a launch, then the scans' status words
  u64* d_arena = nullptr;
  u64 dev_words = 0;           // budget accounting of the above
  nn::BatchJob* h_jobs = nullptr;  // pinned staging of the job table
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  cudaEvent_t ran = nullptr;
  bool pending = false;
  bool started = false;  // nn_batch_run has run it
};

// A kept transform.  Its residues are six-prime words — the finished forward
// transform, or a product's residues as the CRT takes them — or the
// three-prime words of the reference's layout: for scales the six primes do
// not serve, and for products of more than two factors, whose coefficients may
// exceed what six primes hold.
struct nn_transform {
  enum Rep { kThree, kSixForward, kSixProduct };
  u64* res = nullptr;  // [3][2^scale], or [6][2^scale] 32-bit words
  u64 words = 0;       // allocated words (3 * 2^scale at most)
  int scale = 0;
  Rep rep = kThree;
  nn::u32* six() const { return reinterpret_cast<nn::u32*>(res); }
};

namespace {

nn_status fail(nn_context* c, cudaError_t e, const char* what) {
  c->err = std::string(what) + ": " + cudaGetErrorString(e);
  cudaGetLastError();  // clear sticky-free errors
  return e == cudaErrorMemoryAllocation ? NN_ERR_OOM : NN_ERR_CUDA;
}

#define NN_CK(ctx, expr, what)                           \
  do {                                                   \
    cudaError_t _e = (expr);                             \
    if (_e != cudaSuccess) return fail((ctx), _e, what); \
  } while (0)

nn_status dev_alloc(nn_context* c, u64** p, u64 words) {
  const u64 bytes = std::max<u64>(words, 1) * sizeof(u64);
  if (c->budget && c->held + bytes > c->budget) {
    c->err = "HBM budget exceeded";
    return NN_ERR_BUDGET;
  }
  cudaError_t e = cudaMallocAsync((void**)p, bytes, c->stream);
  if (e != cudaSuccess) return fail(c, e, "cudaMallocAsync");
  c->held += bytes;
  return NN_OK;
}

void dev_free(nn_context* c, u64* p, u64 words) {
  if (!p) return;
  cudaFreeAsync(p, c->stream);
  c->held -= std::max<u64>(words, 1) * sizeof(u64);
}

// RAII device buffer tied to the context's stream.
struct DBuf {
  nn_context* c;
  u64* p = nullptr;
  u64 words = 0;
  explicit DBuf(nn_context* ctx) : c(ctx) {}
  nn_status alloc(u64 w) {
    words = w;
    return dev_alloc(c, &p, w);
  }
  ~DBuf() { dev_free(c, p, words); }
};

bool short_of_memory(nn_status st) { return st == NN_ERR_BUDGET || st == NN_ERR_OOM; }

// Whether the context's stream is captured (or cannot tell).
bool capturing(const nn_context* c) {
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(c->stream, &capture) == cudaSuccess) return capture != cudaStreamCaptureStatusNone;
  cudaGetLastError();
  return true;
}

nn_status xform_reserve(nn_context* c, nn_transform* t, int s) {
  const u64 need = 3ull << s;
  if (t->words < need) {
    dev_free(c, t->res, t->words);
    t->res = nullptr;
    t->words = 0;
    nn_status st = dev_alloc(c, &t->res, need);
    if (st != NN_OK) return st;
    t->words = need;
  }
  t->scale = s;
  return NN_OK;
}

// Three-prime transform.
nn_status forward3(nn_context* c, nn_transform* t, const u64* d_limbs, u64 n, int s) {
  NN_CK(c, nn::tables_ensure(c->tables, s, c->stream, &c->retired_tables), "twiddle tables");
  nn_status st = xform_reserve(c, t, s);
  if (st != NN_OK) return st;
  t->rep = nn_transform::kThree;
  const std::vector<nn::Pass> plan = c->passes(s);
  NN_CK(c, nn::ntt_forward(d_limbs, n, t->res, s, c->tables, c->stream, &plan), "forward NTT");
  return NN_OK;
}

nn_status inverse_save3(nn_context* c, nn_transform* t, u64* d_out, u64 size, u64* written,
                        bool skip_last_pass = false) {
  const std::vector<nn::Pass> plan = c->passes(t->scale);
  NN_CK(c, nn::ntt_inverse(t->res, t->scale, c->tables, c->stream, &plan, skip_last_pass), "inverse NTT");
  u64 w = 0;
  NN_CK(c, nn::ntt_save(t->res, t->scale, d_out, size, c->scan, &w, c->stream), "CRT/carry");
  if (written) *written = w;
  return NN_OK;
}

nn_status forward_args(nn_context* c, u64 n, int s) {
  if (s >= 2 && s <= 40 && n != 0 && n <= (1ull << s)) return NN_OK;
  c->err = "forward: need 2 <= scale <= 40 and 1 <= n <= 2^scale";
  return NN_ERR_INVALID;
}
nn_status save_args(nn_context* c, u64 size) {
  if (size >= 2) return NN_OK;
  c->err = "save: size must be at least 2";
  return NN_ERR_INVALID;
}

// Kept transforms over six primes up to this scale (blocks of up to 64
// coefficients; beyond, the three-prime passes are faster).
constexpr int kSixTransformMaxScale = 28;

nn_status forward(nn_context* c, nn_transform* t, const u64* d_limbs, u64 n, int s) {
  nn_status st = forward_args(c, n, s);
  if (st != NN_OK) return st;
  if (s < nn::kSixMinScale || s > kSixTransformMaxScale) return forward3(c, t, d_limbs, n, s);
  NN_CK(c, nn::six_tables_ensure(c->six, s, c->stream, &c->retired_tables), "twiddle tables");
  st = xform_reserve(c, t, s);
  if (st != NN_OK) return st;
  t->rep = nn_transform::kSixForward;
  NN_CK(c, nn::six_forward(d_limbs, n, t->six(), nn::six_plan(s, 1ull << s), c->six, c->stream), "forward NTT");
  return NN_OK;
}

// t's residues modulo the three primes, as the reference's transform has
// them, into dst (on a 16-byte boundary): a six-prime transform's coefficients,
// reduced, through the three-prime forward passes.
nn_status three_words(nn_context* c, const nn_transform* t, u64* dst) {
  if (t->rep == nn_transform::kThree) {
    NN_CK(c, cudaMemcpyAsync(dst, t->res, (3ull << t->scale) * sizeof(u64), cudaMemcpyDeviceToDevice, c->stream),
          "copy residues");
    return NN_OK;
  }
  NN_CK(c, nn::tables_ensure(c->tables, t->scale, c->stream, &c->retired_tables), "twiddle tables");
  DBuf tmp(c);
  const nn::u32* w = t->six();
  if (t->rep == nn_transform::kSixForward) {
    const nn_status st = tmp.alloc(3ull << t->scale);
    if (st != NN_OK && !short_of_memory(st)) return st;
    nn::u32* back = reinterpret_cast<nn::u32*>(st == NN_OK ? tmp.p : dst);
    NN_CK(c, nn::six_inverse(back, w, nn::six_inverse_plan(t->scale), c->six, c->stream), "inverse NTT");
    w = back;
  }
  NN_CK(c, nn::six_to_three(w, t->scale, dst, c->stream), "residues");
  NN_CK(c, nn::ntt_forward_residues(dst, t->scale, c->tables, c->stream, c->passes(t->scale)), "forward NTT");
  return NN_OK;
}

// The same in t's own memory: the transform is still the same one.  Not while
// the stream is captured, where t changes with every replay.
nn_status become_three(nn_context* c, nn_transform* t) {
  NN_CK(c, nn::tables_ensure(c->tables, t->scale, c->stream, &c->retired_tables), "twiddle tables");
  if (t->rep == nn_transform::kSixForward) {
    NN_CK(c, nn::six_inverse(t->six(), t->six(), nn::six_inverse_plan(t->scale), c->six, c->stream), "inverse NTT");
    t->rep = nn_transform::kSixProduct;
  }
  NN_CK(c, nn::six_to_three(t->six(), t->scale, t->res, c->stream), "residues");
  t->rep = nn_transform::kThree;
  NN_CK(c, nn::ntt_forward_residues(t->res, t->scale, c->tables, c->stream, c->passes(t->scale)), "forward NTT");
  NN_CK(c, nn::ntt_canonical(t->res, t->scale, c->stream), "forward NTT");  // it may be taken back alone
  return NN_OK;
}

// t's three-prime words: its own, or a copy in tmp, or, where there is no memory
// for one (a product of three factors took none when every transform had three
// primes), t's own from now on.
nn_status three_operand(nn_context* c, const nn_transform* t, DBuf& tmp, const u64** words) {
  *words = t->res;
  if (t->rep == nn_transform::kThree) return NN_OK;
  nn_status st = tmp.alloc(3ull << t->scale);
  if (st == NN_OK) {
    *words = tmp.p;
    return three_words(c, t, tmp.p);
  }
  if (!short_of_memory(st) || capturing(c)) return st;
  return become_three(c, const_cast<nn_transform*>(t));
}

// A forward transform goes back in place: only kernels on the stream, as a
// captured graph wants them, and no memory beyond the transform's own.
nn_status inverse_save(nn_context* c, nn_transform* t, u64* d_out, u64 size, u64* written) {
  nn_status st = save_args(c, size);
  if (st != NN_OK) return st;
  if (t->rep == nn_transform::kThree) return inverse_save3(c, t, d_out, size, written);
  if (t->rep == nn_transform::kSixForward) {
    NN_CK(c, nn::six_inverse(t->six(), t->six(), nn::six_inverse_plan(t->scale), c->six, c->stream), "inverse NTT");
    t->rep = nn_transform::kSixProduct;
  }
  u64 n = 0;
  NN_CK(c, nn::six_save_words(t->six(), t->scale, d_out, size, c->scan, &n, c->stream), "CRT/carry");
  if (written) *written = n;
  return NN_OK;
}

nn_status pointwise(nn_context* c, nn_transform* dst, const nn_transform* a, const nn_transform* b) {
  if (a->scale != b->scale || a->scale < 2) {
    c->err = "pointwise: transforms differ in scale";
    return NN_ERR_INVALID;
  }
  const int s = a->scale;
  if (a->rep == nn_transform::kSixForward && b->rep == nn_transform::kSixForward) {
    nn_status st = xform_reserve(c, dst, s);
    if (st != NN_OK) return st;
    NN_CK(c, nn::six_pointwise(dst->six(), a->six(), b->six(), nn::six_plan(s, 1ull << s), c->six, c->stream),
          "pointwise");
    dst->rep = nn_transform::kSixProduct;
    return NN_OK;
  }
  DBuf ta(c), tb(c);
  const u64 *pa = nullptr, *pb = nullptr;
  nn_status st = three_operand(c, a, ta, &pa);
  if (st == NN_OK && b != a) st = three_operand(c, b, tb, &pb);
  if (b == a) pb = pa;
  if (st == NN_OK) st = xform_reserve(c, dst, s);
  if (st != NN_OK) return st;
  NN_CK(c, nn::tables_ensure(c->tables, s, c->stream, &c->retired_tables), "twiddle tables");
  NN_CK(c, nn::ntt_pointwise(dst->res, pa, pb, s, c->tables, c->stream), "pointwise");
  dst->rep = nn_transform::kThree;
  return NN_OK;
}

// The second operand's transform up to its last pass, then that pass fused
// with the pointwise product by `other` (nullptr: square) and the first
// inverse pass; the caller finishes with inverse_save(skip_last_pass).
nn_status forward_fused(nn_context* c, nn_transform* t, const u64* d_limbs, u64 n, int s, const nn_transform* other) {
  NN_CK(c, nn::tables_ensure(c->tables, s, c->stream, &c->retired_tables), "twiddle tables");
  nn_status st = xform_reserve(c, t, s);
  if (st != NN_OK) return st;
  const std::vector<nn::Pass> plan = c->passes(s);
  NN_CK(c, nn::ntt_forward_head(d_limbs, n, t->res, s, c->tables, c->stream, plan), "forward NTT");
  NN_CK(c, nn::ntt_fused_last(t->res, other ? other->res : nullptr, s, c->tables, c->stream, plan),
        "fused pass");
  return NN_OK;
}

// Three-prime product at scale s into d_out (size limbs, or wrap).
nn_status ntt_product(nn_context* c, u64* d_out, const u64* a, u64 na, const u64* b, u64 nb, int s, u64 size,
                      u64* written) {
  nn_transform xa, xb;
  nn_status st = forward_args(c, na, s);
  if (st == NN_OK) st = forward_args(c, nb, s);
  if (st == NN_OK) st = save_args(c, size);
  if (st == NN_OK) st = forward3(c, &xa, a, na, s);
  if (st == NN_OK && c->passes(s).size() >= 2) {
    st = forward_fused(c, &xb, b, nb, s, &xa);
    if (st == NN_OK) st = inverse_save3(c, &xb, d_out, size, written, true);
  } else {
    if (st == NN_OK) st = forward3(c, &xb, b, nb, s);
    if (st == NN_OK) st = pointwise(c, &xb, &xa, &xb);
    if (st == NN_OK) st = inverse_save3(c, &xb, d_out, size, written);
  }
  dev_free(c, xa.res, xa.words);
  dev_free(c, xb.res, xb.words);
  return st;
}

// Residues of a product over six primes: ra, then rb where it is used.
nn_status six_residues(nn_context* c, DBuf& buf, nn::SixOperands& op, const nn::SixPlan& pl) {
  NN_CK(c, nn::six_tables_ensure(c->six, pl.s, c->stream, &c->retired_tables), "twiddle tables");
  const u64 each = 3ull << pl.s;  // 6 words of 32 bits a coefficient
  const bool two = op.b && (pl.n > 1 || nn::six_ready(op, pl));
  nn_status st = buf.alloc((op.pieces + (two ? 1 : 0)) * each);
  if (st != NN_OK) return st;
  op.ra = reinterpret_cast<nn::u32*>(buf.p);
  op.rb = two ? reinterpret_cast<nn::u32*>(buf.p + op.pieces * each) : nullptr;
  return NN_OK;
}

// Coefficients of a transform's product: a piece's when the longer operand is split.
u64 six_length(const nn::SixOperands& op) { return op.piece + (op.b ? op.nb : op.na) - 1; }

// op's product over six primes at scale s (op.b nullptr: the square).
nn_status six_product(nn_context* c, u64* d_out, nn::SixOperands op, int s) {
  const nn::SixPlan pl = nn::six_plan(std::max(s, nn::kSixMinScale), six_length(op));
  DBuf buf(c);
  nn_status st = six_residues(c, buf, op, pl);
  if (st != NN_OK) return st;
  NN_CK(c, nn::six_load(op, pl, c->six, c->stream), "first pass");
  NN_CK(c, nn::six_finish(op, pl, c->six, c->stream), "passes");
  NN_CK(c, nn::six_save(op, pl, d_out, c->scan, c->stream), "CRT/carry");
  return NN_OK;
}

// Product of host operands (ha: na limbs, hb: nb limbs, na >= nb) into d_out
// and h_out.  a's copy to da goes a range of columns at a time (kInChunks
// ranges: a 2-D copy of the range in every full row of the first pass, plus
// its part of a last, partial row) on the copy stream, and the first pass
// runs each range's tiles as soon as it has arrived, so the copy overlaps
// that pass; b's copy follows on the same stream.  The product's limbs go
// back range by range (kCopyChunks) behind the carry scan.  *used is false,
// and nothing is done, for transforms of one pass.
// The sixteen and more copies only pay for long operands in page-locked memory
// (from pageable memory each is staged by the driver): in ranges / whole, us, page-
// locked 20000 x 20000 limbs 135 / 57, 2^20 x 2^20 373 / 371, 3000000 x 2000000
// 871 / 902, 8000000 x 8000000 2501 / 2675, pageable 20000 x 20000 309 / 74, 2^20
// x 2^20 592 / 391, 8000000 x 8000000 2985 / 2805.
constexpr int kInChunks = 8, kCopyChunks = 8;
constexpr u64 kChunkedLimbs = 1 << 21;  // of the product, in ranges beyond
bool page_locked(const void* p) {
  cudaPointerAttributes at{};
  if (cudaPointerGetAttributes(&at, p) == cudaSuccess) return at.type == cudaMemoryTypeHost;
  cudaGetLastError();
  return false;
}
nn_status six_product_from_host(nn_context* c, u64* d_out, u64* da, const u64* ha, u64 na, u64* db, const u64* hb,
                                u64 nb, int s, u64* h_out, bool* used) {
  *used = false;
  const nn::SixPlan pl = nn::six_plan(std::max(s, nn::kSixMinScale), na + nb - 1);
  const u64 tiles = nn::six_first_pass_tiles(pl), width = nn::six_first_pass_columns(pl);
  if (pl.n < 2) return NN_OK;
  *used = true;
  nn::SixOperands op{da, na, na, 1, db, nb, nullptr, nullptr};
  DBuf buf(c);
  nn_status st = six_residues(c, buf, op, pl);
  if (st != NN_OK) return st;
  const nn::SixOperands first{da, na, na, 1, nullptr, 0, op.ra, nullptr}, second{db, nb, nb, 1, nullptr, 0, op.rb, nullptr};
  const u64 row = 1ull << (pl.s - pl.R[0]);            // limbs a row of the first pass
  const u64 full = na / row, part = na - full * row;  // full rows, limbs of the partial row
  const u64 k = std::min<u64>(kInChunks, tiles);
  cudaError_t e = cudaEventRecord(c->ev_first, c->stream);  // da and db are reused: after earlier work
  if (e == cudaSuccess) e = cudaStreamWaitEvent(c->copy, c->ev_first, 0);
  for (u64 j = 0; j < k && e == cudaSuccess; ++j) {
    const u64 t0 = tiles * j / k, t1 = tiles * (j + 1) / k, c0 = width * t0, c1 = width * t1;
    if (full)
      e = cudaMemcpy2DAsync(da + c0, row * 8, ha + c0, row * 8, (c1 - c0) * 8, full, cudaMemcpyHostToDevice, c->copy);
    if (e == cudaSuccess && part > c0)
      e = cudaMemcpyAsync(da + full * row + c0, ha + full * row + c0, (std::min(c1, part) - c0) * 8,
                          cudaMemcpyHostToDevice, c->copy);
    if (e == cudaSuccess) e = cudaEventRecord(c->ev_in, c->copy);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(c->stream, c->ev_in, 0);
    if (e == cudaSuccess) e = nn::six_load(first, pl, c->six, c->stream, (nn::u32)t0, (nn::u32)t1);
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(db, hb, nb * 8, cudaMemcpyHostToDevice, c->copy);
  if (e == cudaSuccess) e = cudaEventRecord(c->ev_second, c->copy);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(c->stream, c->ev_second, 0);
  if (e == cudaSuccess) e = nn::six_load(second, pl, c->six, c->stream);
  if (e == cudaSuccess) e = nn::six_finish(op, pl, c->six, c->stream);
  if (e == cudaSuccess)
    e = nn::six_save(op, pl, d_out, c->scan, c->stream, kCopyChunks, [&](u64 lo, u64 hi) {
      cudaError_t r = cudaEventRecord(c->ev_chunk, c->stream);
      if (r == cudaSuccess) r = cudaStreamWaitEvent(c->copy, c->ev_chunk, 0);
      if (r == cudaSuccess)
        r = cudaMemcpyAsync(h_out + lo, d_out + lo, (hi - lo) * 8, cudaMemcpyDeviceToHost, c->copy);
      return r;
    });
  if (e != cudaSuccess) return fail(c, e, "product from host operands");
  return NN_OK;
}

// An unbalanced product nx x ny (nx >= ny) at scale s may run as P pieces of k
// limbs of the longer operand, each through a transform of scale s2 < s
// sharing the shorter operand's: 2P + 1 transforms of 2^s2 words and s2 - 3
// levels against 3 of 2^s.  k is the most that keeps a piece's product within
// its transform (k + ny - 1 <= 2^s2), rounded down to a multiple of 8 (the CRT
// scan's vector loads stay within a piece), and at least ny, so that at most
// two pieces overlap at any position.  The cost of a word is its levels plus
// about four levels' worth of load, block products and CRT.
int six_split(u64 nx, u64 ny, int s, u64* k, u64* P) {
  // one transform: the eighths of it that hold the product
  const double part = (double)std::clamp<u64>(((nx + ny - 1) * 8 + (1ull << s) - 1) >> s, 5, 8) / 8;
  double best = 3.0 * part * (double)(1ull << s) * (s + 1);
  int s_best = s;
  *k = nx;
  *P = 1;
  for (int s2 = s - 1; s2 >= nn::kSixMinScale; --s2) {
    const u64 L2 = 1ull << s2;
    if (L2 + 1 < 2 * ny) break;
    const u64 kk = (L2 - ny + 1) & ~7ull;
    if (kk < ny || kk >= nx) continue;
    const u64 pieces = (nx + kk - 1) / kk;
    if (pieces > 32768) break;  // a grid dimension of the passes
    const double cost = (2.0 * pieces + 1.0) * (double)L2 * (s2 + 1);
    if (cost < 0.95 * best) {
      best = cost;
      s_best = s2;
      *k = kk;
      *P = pieces;
    }
  }
  return s_best;
}

// Whether na x nb limbs (na >= nb) run as the base case.  Both ways give the
// same limbs; with a product's launches 1.3 us apart the transforms win well
// below the reference's 384 limbs.  Measured, transforms / base case, us: 224 x
// 224 6.1 / 5.6, 256 x 256 6.4 / 6.8, 383 x 383 6.5 / 8.1; beyond the one
// cluster of 1024 positions 1024 x 96 7.0 / 7.1, 2048 x 192 7.4 / 9.5, 2048 x 64
// 6.8 / 6.7; long operands 16384 x 32 9.0 / 10.6, 2^20 x 32 58.8 / 81.1, 2^20 x
// 300 70 / 743, but 2^20 x 16 74.3 / 44.7.
bool base_case(u64 na, u64 nb) {
  return !(nb >= 256 || (nb >= 96 && na + nb > 1024) || (nb >= 32 && na >= 16384));
}

// Base-case product.  Tiles of a longer one write limbs while others still read
// operands: an operand that lies in the output's limbs (a product in place, which
// the transforms take as it is) is copied first.
nn_status base_product(nn_context* c, u64* d_out, const u64* a, u64 na, const u64* b, u64 nb) {
  auto lies = [&](const u64* x, u64 n) { return x < d_out + (na + nb) && d_out < x + n; };
  u64* copy = nullptr;
  if (!nn::school_whole(na, nb) && (lies(a, na) || lies(b, nb))) {
    NN_CK(c, cudaMallocAsync((void**)&copy, (na + nb) * 8, c->stream), "operands in place");
    cudaError_t e = cudaMemcpyAsync(copy, a, na * 8, cudaMemcpyDeviceToDevice, c->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(copy + na, b, nb * 8, cudaMemcpyDeviceToDevice, c->stream);
    if (e != cudaSuccess) {
      cudaFreeAsync(copy, c->stream);
      return fail(c, e, "operands in place");
    }
    a = copy;
    b = copy + na;
  }
  const cudaError_t e = nn::school_mul(a, na, b, nb, d_out, c->scan, c->stream);
  if (copy) cudaFreeAsync(copy, c->stream);
  NN_CK(c, e, "base-case product");
  return NN_OK;
}

// A product of fewer than kNttMulThreshold limbs needs no memory as the base
// case: it takes that where the transforms' would not fit the budget, and while
// the stream is captured, where their memory would be a part of the graph (which
// then has one instance at a time and cannot be part of another graph).
nn_status short_product(nn_context* c, u64* d_out, const nn::SixOperands& op, int s) {
  if (!capturing(c)) {
    const nn_status st = six_product(c, d_out, op, s);
    if (!short_of_memory(st)) return st;
  }
  return base_product(c, d_out, op.a, op.na, op.b ? op.b : op.a, op.nb);
}

nn_status mul_impl(nn_context* c, u64* d_out, const u64* a, u64 na, const u64* b, u64 nb) {
  if (!d_out || !a || !b || na == 0 || nb == 0) {
    c->err = "mul: null pointer or empty operand";
    return NN_ERR_INVALID;
  }
  if (na < nb) {
    std::swap(a, b);
    std::swap(na, nb);
  }
  if (base_case(na, nb)) return base_product(c, d_out, a, na, b, nb);  // natural.h:445-446 -> _mul_base
  // natural::_mul_NTT (natural.h:391-419) cuts the longer operand in two when
  // that lowers the scale; here it may go in any number of pieces.
  u64 piece, pieces;
  const int s = six_split(na, nb, ntt_scale(na, nb), &piece, &pieces);
  if (s > nn::kSixMaxScale) return ntt_product(c, d_out, a, na, b, nb, s, na + nb, nullptr);
  const nn::SixOperands op{a, na, piece, (nn::u32)pieces, b, nb, nullptr, nullptr};
  return nb < kNttMulThreshold ? short_product(c, d_out, op, s) : six_product(c, d_out, op, s);
}

nn_status sqr_impl(nn_context* c, u64* d_out, const u64* a, u64 n) {
  if (!d_out || !a || n == 0) {
    c->err = "sqr: null pointer or empty operand";
    return NN_ERR_INVALID;
  }
  if (base_case(n, n)) return base_product(c, d_out, a, n, a, n);  // natural.h:530-531 -> _sqr_base
  // natural::_sqr_NTT (natural.h:433-442): one transform.
  const int s = ntt_scale(n, n);
  if (s > nn::kSixMaxScale) return ntt_product(c, d_out, a, n, a, n, s, 2 * n, nullptr);
  const nn::SixOperands op{a, n, n, 1, nullptr, n, nullptr, nullptr};
  return n < kNttMulThreshold ? short_product(c, d_out, op, s) : six_product(c, d_out, op, s);
}

// Grow-only device staging buffer `slot` of at least `words` limbs.
nn_status scratch(nn_context* c, int slot, u64 words, u64** p) {
  if (c->scratch_words[slot] < words) {
    dev_free(c, c->scratch[slot], c->scratch_words[slot]);
    c->scratch[slot] = nullptr;
    c->scratch_words[slot] = 0;
    u64 w = std::bit_ceil(std::max<u64>(words, 1024));
    nn_status st = dev_alloc(c, &c->scratch[slot], w);
    if (st != NN_OK) return st;
    c->scratch_words[slot] = w;
  }
  *p = c->scratch[slot];
  return NN_OK;
}

// ---------------------------------------------------------------------------
// Batches: launches of one step and tile shape over all jobs (batch.cu).
// ---------------------------------------------------------------------------

// How a product of a batch runs: as column sums (plan.s 0), through transforms,
// by itself after the batch's launches, or not at all.
enum class BatchRoute { kColumns, kTransforms, kSolo, kTooLong };

bool batch_columns(const nn_context* c, u64 na, u64 nb) {
  const u64 mn = std::min(na, nb), mx = std::max(na, nb);
  return mn < c->batch_ntt_min || (mn < c->batch_school_balanced && mx <= 2 * mn);
}

// J's pieces, plan and rows from its sizes (na >= nb) and `square`; one of a
// scale up to few_s takes that, and one of a scale up to `whole` its own, unsplit
// (0: none).
BatchRoute batch_route(const nn_context* c, nn::BatchJob& J, int few_s, int whole) {
  J.piece = J.na;
  J.pieces = 1;
  if (batch_columns(c, J.na, J.nb)) return BatchRoute::kColumns;
  int s = std::max(ntt_scale(J.na, J.nb), nn::kSixMinScale);
  // From this scale on one product fills the GPU by itself: no items, no
  // arena; the launch runs it alone.
  if (c->batch_solo_scale > 0 && s >= c->batch_solo_scale) return BatchRoute::kSolo;
  if (s <= few_s)
    s = few_s;
  else if (c->batch_split && !J.square && s > whole)
    s = six_split(J.na, J.nb, s, &J.piece, &J.pieces);
  if (s > nn::kSixMaxScale) return BatchRoute::kTooLong;
  J.plan = nn::six_plan(s, J.pieces > 1 ? 1ull << s : J.na + J.nb - 1, c->batch_r_last_at[s]);
  J.rows = J.pieces > 1 ? nn::kBatchRowsB : J.plan.n > 1 && !c->batch_fused ? nn::kBatchRowsAll : nn::kBatchRowsNone;
  return BatchRoute::kTransforms;
}
// Words of a transforms job's residues: operand 0's, and operand 1's where they are used.
u64 batch_words_a(const nn::BatchJob& J) { return J.pieces * (3ull << J.plan.s); }
u64 batch_words_b(const nn::BatchJob& J) { return !J.square && (J.plan.n > 1 || J.rows) ? 3ull << J.plan.s : 0; }

nn_status batch_plan(nn_context* c, nn_batch* B, const u64* na, const u64* nb, const int* square, u64 count) {
  if (count >= 0xffffffffull) {  // BatchItem::job is 32-bit
    c->err = "batch: too many products";
    return NN_ERR_INVALID;
  }
  B->count = count;
  B->na.assign(na, na + count);
  B->nb.assign(nb, nb + count);
  B->jobs.resize(count);
  B->off_a.assign(count, 0);
  B->off_b.assign(count, 0);
  B->swap.assign(count, 0);
  std::vector<u64> order;  // jobs with items
  int max_s = nn::kSixMinScale;
  // A few short products are bound by the number of launches, not by their
  // work: up to 152 jobs whose operands fit one pass take one scale, the
  // largest such one of the batch, so that their passes are one launch (six
  // CTAs a job, under a wave), and where the batch has launches of two passes
  // anyhow, products of up to 2^14 limbs are not split.  (Contexts with a budget,
  // or "batch_few" 0, keep the smaller arenas.)  With and without, us: 64 jobs of
  // 8 to 1024 limbs 38 and 45, one of 2000 x 2000 limbs beside 150 of 64 x 200 42
  // and 49, beside 150 of 500 x 500 42 and 54, 111 of 44 to 6439 limbs 114 and 140.
  // Unsplit by themselves five products of 16000 x 300 limbs take 79, split 32.
  constexpr int kOnePass = 12, kFewWhole = 14;
  const bool few = c->batch_few && count <= 152 && !c->budget;
  int few_s = 0, whole = 0;
  for (u64 j = 0; few && j < count; ++j) {
    const u64 mx = std::max(na[j], nb[j]), mn = std::min(na[j], nb[j]);
    if (!mn || mn < c->batch_ntt_min) continue;
    const int s = ntt_scale(mx, mn);
    if (s <= kOnePass) {
      few_s = std::max(few_s, s);
    } else if (!whole && (c->batch_solo_scale == 0 || s < c->batch_solo_scale)) {
      u64 piece, pieces = 1;
      if (c->batch_split && !(square && square[j])) six_split(mx, mn, s, &piece, &pieces);
      if (pieces == 1) whole = kFewWhole;
    }
  }
  for (u64 j = 0; j < count; ++j) {
    if (!na[j] || !nb[j]) {
      c->err = "batch: empty operand";
      return NN_ERR_INVALID;
    }
    nn::BatchJob& J = B->jobs[j];
    J = nn::BatchJob{};
    J.na = na[j];
    J.nb = nb[j];
    J.piece = na[j];
    J.pieces = 1;
    J.flag_base = B->n_flags;
    if (batch_columns(c, na[j], nb[j])) {
      B->n_flags += (nn::u32)((na[j] + nb[j] + nn::kBatchSumTile - 1) / nn::kBatchSumTile);
      order.push_back(j);
      continue;
    }
    J.square = square ? square[j] : 0;
    if (J.square && na[j] != nb[j]) {
      c->err = "batch: a square needs equal operand sizes";
      return NN_ERR_INVALID;
    }
    // operand 0 is the longer one; it may be split into pieces
    B->swap[j] = na[j] < nb[j];
    J.na = std::max(na[j], nb[j]);
    J.nb = std::min(na[j], nb[j]);
    const BatchRoute route = batch_route(c, J, few_s, whole);
    if (route == BatchRoute::kSolo) {
      B->solo.push_back(j);
      continue;
    }
    if (route == BatchRoute::kTooLong) {
      c->err = "batch: transform too long for one batch";
      return NN_ERR_INVALID;
    }
    max_s = std::max(max_s, J.plan.s);
    B->n_flags += (nn::u32)nn::scan_tiles(na[j] + nb[j]);
    B->off_a[j] = B->arena_words;
    B->arena_words += batch_words_a(J);
    if (const u64 words = batch_words_b(J)) {
      B->off_b[j] = B->arena_words;
      B->arena_words += words;
    }
    order.push_back(j);
  }
  // The longest jobs' items first in each launch, so that it ends with its
  // smallest; jobs of one scale one after another.
  std::stable_sort(order.begin(), order.end(), [&](u64 x, u64 y) { return B->jobs[x].plan.s > B->jobs[y].plan.s; });

  // One launch a (phase, kind, pass, R, block length): its items.
  std::map<std::array<int, 5>, std::vector<nn::BatchItem>> launches;
  for (u64 j : order) {
    const nn::BatchJob& J = B->jobs[j];
    const nn::SixPlan& pl = J.plan;
    auto item = [&](u64 tile, u64 ntile, int prime, int operand) {
      nn::BatchItem it{};
      it.job = (nn::u32)j;
      it.tile = (nn::u32)tile;
      it.ntile = (unsigned short)ntile;
      it.prime = (unsigned char)prime;
      it.operand = (unsigned char)operand;
      return it;
    };
    if (pl.s == 0) {
      auto& v = launches[{0, nn::kBatchColumns, 0, 0, 0}];
      for (u64 t = 0; t * nn::kBatchSumTile < J.na + J.nb; ++t) v.push_back(item(t, 1, 0, 0));
      continue;
    }
    const int m = pl.n;
    // items of pass k over operand 0's pieces (tiles numbered across them) or operand 1
    auto pass_items = [&](int phase, int kind, int k, int operand) {
      const bool row = k == m - 1;
      auto& v = launches[{phase, kind, row ? J.rows : k, pl.R[k], row ? pl.lgm : 0}];
      const u64 each = nn::batch_pass_tiles(pl, k), tiles = each * (operand == 0 ? J.pieces : 1);
      const u64 words = std::max<u64>((1ull << pl.s) / 8 * (k > 0 ? pl.k8 : 8) / each, 1);
      const u64 per = std::clamp<u64>(c->batch_item_words / words, 1, 0xffff);  // BatchItem::ntile is 16-bit
      for (u64 t = 0; t < tiles; t += per)  // the six primes of a tile's limbs or words one after another
        for (int pr = 0; pr < 6; ++pr) v.push_back(item(t, std::min(per, tiles - t), pr, operand));
    };
    const int operands = J.square ? 1 : 2;
    if (m == 1) {
      if (J.rows)
        for (int pr = 0; pr < 6; ++pr) launches[{3, nn::kBatchSmallRow, 0, pl.R[0], 0}].push_back(item(0, 1, pr, 1));
      auto& v = launches[{4, nn::kBatchSmall, J.rows, pl.R[0], 0}];
      for (u64 i = 0; i < J.pieces; ++i)
        for (int pr = 0; pr < 6; ++pr) v.push_back(item(i, 1, pr, 0));
    } else {
      for (int op = 0; op < operands; ++op) {
        pass_items(0, nn::kBatchLoad, 0, op);
        for (int k = 1; k < m - 1; ++k) pass_items(k, nn::kBatchCol, k, op);
        if (J.rows == nn::kBatchRowsAll || (J.rows && op == 1)) pass_items(3, nn::kBatchRow, m - 1, op);
      }
      pass_items(4, nn::kBatchFused, m - 1, 0);
      for (int k = m - 2; k >= 0; --k) pass_items(7 - k, nn::kBatchInvCol, k, 0);
    }
    auto& v = launches[{8, J.pieces > 1 ? nn::kBatchPieceCrt : nn::kBatchCrt, 0, 0, 0}];
    for (u64 t = 0; t < nn::scan_tiles(J.na + J.nb); ++t) v.push_back(item(t, 1, 0, 0));
  }
  u64 total = 0;
  for (const auto& [key, v] : launches) total += v.size();
  B->items.reserve(total);
  for (auto& [key, v] : launches) {
    if (B->items.size() + v.size() >= 0xffffffffull) {
      c->err = "batch: too many work items";
      return NN_ERR_INVALID;
    }
    B->segments.push_back({key[0], key[1], key[2], key[3], key[4], (nn::u32)B->items.size(), (nn::u32)v.size()});
    B->items.insert(B->items.end(), v.begin(), v.end());
  }
  NN_CK(c, nn::six_tables_ensure(c->six, max_s, c->stream, &c->retired_tables), "twiddle tables");
  // Regions in one allocation, each rounded to 256 bytes: the residues are
  // read and written with 16-byte vector accesses.
  auto words = [](u64 bytes) { return (bytes + 255) / 256 * 32; };
  const u64 w_jobs = words(count * sizeof(nn::BatchJob)), w_items = words(B->items.size() * sizeof(nn::BatchItem)),
            w_state = words(4ull * (B->segments.size() + B->n_flags + 2));
  u64* p = nullptr;
  B->dev_words = w_jobs + w_items + w_state + B->arena_words;
  nn_status st = dev_alloc(c, &p, B->dev_words);
  if (st != NN_OK) return st;
  B->d_jobs = reinterpret_cast<nn::BatchJob*>(p);
  B->d_items = reinterpret_cast<nn::BatchItem*>(p + w_jobs);
  B->d_state = reinterpret_cast<nn::u32*>(p + w_jobs + w_items);
  B->d_arena = p + w_jobs + w_items + w_state;
  NN_CK(c, c->stage.upload(B->d_items, B->items.data(), B->items.size() * sizeof(nn::BatchItem), c->stream),
        "upload items");
  NN_CK(c, cudaEventCreateWithFlags(&B->ran, cudaEventDisableTiming), "event");
  return NN_OK;
}

// The run's launches on `st` (after the job table's upload): counters and
// status words cleared, then phase by phase; with `side` streams, the launches
// of one phase side by side.
cudaError_t batch_sequence(nn_context* c, nn_batch* B, cudaStream_t st, cudaStream_t* side = nullptr, int n_side = 0,
                           cudaEvent_t ev = nullptr) {
  const u64 n = B->segments.size();
  cudaError_t e = cudaMemsetAsync(B->d_state, 0, (n + B->n_flags + 2) * 4, st);
  nn::u32* flags = B->d_state + n;
  for (u64 i = 0; i < n && e == cudaSuccess;) {
    u64 end = i + 1;
    while (end < n && B->segments[end].phase == B->segments[i].phase) ++end;
    const int used = (int)std::min<u64>(end - i - 1, n_side);  // side streams of this phase
    if (used) e = cudaEventRecord(ev, st);
    for (int k = 0; k < used && e == cudaSuccess; ++k) e = cudaStreamWaitEvent(side[k], ev, 0);
    for (u64 g = i; g < end && e == cudaSuccess; ++g) {
      const int lane = (int)((g - i) % (used + 1));
      const cudaStream_t s = lane ? side[lane - 1] : st;
      if (!side) nn::launch_begin("batch_launch", s);
      e = nn::batch_launch_segment(B->segments[g], B->d_jobs, B->d_items, B->d_state + g, flags, c->scan.err, c->six, s);
      if (!side) nn::launch_end(s);
    }
    for (int k = 0; k < used && e == cudaSuccess; ++k) {
      e = cudaEventRecord(ev, side[k]);
      if (e == cudaSuccess) e = cudaStreamWaitEvent(st, ev, 0);
    }
    i = end;
  }
  return e;
}

nn_status side_streams(nn_context* c) {
  for (cudaStream_t& s : c->side)
    if (!s) NN_CK(c, cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking), "side stream");
  if (!c->ev_side) NN_CK(c, cudaEventCreateWithFlags(&c->ev_side, cudaEventDisableTiming), "event");
  return NN_OK;
}

// Records the run (job table upload, then batch_sequence) into a CUDA graph.
nn_status batch_capture(nn_context* c, nn_batch* B) {
  cudaStream_t cs = c->own;
  cudaError_t e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
  if (e == cudaSuccess) {
    cudaError_t le =
        cudaMemcpyAsync(B->d_jobs, B->h_jobs, B->count * sizeof(nn::BatchJob), cudaMemcpyHostToDevice, cs);
    if (le == cudaSuccess) le = batch_sequence(c, B, cs, c->side, c->kSide, c->ev_side);
    e = cudaStreamEndCapture(cs, &B->graph);
    if (le != cudaSuccess) e = le;
  }
  if (e == cudaSuccess) e = cudaGraphInstantiate(&B->exec, B->graph, 0);
  NN_CK(c, e, "batch graph");
  return NN_OK;
}

void batch_release(nn_context* c, nn_batch* B) {
  if (B->pending) cudaEventSynchronize(B->ran);
  if (B->exec) cudaGraphExecDestroy(B->exec);
  if (B->graph) cudaGraphDestroy(B->graph);
  if (B->ran) cudaEventDestroy(B->ran);
  if (B->h_jobs) cudaFreeHost(B->h_jobs);
  dev_free(c, reinterpret_cast<u64*>(B->d_jobs), B->dev_words);
  delete B;
}

u64 normalized(const u64* x, u64 n) {  // natural::std (natural.h:82-93)
  while (n > 1 && x[n - 1] == 0) --n;
  return n;
}

}  // namespace

// Context access for the other host translation units (context_access.h).
namespace nn {
cudaStream_t ctx_stream(nn_context* c) { return c->stream; }
Scan& ctx_scan(nn_context* c) { return c->scan; }
nn_status ctx_alloc(nn_context* c, u64** p, u64 words) { return dev_alloc(c, p, words); }
void ctx_free(nn_context* c, u64* p, u64 words) { dev_free(c, p, words); }
nn_status ctx_mul(nn_context* c, u64* out, const u64* a, u64 na, const u64* b, u64 nb) {
  return mul_impl(c, out, a, na, b, nb);
}
nn_status ctx_fail(nn_context* c, cudaError_t e, const char* what) { return fail(c, e, what); }
cudaError_t ctx_upload(nn_context* c, void* d_dst, const void* h_src, u64 bytes) {
  return c->stage.upload(d_dst, h_src, bytes, c->stream);
}
void ctx_error(nn_context* c, const char* msg) { c->err = msg; }
nn_status ctx_scratch(nn_context* c, int slot, u64 words, u64** p) { return scratch(c, slot, words, p); }
u64 ctx_batch_job_bytes(const nn_context* c, u64 na, u64 nb) {
  BatchJob J{};
  J.na = std::max(na, nb);
  J.nb = std::min(na, nb);
  if (batch_route(c, J, 0, 0) != BatchRoute::kTransforms) return (na + nb) / 16;  // an item and a flag a tile
  const u64 bytes = 8 * (batch_words_a(J) + batch_words_b(J));
  return bytes + bytes / 512;  // its items: 12 bytes for 8192 words of a prime, a pass
}
}  // namespace nn

extern "C" {

const char* nn_status_string(nn_status s) {
  switch (s) {
    case NN_OK: return "ok";
    case NN_ERR_INVALID: return "invalid argument";
    case NN_ERR_OOM: return "device out of memory";
    case NN_ERR_CUDA: return "CUDA error";
    case NN_ERR_TIMEOUT: return "device wait timed out";
    case NN_ERR_BUDGET: return "HBM budget exceeded";
    case NN_ERR_NO_DEVICE: return "no CUDA device";
  }
  return "unknown";
}

uint64_t nn_launch_count(void) { return nn::launch_count(); }

void nn_profile_enable(int on) { nn::profile_enable(on != 0); }

uint64_t nn_profile_report(char* buf, uint64_t cap) {
  std::string r = nn::profile_report();
  if (buf && cap) {
    u64 n = std::min<u64>(cap - 1, r.size());
    std::memcpy(buf, r.data(), n);
    buf[n] = 0;
  }
  return r.size();
}

// The tunables autotune.py measured on this GPU model (the "tunables" object
// of tuning.json: "name": integer pairs), applied to every new context, so
// that contexts made through the C ABI (the drop-in header's, the request
// server's) run the same tuned pass splits and batch shapes as Python ones.
// The file: $NN_TUNING ("off": none), else tuning.json in the directory above
// the one holding this library.  A missing or unreadable file leaves the
// defaults.
static void apply_tuning_file(nn_context* c) {
  std::string path;
  if (const char* e = std::getenv("NN_TUNING")) {
    if (std::strcmp(e, "off") == 0) return;
    path = e;
  } else {
    Dl_info info{};
    if (!dladdr(reinterpret_cast<void*>(&apply_tuning_file), &info) || !info.dli_fname) return;
    std::string lib(info.dli_fname);
    const size_t slash = lib.rfind('/');
    const std::string dir = slash == std::string::npos ? "." : lib.substr(0, slash);
    path = dir + "/../tuning.json";
  }
  FILE* f = std::fopen(path.c_str(), "rb");
  if (!f) return;
  std::string text;
  char buf[4096];
  for (size_t n; (n = std::fread(buf, 1, sizeof buf, f)) > 0;) text.append(buf, n);
  std::fclose(f);
  size_t at = text.find("\"tunables\"");
  if (at == std::string::npos) return;
  at = text.find('{', at);
  const size_t end = at == std::string::npos ? at : text.find('}', at);
  if (end == std::string::npos) return;
  for (size_t q = text.find('"', at); q != std::string::npos && q < end; q = text.find('"', q)) {
    const size_t q2 = text.find('"', q + 1);
    if (q2 == std::string::npos || q2 > end) break;
    const std::string key = text.substr(q + 1, q2 - q - 1);
    const size_t colon = text.find(':', q2);
    if (colon == std::string::npos || colon > end) break;
    char* stop = nullptr;
    const long long v = std::strtoll(text.c_str() + colon + 1, &stop, 10);
    if (stop != text.c_str() + colon + 1) nn_context_set_tunable(c, key.c_str(), v);
    q = stop ? (size_t)(stop - text.c_str()) : colon + 1;
  }
  c->err.clear();  // an unknown key from another version is not an error of this context
}

nn_status nn_context_create(int device, uint64_t budget, nn_context** out) {
  if (!out) return NN_ERR_INVALID;
  *out = nullptr;
  int count = 0;
  if (cudaGetDeviceCount(&count) != cudaSuccess || count <= device || device < 0) {
    cudaGetLastError();
    return NN_ERR_NO_DEVICE;
  }
  nn_context* c = new nn_context;
  c->device = device;
  c->budget = budget;
  cudaError_t e = cudaSetDevice(device);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&c->own, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&c->copy, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&c->ev_first, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&c->ev_second, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&c->ev_chunk, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&c->ev_in, cudaEventDisableTiming);
  if (e == cudaSuccess) e = nn::upload_primes();
  if (e == cudaSuccess) {
    cudaMemPool_t pool;
    e = cudaDeviceGetDefaultMemPool(&pool, device);
    if (e == cudaSuccess) {
      uint64_t keep = ~0ull;  // keep freed blocks cached for reuse
      e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    }
  }
  if (e == cudaSuccess) e = nn::scan_reserve(c->scan, 1024);
  c->tables.err = c->scan.err;
  if (e != cudaSuccess) {
    nn_status st = e == cudaErrorNoDevice || e == cudaErrorNoKernelImageForDevice ? NN_ERR_NO_DEVICE : NN_ERR_CUDA;
    cudaGetLastError();
    if (c->ev_in) cudaEventDestroy(c->ev_in);
    if (c->ev_chunk) cudaEventDestroy(c->ev_chunk);
    if (c->ev_second) cudaEventDestroy(c->ev_second);
    if (c->ev_first) cudaEventDestroy(c->ev_first);
    if (c->copy) cudaStreamDestroy(c->copy);
    if (c->own) cudaStreamDestroy(c->own);
    delete c;
    return st;
  }
  c->stream = c->own;
  apply_tuning_file(c);
  *out = c;
  return NN_OK;
}

nn_status nn_context_destroy(nn_context* c) {
  if (!c) return NN_ERR_INVALID;
  cudaSetDevice(c->device);
  // Work the caller ordered on its own stream must be finished (or that
  // stream still alive); teardown itself only uses the context's stream.
  if (c->stream != c->own) cudaStreamSynchronize(c->stream);
  c->stream = c->own;
  cudaStreamSynchronize(c->own);
  for (int i = 0; i < 3; ++i) dev_free(c, c->scratch[i], c->scratch_words[i]);
  cudaStreamSynchronize(c->own);
  nn::tables_free(c->tables);
  nn::six_tables_free(c->six);
  for (u64* p : c->retired_tables) cudaFree(p);
  c->retired_tables.clear();
  nn::scan_free(c->scan);
  c->stage.release();
  cudaStreamSynchronize(c->copy);
  for (cudaStream_t s : c->side)
    if (s) cudaStreamSynchronize(s), cudaStreamDestroy(s);
  if (c->ev_side) cudaEventDestroy(c->ev_side);
  cudaEventDestroy(c->ev_in);
  cudaEventDestroy(c->ev_chunk);
  cudaEventDestroy(c->ev_second);
  cudaEventDestroy(c->ev_first);
  cudaStreamDestroy(c->copy);
  if (c->own) cudaStreamDestroy(c->own);
  delete c;
  return NN_OK;
}

nn_status nn_context_set_stream(nn_context* c, void* s) {
  if (!c) return NN_ERR_INVALID;
  c->stream = (cudaStream_t)s;  // NULL is the legacy default stream, as in CUDA
  return NN_OK;
}

nn_status nn_context_use_own_stream(nn_context* c) {
  if (!c) return NN_ERR_INVALID;
  c->stream = c->own;
  return NN_OK;
}

void* nn_context_stream(nn_context* c) { return c ? (void*)c->stream : nullptr; }

nn_status nn_context_synchronize(nn_context* c) {
  if (!c) return NN_ERR_INVALID;
  NN_CK(c, cudaStreamSynchronize(c->stream), "synchronize");
  nn::u32 err = 0;
  NN_CK(c, cudaMemcpy(&err, c->scan.err, sizeof err, cudaMemcpyDeviceToHost), "read error flag");
  if (err) {
    cudaMemset(c->scan.err, 0, sizeof err);
    c->err = "carry lookback wait exceeded its bound";
    return NN_ERR_TIMEOUT;
  }
  return NN_OK;
}

nn_status nn_context_probe_wait(nn_context* c, int spin_limit) {
  if (!c || spin_limit < 0) return NN_ERR_INVALID;
  NN_CK(c, nn::wait_probe(c->scan, spin_limit, c->stream), "wait probe");
  return nn_context_synchronize(c);
}

const char* nn_last_error(const nn_context* c) { return c ? c->err.c_str() : "no context"; }

uint64_t nn_context_device_bytes(const nn_context* c) {
  if (!c) return 0;
  return c->held + 2 * 3 * c->tables.cap * sizeof(u64) + 2 * 6 * c->six.cap * sizeof(int2) +
         c->scan.held_tiles * 4;
}

nn_status nn_transform_create(nn_context* c, nn_transform** out) {
  if (!c || !out) return NN_ERR_INVALID;
  *out = new nn_transform;
  return NN_OK;
}

nn_status nn_transform_destroy(nn_context* c, nn_transform* t) {
  if (!c || !t) return NN_ERR_INVALID;
  dev_free(c, t->res, t->words);
  delete t;
  return NN_OK;
}

int nn_transform_scale(const nn_transform* t) { return t ? t->scale : 0; }
void nn_transform_set_scale(nn_transform* t, int s) {
  if (t) t->scale = s;
}

nn_status nn_transform_forward(nn_context* c, nn_transform* t, const uint64_t* d, uint64_t n, int s) {
  if (!c || !t || !d) return NN_ERR_INVALID;
  return forward(c, t, d, n, s);
}

nn_status nn_transform_pointwise(nn_context* c, nn_transform* dst, const nn_transform* a, const nn_transform* b) {
  if (!c || !dst || !a || !b || !a->res || !b->res) return NN_ERR_INVALID;
  return pointwise(c, dst, a, b);
}

nn_status nn_transform_inverse_save(nn_context* c, nn_transform* t, uint64_t* d_out, uint64_t size,
                                    uint64_t* written) {
  if (!c || !t || !t->res || !d_out) return NN_ERR_INVALID;
  return inverse_save(c, t, d_out, size, written);
}

nn_status nn_transform_residues(nn_context* c, const nn_transform* t, uint64_t* d_out) {
  if (!c || !t || !t->res || !d_out) return NN_ERR_INVALID;
  if (t->rep == nn_transform::kThree || !(reinterpret_cast<std::uintptr_t>(d_out) & 15)) return three_words(c, t, d_out);
  // the passes read and write 16 bytes at a time
  DBuf tmp(c);
  const u64* words = nullptr;
  const nn_status st = three_operand(c, t, tmp, &words);
  if (st != NN_OK) return st;
  NN_CK(c, cudaMemcpyAsync(d_out, words, (3ull << t->scale) * sizeof(u64), cudaMemcpyDeviceToDevice, c->stream),
        "copy residues");
  return NN_OK;
}

nn_status nn_mul(nn_context* c, uint64_t* d_out, const uint64_t* a, uint64_t na, const uint64_t* b, uint64_t nb) {
  if (!c) return NN_ERR_INVALID;
  return mul_impl(c, d_out, a, na, b, nb);
}

nn_status nn_sqr(nn_context* c, uint64_t* d_out, const uint64_t* a, uint64_t n) {
  if (!c) return NN_ERR_INVALID;
  return sqr_impl(c, d_out, a, n);
}

nn_status nn_ntt_mul(nn_context* c, uint64_t* d_out, const uint64_t* a, uint64_t na, const uint64_t* b, uint64_t nb,
                     int s, uint64_t size, uint64_t* written) {
  if (!c || !d_out || !a || !b) return NN_ERR_INVALID;
  return ntt_product(c, d_out, a, na, b, nb, s, size, written);
}

nn_status nn_mul_base(nn_context* c, uint64_t* d_out, const uint64_t* a, uint64_t na, const uint64_t* b,
                      uint64_t nb) {
  if (!c || !d_out || !a || !b || !na || !nb) return NN_ERR_INVALID;
  return base_product(c, d_out, a, na, b, nb);
}

nn_status nn_mul_host(nn_context* c, uint64_t* out, uint64_t* out_n, const uint64_t* a, uint64_t na,
                      const uint64_t* b, uint64_t nb) {
  if (!c || !out || !a || !b || !na || !nb) return NN_ERR_INVALID;
  if (na < nb) {  // the longer operand first: it is transformed first
    std::swap(a, b);
    std::swap(na, nb);
  }
  // Copies, not kernels reading and writing page-locked host memory in
  // place: measured on GB300 at 2^27 limbs, in-place access over the host
  // link made the product 7 to 95 ms slower than these copies.
  u64 *da, *db, *dout;
  nn_status st = scratch(c, 0, na, &da);
  if (st == NN_OK) st = scratch(c, 1, nb, &db);
  if (st == NN_OK) st = scratch(c, 2, na + nb, &dout);
  if (st != NN_OK) return st;
  u64 piece, pieces;
  const bool chunked = na + nb > kChunkedLimbs && nb >= kNttMulThreshold && page_locked(a) && page_locked(b) &&
                       page_locked(out);
  const int s = chunked ? six_split(na, nb, ntt_scale(na, nb), &piece, &pieces) : 0;
  if (s && s <= nn::kSixMaxScale && pieces == 1) {
    bool used = false;
    st = six_product_from_host(c, dout, da, a, na, db, b, nb, s, out, &used);
    if (used) {
      if (st == NN_OK) st = nn_context_synchronize(c);
      const cudaError_t e = cudaStreamSynchronize(c->copy);
      if (st == NN_OK && e != cudaSuccess) st = fail(c, e, "copy-back");
      if (st == NN_OK && out_n) *out_n = normalized(out, na + nb);
      return st;
    }
    if (st != NN_OK) return st;
  }
  NN_CK(c, cudaMemcpyAsync(da, a, na * 8, cudaMemcpyHostToDevice, c->stream), "H2D");
  NN_CK(c, cudaMemcpyAsync(db, b, nb * 8, cudaMemcpyHostToDevice, c->stream), "H2D");
  st = mul_impl(c, dout, da, na, db, nb);
  if (st != NN_OK) return st;
  NN_CK(c, cudaMemcpyAsync(out, dout, (na + nb) * 8, cudaMemcpyDeviceToHost, c->stream), "D2H");
  st = nn_context_synchronize(c);
  if (st == NN_OK && out_n) *out_n = normalized(out, na + nb);
  return st;
}

nn_status nn_sqr_host(nn_context* c, uint64_t* out, uint64_t* out_n, const uint64_t* a, uint64_t n) {
  if (!c || !out || !a || !n) return NN_ERR_INVALID;
  u64 *da, *dout;
  nn_status st = scratch(c, 0, n, &da);
  if (st == NN_OK) st = scratch(c, 2, 2 * n, &dout);
  if (st != NN_OK) return st;
  NN_CK(c, cudaMemcpyAsync(da, a, n * 8, cudaMemcpyHostToDevice, c->stream), "H2D");
  st = sqr_impl(c, dout, da, n);
  if (st != NN_OK) return st;
  NN_CK(c, cudaMemcpyAsync(out, dout, 2 * n * 8, cudaMemcpyDeviceToHost, c->stream), "D2H");
  st = nn_context_synchronize(c);
  if (st == NN_OK && out_n) *out_n = normalized(out, 2 * n);
  return st;
}

nn_status nn_mul_base_host(nn_context* c, uint64_t* out, const uint64_t* a, uint64_t na, const uint64_t* b,
                           uint64_t nb) {
  if (!c || !out || !a || !b || !na || !nb) return NN_ERR_INVALID;
  u64 *da, *db, *dout;
  nn_status st = scratch(c, 0, na, &da);
  if (st == NN_OK) st = scratch(c, 1, nb, &db);
  if (st == NN_OK) st = scratch(c, 2, na + nb, &dout);
  if (st != NN_OK) return st;
  NN_CK(c, cudaMemcpyAsync(da, a, na * 8, cudaMemcpyHostToDevice, c->stream), "H2D");
  NN_CK(c, cudaMemcpyAsync(db, b, nb * 8, cudaMemcpyHostToDevice, c->stream), "H2D");
  NN_CK(c, nn::school_mul(da, na, db, nb, dout, c->scan, c->stream), "base-case product");
  NN_CK(c, cudaMemcpyAsync(out, dout, (na + nb) * 8, cudaMemcpyDeviceToHost, c->stream), "D2H");
  return nn_context_synchronize(c);
}

nn_status nn_transform_forward_host(nn_context* c, nn_transform* t, const uint64_t* limbs, uint64_t n, int s) {
  if (!c || !t || !limbs || !n) return NN_ERR_INVALID;
  u64* d;
  nn_status st = scratch(c, 0, n, &d);
  if (st != NN_OK) return st;
  NN_CK(c, cudaMemcpyAsync(d, limbs, n * 8, cudaMemcpyHostToDevice, c->stream), "H2D");
  return forward(c, t, d, n, s);
}

nn_status nn_transform_inverse_save_host(nn_context* c, nn_transform* t, uint64_t* out, uint64_t size,
                                         uint64_t* written) {
  if (!c || !t || !t->res || !out) return NN_ERR_INVALID;
  const u64 L = 1ull << t->scale;
  u64* d;
  nn_status st = scratch(c, 2, std::max<u64>(size, L), &d);
  if (st != NN_OK) return st;
  u64 w = 0;
  st = inverse_save(c, t, d, size, &w);
  if (st != NN_OK) return st;
  NN_CK(c, cudaMemcpyAsync(out, d, w * 8, cudaMemcpyDeviceToHost, c->stream), "D2H");
  st = nn_context_synchronize(c);
  if (written) *written = w;
  return st;
}

nn_status nn_context_set_tunable(nn_context* c, const char* name, int64_t v) {
  if (!c || !name) return NN_ERR_INVALID;
  std::string k(name);
  const size_t at = k.find('@');
  if (at != std::string::npos) {  // per-scale pass split: "r_last@28", "r_col@28", "batch_r_last@16"
    const std::string base = k.substr(0, at);
    const int sc = std::atoi(k.c_str() + at + 1);
    const bool rl = base == "r_last" || base == "batch_r_last";
    if (sc >= 2 && sc < 64 && ((rl && (v == 0 || (v >= 3 && v <= 12))) || (base == "r_col" && v >= 0 && v <= 9))) {
      (base == "r_last" ? c->r_last_at : base == "r_col" ? c->r_col_at : c->batch_r_last_at)[sc] = (int)v;
      return NN_OK;
    }
    c->err = "unknown tunable or value out of range: " + k;
    return NN_ERR_INVALID;
  }
  if (k == "r_last" && v >= 3 && v <= 12)
    c->r_last = (int)v;
  else if (k == "r_col" && v >= 1 && v <= 9)
    c->r_col = (int)v;
  else if (k == "batch_ntt_min" && v >= 1)
    c->batch_ntt_min = (u64)v;
  else if (k == "batch_item_words" && v >= 1 && v <= (1 << 20))
    c->batch_item_words = (u64)v;
  else if (k == "batch_fused" && (v == 0 || v == 1))
    c->batch_fused = (int)v;
  else if (k == "batch_merge" && (v == 0 || v == 1))
    c->batch_merge = (int)v;
  else if (k == "batch_split" && (v == 0 || v == 1))
    c->batch_split = (int)v;
  else if (k == "batch_blocks_per_sm" && v >= 0 && v <= 32)
    c->batch_blocks_per_sm = (int)v;
  else if (k == "batch_solo_scale" && (v == 0 || (v >= 2 && v < 64)))
    c->batch_solo_scale = (int)v;
  else if (k == "batch_few" && (v == 0 || v == 1))
    c->batch_few = (int)v;
  else if (k == "batch_school_balanced" && v >= 0)
    c->batch_school_balanced = (u64)v;
  else {
    c->err = "unknown tunable or value out of range: " + k;
    return NN_ERR_INVALID;
  }
  return NN_OK;
}

int64_t nn_context_get_tunable(const nn_context* c, const char* name) {
  if (!c || !name) return -1;
  std::string k(name);
  const size_t at = k.find('@');
  if (at != std::string::npos) {
    const int sc = std::atoi(k.c_str() + at + 1);
    if (sc < 2 || sc >= 64) return -1;
    if (k.substr(0, at) == "r_last") return c->r_last_at[sc];
    if (k.substr(0, at) == "r_col") return c->r_col_at[sc];
    if (k.substr(0, at) == "batch_r_last") return c->batch_r_last_at[sc];
    return -1;
  }
  if (k == "r_last") return c->r_last;
  if (k == "r_col") return c->r_col;
  if (k == "batch_ntt_min") return (int64_t)c->batch_ntt_min;
  if (k == "batch_item_words") return (int64_t)c->batch_item_words;
  if (k == "batch_fused") return (int64_t)c->batch_fused;
  if (k == "batch_merge") return (int64_t)c->batch_merge;
  if (k == "batch_split") return (int64_t)c->batch_split;
  if (k == "batch_blocks_per_sm") return c->batch_blocks_per_sm;
  if (k == "batch_solo_scale") return c->batch_solo_scale;
  if (k == "batch_few") return c->batch_few;
  if (k == "batch_school_balanced") return (int64_t)c->batch_school_balanced;
  return -1;
}

nn_status nn_batch_create(nn_context* c, const uint64_t* na, const uint64_t* nb, const int* square, uint64_t count,
                          nn_batch** out) {
  if (!c || !na || !nb || !count || !out) return NN_ERR_INVALID;
  *out = nullptr;
  nn_batch* B = new nn_batch;
  nn_status st = batch_plan(c, B, na, nb, square, count);
  if (st != NN_OK) {
    batch_release(c, B);
    return st;
  }
  *out = B;
  return NN_OK;
}

}  // extern "C"

namespace {  // helpers of the batch entry points, not exported

// Fills a job table (the plan's pinned one, or `into`) for one run.
nn_status batch_fill(nn_context* c, nn_batch* B, const nn_mul_job* jobs, nn::BatchJob* into = nullptr) {
  nn::BatchJob* dst = into ? into : B->h_jobs;
  for (u64 j = 0; j < B->count; ++j) {
    if (jobs[j].n_a != B->na[j] || jobs[j].n_b != B->nb[j] || !jobs[j].d_a || !jobs[j].d_b || !jobs[j].d_out) {
      c->err = "batch run: job does not match the plan";
      return NN_ERR_INVALID;
    }
    nn::BatchJob J = B->jobs[j];
    J.a = B->swap[j] ? jobs[j].d_b : jobs[j].d_a;
    J.b = B->swap[j] ? jobs[j].d_a : jobs[j].d_b;
    J.out = jobs[j].d_out;
    J.res_a = reinterpret_cast<nn::u32*>(B->d_arena + B->off_a[j]);
    J.res_b = reinterpret_cast<nn::u32*>(B->d_arena + B->off_b[j]);
    dst[j] = J;
  }
  return NN_OK;
}

// The plan's large products, one at a time on the context's stream.
nn_status batch_solo(nn_context* c, const nn_batch* B, const nn_mul_job* jobs) {
  for (u64 j : B->solo) {
    const nn_mul_job& m = jobs[j];
    const nn_status st = B->jobs[j].square ? sqr_impl(c, m.d_out, m.d_a, m.n_a)
                                           : mul_impl(c, m.d_out, m.d_a, m.n_a, m.d_b, m.n_b);
    if (st != NN_OK) return st;
  }
  return NN_OK;
}

}  // namespace

extern "C" {

nn_status nn_batch_launch(nn_context* c, nn_batch* B, const nn_mul_job* jobs) {
  if (!c || !B || !jobs) return NN_ERR_INVALID;
  if (B->pending) NN_CK(c, cudaEventSynchronize(B->ran), "previous batch run");
  // The table goes up through the context's page-locked ring: the call
  // returns without waiting for the stream's earlier work.
  std::vector<nn::BatchJob> table(B->count);
  nn_status st = batch_fill(c, B, jobs, table.data());
  if (st != NN_OK) return st;
  if (!B->items.empty()) {
    NN_CK(c, c->stage.upload(B->d_jobs, table.data(), B->count * sizeof(nn::BatchJob), c->stream), "upload jobs");
    const cudaError_t le = batch_sequence(c, B, c->stream);
    NN_CK(c, le, "batch launch");
  }
  st = batch_solo(c, B, jobs);
  if (st != NN_OK) return st;
  NN_CK(c, cudaEventRecord(B->ran, c->stream), "event record");
  B->pending = true;
  return NN_OK;
}

// A plan's first run goes launch by launch, later ones as a graph: making that
// costs more than it saves one run.  Plan, run and release together, us, first run
// as a graph / so: one product of 8 to 1024 limbs 180 / 40, 153 of them 272 / 98,
// 400 of 300 to 5000 507 / 274, 4096 of 64 to 2^18 20080 / 19870.
nn_status nn_batch_run(nn_context* c, nn_batch* B, const nn_mul_job* jobs) {
  if (!c || !B || !jobs) return NN_ERR_INVALID;
  if (B->pending) NN_CK(c, cudaEventSynchronize(B->ran), "previous batch run");
  nn_status st = B->items.empty() ? NN_OK : side_streams(c);
  if (st != NN_OK) return st;
  const bool direct = !B->started && !capturing(c);
  B->started = true;
  std::vector<nn::BatchJob> table(direct ? B->count : 0);
  if (!direct && !B->h_jobs)  // pinned, so the graph's upload node can read it at replay time
    NN_CK(c, cudaHostAlloc((void**)&B->h_jobs, B->count * sizeof(nn::BatchJob), cudaHostAllocDefault),
          "pinned jobs");
  st = batch_fill(c, B, jobs, direct ? table.data() : nullptr);
  if (st != NN_OK) return st;
  if (!B->items.empty()) {
    if (!direct && !B->exec) {
      st = batch_capture(c, B);
      if (st != NN_OK) return st;
    }
    if (direct)
      NN_CK(c, c->stage.upload(B->d_jobs, table.data(), B->count * sizeof(nn::BatchJob), c->stream), "upload jobs");
    nn::launch_begin(direct ? "batch_launches" : "batch_graph", c->stream);
    const cudaError_t e = direct ? batch_sequence(c, B, c->stream, c->side, c->kSide, c->ev_side)
                                 : cudaGraphLaunch(B->exec, c->stream);
    nn::launch_end(c->stream);
    if (direct && e != cudaSuccess)  // what has started beside the stream is not behind it
      for (cudaStream_t s : c->side) cudaStreamSynchronize(s);
    NN_CK(c, e, "batch run");
  }
  st = batch_solo(c, B, jobs);
  if (st != NN_OK) return st;
  NN_CK(c, cudaEventRecord(B->ran, c->stream), "event record");
  B->pending = true;
  return NN_OK;
}

nn_status nn_batch_destroy(nn_context* c, nn_batch* B) {
  if (!c || !B) return NN_ERR_INVALID;
  batch_release(c, B);
  return NN_OK;
}

uint64_t nn_batch_items(const nn_batch* B) { return B ? B->items.size() : 0; }

nn_status nn_mul_each(nn_context* c, const nn_mul_job* jobs, uint64_t count) {
  if (!c || !jobs) return NN_ERR_INVALID;
  for (u64 j = 0; j < count; ++j) {
    nn_status st = mul_impl(c, jobs[j].d_out, jobs[j].d_a, jobs[j].n_a, jobs[j].d_b, jobs[j].n_b);
    if (st != NN_OK) return st;
  }
  return NN_OK;
}

nn_status nn_batch_mul(nn_context* c, const nn_mul_job* jobs, uint64_t count) {
  if (!c || !jobs || !count) return NN_ERR_INVALID;
  std::vector<u64> na(count), nb(count);
  std::vector<int> sq(count);
  for (u64 j = 0; j < count; ++j) {
    na[j] = jobs[j].n_a;
    nb[j] = jobs[j].n_b;
    sq[j] = jobs[j].d_a == jobs[j].d_b && na[j] == nb[j];
  }
  nn_batch* B = nullptr;
  nn_status st = nn_batch_create(c, na.data(), nb.data(), sq.data(), count, &B);
  if (st != NN_OK) return st;
  st = nn_batch_run(c, B, jobs);
  batch_release(c, B);
  return st;
}

nn_context* nn_default_context(void) {
  static nn_context* ctx = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    int dev = 0;
    cudaGetDevice(&dev);
    if (nn_context_create(dev, 0, &ctx) != NN_OK) ctx = nullptr;
  }
  return ctx;
}

}  // extern "C"
