// Host engine of the GB300 row-boundary contraction and the C ABI of
// include/qpeps.h.
//
// Mirrors the reference's drivers:
//   contract_rows(n)                       src/lib.rs:758 -> 784 -> 5287-5415
//   CompiledRowOperator::compile           src/lib.rs:430-485
//   top-row vertical-reflection orbits     src/lib.rs:721-749
//   known_count                            src/lib.rs:5752-5784
//   CRT certificate (product > N!)         src/lib.rs:3859-3886, 4134-4163
// with the row loop's expand/sort/reduce replaced by device kernels over an
// HBM-resident boundary store.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <map>
#include <mutex>
#include <new>
#include <string>
#include <thread>
#include <vector>

#include "../../include/qpeps.h"
#include "qpeps_device.cuh"
#include "qpeps_internal.h"

namespace qpeps {

// ---------------------------------------------------------------------------
// Errors

struct Failure {
  int code;
  std::string msg;
};

[[noreturn]] static void fail(int code, const std::string& msg) { throw Failure{code, msg}; }

static void cuda_check(cudaError_t e, const char* what) {
  if (e == cudaSuccess) return;
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    fail(QPEPS_ERR_OOM, std::string("device allocation failed: ") + what);
  }
  fail(QPEPS_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

static std::string row_msg(const char* prefix, unsigned row) {
  char buf[96];
  std::snprintf(buf, sizeof buf, "%s %u", prefix, row);
  return buf;
}

// ---------------------------------------------------------------------------
// u128 helpers

static bool add_u128(u128 a, u128 b, u128* out) {
  u128 s = a + b;
  if (s < a) return false;
  *out = s;
  return true;
}
static bool mul_u128(u128 a, u128 b, u128* out) {
  if (a == 0 || b == 0) {
    *out = 0;
    return true;
  }
  u128 p = a * b;
  if (p / a != b) return false;
  *out = p;
  return true;
}
static qpeps_u128 to_abi(u128 v) { return qpeps_u128{(uint64_t)v, (uint64_t)(v >> 64)}; }

// ---------------------------------------------------------------------------
// Local tensor C from B (Sec. VI, Eq. 16-18) and its certification.

struct Legs {
  uint8_t ci, co, ri, ro, dri, dro, dli, dlo;
};

static unsigned legs_key(const Legs& l) {
  return l.ci | (l.co << 1) | (l.ri << 2) | (l.ro << 3) | (l.dri << 4) | (l.dro << 5) | (l.dli << 6) | (l.dlo << 7);
}
static Legs legs_from_key(unsigned k) {
  return Legs{(uint8_t)(k & 1),        (uint8_t)((k >> 1) & 1), (uint8_t)((k >> 2) & 1), (uint8_t)((k >> 3) & 1),
              (uint8_t)((k >> 4) & 1), (uint8_t)((k >> 5) & 1), (uint8_t)((k >> 6) & 1), (uint8_t)((k >> 7) & 1)};
}

struct CEntryH {
  unsigned legs;  // legs_key
  u128 value;
};

// B has 16 alpha=0 identity entries (one per incoming signature) and one
// alpha=1 entry emitting 0->1 on all four channels; C sums alpha out.
static std::vector<CEntryH> build_c_sec_vi() {
  std::map<unsigned, u128> acc;
  for (unsigned sig = 0; sig < 16; ++sig) {
    uint8_t c = sig & 1, r = (sig >> 1) & 1, d = (sig >> 2) & 1, l = (sig >> 3) & 1;
    acc[legs_key(Legs{c, c, r, r, d, d, l, l})] += 1;
  }
  acc[legs_key(Legs{0, 1, 0, 1, 0, 1, 0, 1})] += 1;
  std::vector<CEntryH> out;
  for (auto& kv : acc) out.push_back(CEntryH{kv.first, kv.second});
  return out;
}

static unsigned input_signature(const Legs& l) { return l.ci | (l.ri << 1) | (l.dri << 2) | (l.dli << 3); }

// Fails closed exactly where CompiledRowOperator::compile does.
static void certify_c(const std::vector<CEntryH>& c) {
  bool pass[16] = {false};
  bool have_occ = false;
  for (const CEntryH& e : c) {
    Legs l = legs_from_key(e.legs);
    const bool is_pass = l.ci == l.co && l.ri == l.ro && l.dri == l.dro && l.dli == l.dlo;
    const bool is_occ = l.ci == 0 && l.co == 1 && l.ri == 0 && l.ro == 1 && l.dri == 0 && l.dro == 1 && l.dli == 0 &&
                        l.dlo == 1;
    if (e.value != 1) fail(QPEPS_ERR_INVALID, "compiled row operator requires unit Sec. VI coefficients");
    if (is_pass) {
      unsigned k = input_signature(l);
      if (pass[k]) {
        char buf[64];
        std::snprintf(buf, sizeof buf, "duplicate C pass-through signature %u%u%u%u", (k >> 3) & 1, (k >> 2) & 1,
                      (k >> 1) & 1, k & 1);
        fail(QPEPS_ERR_INVALID, buf);
      }
      pass[k] = true;
    } else if (is_occ) {
      if (have_occ) fail(QPEPS_ERR_INVALID, "multiple occupied C entries");
      have_occ = true;
    } else {
      fail(QPEPS_ERR_INVALID, "C contains an entry outside the Sec. VI row automaton");
    }
  }
  for (bool p : pass)
    if (!p) fail(QPEPS_ERR_INVALID, "C is missing a pass-through signature");
  if (!have_occ) fail(QPEPS_ERR_INVALID, "C is missing the occupied entry");
}

static CTableDev c_table_for_device(const std::vector<CEntryH>& c) {
  CTableDev t;
  std::memset(&t, 0, sizeof t);
  for (const CEntryH& e : c) {
    Legs l = legs_from_key(e.legs);
    unsigned sig = input_signature(l);
    unsigned slot = t.count[sig]++;
    if (slot >= 4) fail(QPEPS_ERR_INVALID, "more than four C entries share one input signature");
    t.out[sig][slot] = l.co | (l.ro << 1) | (l.dro << 2) | (l.dlo << 3);
    for (int r = 0; r < kMaxResidues; ++r) t.value_mod[sig][slot][r] = (uint32_t)(e.value % kPrimes[r]);
  }
  return t;
}

// ---------------------------------------------------------------------------
// Known counts (OEIS A000170), CRT plan and reconstruction.

static const char* kKnown[28] = {"1",
                                 "1",
                                 "0",
                                 "0",
                                 "2",
                                 "10",
                                 "4",
                                 "40",
                                 "92",
                                 "352",
                                 "724",
                                 "2680",
                                 "14200",
                                 "73712",
                                 "365596",
                                 "2279184",
                                 "14772512",
                                 "95815104",
                                 "666090624",
                                 "4968057848",
                                 "39029188884",
                                 "314666222712",
                                 "2691008701644",
                                 "24233937684440",
                                 "227514171973736",
                                 "2207893435808352",
                                 "22317699616364044",
                                 "234907967154122528"};

static bool known_count(unsigned n, u128* out) {
  if (n >= 28) return false;
  u128 v = 0;
  for (const char* p = kKnown[n]; *p; ++p) v = v * 10 + (u128)(*p - '0');
  *out = v;
  return true;
}

static u128 factorial(unsigned n) {
  u128 f = 1;
  for (unsigned i = 2; i <= n; ++i)
    if (!mul_u128(f, i, &f)) fail(QPEPS_ERR_RANGE, "N! exactness bound does not fit u128");
  return f;
}

// Shortest prefix of the residue primes whose product exceeds N! (the count
// and every row weight are at most N!).
static int crt_plan(unsigned n) {
  u128 bound = factorial(n), prod = 1;
  for (int r = 0; r < kMaxResidues; ++r) {
    prod *= kPrimes[r];
    if (prod > bound) return r + 1;
  }
  fail(QPEPS_ERR_RANGE, "available certified CRT product does not exceed N! bound");
}

// Modular inverse by the extended Euclidean algorithm.
static u64 inv_mod(u64 a, u64 p) {
  int64_t t = 0, nt = 1;
  int64_t r = (int64_t)p, nr = (int64_t)(a % p);
  while (nr != 0) {
    int64_t q = r / nr;
    int64_t tmp = t - q * nt;
    t = nt;
    nt = tmp;
    tmp = r - q * nr;
    r = nr;
    nr = tmp;
  }
  if (t < 0) t += (int64_t)p;
  return (u64)t;
}

// Garner's mixed-radix reconstruction with checked u128 arithmetic.
static u128 crt_reconstruct(const u64* residues, int count) {
  u128 value = 0, modulus = 1;
  for (int i = 0; i < count; ++i) {
    const u64 p = kPrimes[i];
    const u64 vm = (u64)(value % p);
    const u64 rm = residues[i] % p;
    const u64 delta = rm >= vm ? rm - vm : rm + p - vm;
    const u64 step = (u64)(((u128)delta * inv_mod((u64)(modulus % p), p)) % p);
    u128 term;
    if (!mul_u128(modulus, step, &term) || !add_u128(value, term, &value))
      fail(QPEPS_ERR_OVERFLOW, "CRT reconstruction overflow");
    if (!mul_u128(modulus, p, &modulus)) fail(QPEPS_ERR_OVERFLOW, "CRT reconstruction modulus overflow");
  }
  return value;
}

// ---------------------------------------------------------------------------
// Context: one device, one stream, a grow-only pool of device buffers.

struct DevBuf {
  void* ptr = nullptr;
  size_t bytes = 0;
};

struct GraphRecorder;
struct GraphPlan;

struct Ctx {
  int device = 0;
  int sms = 0;
  cudaStream_t stream = nullptr;
  DevBuf front[2];  // boundary buffers (keys then residue planes)
  DevBuf table;
  StepScalars* d_sc = nullptr;
  StepScalars* h_sc = nullptr;  // pinned
  cudaEvent_t ev[6] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
  size_t pool_bytes = 0, peak_pool_bytes = 0;
  size_t free_at_create = 0;
  uint64_t launches = 0;
  std::vector<CEntryH> c;
  CTableDev c_dev;
  bool c_uploaded = false;
  double partition_fill = 0.83;  // live target candidates per partition / slots (lowered after an overflow)
  double chain_fill = 1.0;       // the same of queued steps, where it is lower
  uint64_t h2d_bytes = 0, d2h_bytes = 0;  // host<->device copies issued (since context creation)
  struct Tune {
    uint32_t parents_per_lane = 4;              // partition scatter: 2 or 4
    uint32_t spread_cursors_below = 262144;     // pad cursors to 32 B when partitions <= this
    uint32_t wide_merge = 2;                    // 0 never, 1 always, 2 above wide_above_parts partitions:
                                                // 8192-slot merge CTAs (4096-candidate partitions);
                                                // 3: 2048-slot CTAs, four per SM (1024-candidate partitions)
    uint32_t wide_above_parts = 524288;         // 2048-candidate partitions beyond which auto goes wide
    uint32_t scatter_kind = 1;                  // PartitionCfg::scatter_kind
    uint32_t merge_kind = 1;                    // PartitionCfg::merge_kind
    uint32_t fold_weights = 2;                  // 0 residues, 1 CRT fold, 2 exact 64-bit weights in the
                                                // boundary (modes 1-2 only where exact: R = 2, N - k <= 20)
    double partition_fill = 0.83;               // starting value of Ctx::partition_fill
    double slice_margin = 5.0;                  // predictive slicing: slice peak / mean slice peak
    uint32_t unit_target = 1000;                // class-grouped partitions: planned candidates per partition
    uint32_t unit_sample = 8;                   // class-grouped partitions: 1 in unit_sample parents sampled
    uint32_t batch_lanes = 1;                   // CUDA-graph replay: device batches run on this many streams
    uint32_t merge_compact = 0;                 // claim-list merge: 1 = first claimants write from registers
    uint32_t scatter_block = 256;               // one-level scatters: threads per CTA (128, 256, 512)
    uint32_t merge_auto = QPEPS_MERGE_PARTITION;  // what QPEPS_MERGE_AUTO resolves to where both apply
    uint32_t slice_rows = 1;                    // rows enumerated on the host before slicing is considered
  } tune;
  DevBuf tail;                   // TailControl + overflow list
  DevBuf grp_side[2];            // column-grouped rows: the two boundaries' keys and weights
  DevBuf grp_dir;                // group and bucket directories, unit list, row scalars, binomials, seed
  void* grp_pin = nullptr;       // pinned: row scalars read back, seed uploads
  size_t grp_pin_bytes = 0;
  DevBuf plan;                   // class-grouped partitions: histogram, bucket table, scan partials
  DevBuf queue;                  // queued steps: their scalars
  StepScalars* h_queue = nullptr;  // pinned: the scalars as uploaded, then as read back
  size_t h_queue_steps = 0;
  uint8_t* h_seed = nullptr;     // pinned: a small chunk on its way to the device (kSeedStage bytes)
  uint64_t pool_gen = 0;         // bumped whenever a pool buffer is allocated or freed
  GraphRecorder* rec = nullptr;  // row steps of the running contraction (use_graph)
  GraphPlan* graph = nullptr;    // captured contraction (use_graph)
};

// Device memory a call may hold: the caller's figure, or 90 % of what is free
// or already in the context's pool. Free memory is asked for only when the
// pool alone does not answer the question (the query takes about 15 us, more
// than a small board's launches).
class Budget {
 public:
  Budget() = default;
  explicit Budget(size_t bytes) : bytes_(bytes) {}
  explicit Budget(const Ctx& ctx) : ctx_(&ctx) {}
  bool known() const { return !ctx_ || bytes_; }
  operator size_t() const {
    if (!known()) {
      size_t fr = 0, tot = 0;
      cuda_check(cudaMemGetInfo(&fr, &tot), "cudaMemGetInfo");
      bytes_ = (size_t)((double)(fr + ctx_->pool_bytes) * 0.90);
    }
    return bytes_;
  }
  bool holds(size_t need) const {
    if (!known() && (double)need <= 0.90 * (double)ctx_->pool_bytes) return true;
    return need <= (size_t)*this;
  }

 private:
  const Ctx* ctx_ = nullptr;
  mutable size_t bytes_ = 0;
};

static void buf_release(Ctx& ctx, DevBuf& b) {
  if (b.ptr) {
    cudaFree(b.ptr);
    ctx.pool_bytes -= b.bytes;
    ++ctx.pool_gen;
  }
  b.ptr = nullptr;
  b.bytes = 0;
}

// The column-grouped rows' buffers hold nothing between calls: another
// buffer that does not fit beside them takes their room.
static bool group_release(Ctx& ctx) {
  bool any = false;
  for (DevBuf* b : {&ctx.grp_side[0], &ctx.grp_side[1], &ctx.grp_dir}) {
    any = any || b->ptr;
    buf_release(ctx, *b);
  }
  return any;
}

static void buf_reserve(Ctx& ctx, DevBuf& b, size_t bytes, const Budget& budget, const char* what) {
  if (b.bytes >= bytes) return;
  size_t want = bytes + bytes / 4;
  if (ctx.pool_bytes - b.bytes + want > budget) want = bytes;
  if (ctx.pool_bytes - b.bytes + want > budget) group_release(ctx);
  if (ctx.pool_bytes - b.bytes + want > budget)
    fail(QPEPS_ERR_CAPACITY, std::string("device budget exceeded by ") + what);
  buf_release(ctx, b);
  cudaError_t e = cudaMalloc(&b.ptr, want);
  if (e != cudaSuccess && group_release(ctx)) {
    cudaGetLastError();
    e = cudaMalloc(&b.ptr, want);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    fail(QPEPS_ERR_CAPACITY, std::string("device allocation failed for ") + what);
  }
  b.bytes = want;
  ctx.pool_bytes += want;
  ctx.peak_pool_bytes = std::max(ctx.peak_pool_bytes, ctx.pool_bytes);
  ++ctx.pool_gen;
}

// buf_reserve's answer instead of its exception.
static bool try_reserve(Ctx& ctx, DevBuf& b, size_t bytes, const Budget& budget, const char* what) {
  try {
    buf_reserve(ctx, b, bytes, budget, what);
    return true;
  } catch (const Failure& e) {
    if (e.code != QPEPS_ERR_CAPACITY) throw;
    return false;
  }
}

// The scalars of queued steps. No captured graph holds their buffer (a replay has
// scalars of its own), so neither its growth nor its release ends one.
static bool queue_reserve(Ctx& ctx, size_t bytes, const Budget& budget) {
  const uint64_t gen = ctx.pool_gen;
  const bool ok = try_reserve(ctx, ctx.queue, bytes, budget, "queued step scalars");
  ctx.pool_gen = gen;
  return ok;
}

// What a row or site that runs by itself does not use: the buffers of other
// forms, of the slice tail and of the explicit-C frontier's steps (`plan` is
// also the class-grouped partitions' scratch).
static void idle_release(Ctx& ctx, bool plan) {
  group_release(ctx);
  const uint64_t gen = ctx.pool_gen;
  buf_release(ctx, ctx.queue);
  ctx.pool_gen = gen;
  buf_release(ctx, ctx.tail);
  if (plan) buf_release(ctx, ctx.plan);
}

static void graph_free(Ctx& ctx);

static void ctx_free(Ctx* ctx) {
  if (!ctx) return;
  cudaSetDevice(ctx->device);
  graph_free(*ctx);
  buf_release(*ctx, ctx->front[0]);
  buf_release(*ctx, ctx->front[1]);
  buf_release(*ctx, ctx->table);
  buf_release(*ctx, ctx->tail);
  buf_release(*ctx, ctx->plan);
  buf_release(*ctx, ctx->queue);
  group_release(*ctx);
  if (ctx->grp_pin) cudaFreeHost(ctx->grp_pin);
  if (ctx->h_queue) cudaFreeHost(ctx->h_queue);
  if (ctx->h_seed) cudaFreeHost(ctx->h_seed);
  if (ctx->d_sc) cudaFree(ctx->d_sc);
  if (ctx->h_sc) cudaFreeHost(ctx->h_sc);
  for (auto& e : ctx->ev)
    if (e) cudaEventDestroy(e);
  if (ctx->stream) cudaStreamDestroy(ctx->stream);
  delete ctx;
}

static Ctx* ctx_create(int device) {
  int count = 0;
  cuda_check(cudaGetDeviceCount(&count), "cudaGetDeviceCount");
  if (device < 0 || device >= count) fail(QPEPS_ERR_CUDA, "no such CUDA device");
  Ctx* ctx = new Ctx();
  try {
    ctx->device = device;
    cuda_check(cudaSetDevice(device), "cudaSetDevice");
    cuda_check(cudaDeviceGetAttribute(&ctx->sms, cudaDevAttrMultiProcessorCount, device), "SM count");
    cuda_check(cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking), "cudaStreamCreate");
    cuda_check(cudaMalloc(&ctx->d_sc, sizeof(StepScalars)), "step scalars");
    cuda_check(cudaMallocHost(&ctx->h_sc, sizeof(StepScalars)), "pinned step scalars");
    for (auto& e : ctx->ev) cuda_check(cudaEventCreate(&e), "cudaEventCreate");
    size_t fr = 0, tot = 0;
    cuda_check(cudaMemGetInfo(&fr, &tot), "cudaMemGetInfo");
    ctx->free_at_create = fr;
    ctx->c = build_c_sec_vi();
    certify_c(ctx->c);
    ctx->c_dev = c_table_for_device(ctx->c);
  } catch (...) {
    ctx_free(ctx);
    throw;
  }
  return ctx;
}

// ---------------------------------------------------------------------------
// Contraction driver.

struct Item {
  u128 key;     // packed boundary (reference layout)
  u128 weight;  // exact multiplicity (orbit weight)
};

struct RowAcc {
  bool used = false;
  u64 input_states = 0, output_states = 0;
  u128 candidates = 0, matched = 0, completed = 0, examined = 0, tmatched = 0;
  u128 weight_exact = 0;      // rows computed on the host
  u64 weight_res[kMaxResidues] = {0, 0, 0, 0};  // sums mod p of device rows
  bool device_row = false;
  double elapsed = 0;
};

struct RunStats {
  u64 entries_in = 0, entries_out = 0, candidates = 0, launches = 0;
  u64 peak_states = 0;
  u64 tail_items = 0, tail_overflow = 0;
  double device_ms = 0, merge_ms = 0, scatter_ms = 0, tail_ms = 0;
  u64 merge_launches = 0, merge_bytes = 0;
  u64 final_res[kMaxResidues] = {0, 0, 0, 0};
  unsigned batches = 0;
  uint32_t forms = 0;  // QPEPS_ROWS_* of the rows that ran
};

struct Plan {
  unsigned n;
  unsigned free_rows;  // rows after the placed prefix: the count and every row weight are at most free_rows!
  int R;
  int key_bits;
  int grain;
  int merge;  // QPEPS_MERGE_HASH or QPEPS_MERGE_PARTITION
  Budget budget;
  int threads;
  unsigned tail_row;  // rows >= tail_row go to the slice-tail kernel (n = none)
  bool prefix = false;      // a partly placed board
  double batch_states = 0;  // expected largest boundary of one device batch (0: unknown)
  double group_states = 0;  // column-grouped rows: expected largest boundary of a device batch (0: not used)
  bool w64 = false;   // residue planes 0/1 hold the low/high words of exact weights (partitioned row merge)
  int Rc = 0;         // residues of the CRT bookkeeping (= R except with w64, where R = 2 planes)
};

static size_t entry_bytes(const Plan& p) { return (size_t)(p.key_bits / 8) + 4u * p.R; }
// Bytes of one partitioned-merge candidate (key and residue words, padded).
static size_t cand_bytes(const Plan& p) { return p.key_bits == 128 ? 32 : candidate_bytes(p.R); }

static FrontierView view_of(const Plan& p, DevBuf& b, u64 cap) {
  FrontierView v;
  v.keys = b.ptr;
  v.res = reinterpret_cast<uint32_t*>(reinterpret_cast<char*>(b.ptr) + (size_t)cap * (p.key_bits / 8));
  v.cap = cap;
  return v;
}

static u64 pow2_at_least(u64 x) {
  u64 p = 1;
  while (p < x) p <<= 1;
  return p;
}

static void sync_scalars(Ctx& ctx) {
  cuda_check(cudaMemcpyAsync(ctx.h_sc, ctx.d_sc, sizeof(StepScalars), cudaMemcpyDeviceToHost, ctx.stream),
             "read step scalars");
  ctx.d2h_bytes += sizeof(StepScalars);
  cuda_check(cudaStreamSynchronize(ctx.stream), "step synchronize");
}

// The live device boundary: ctx.front[0] holds `count` entries, keys first,
// then R residue planes of stride `cap`. Merge steps run in place: the expand
// kernel consumes every input entry before the merge kernel writes outputs
// into the same buffer.
struct DevFrontier {
  u64 count = 0;
  u64 cap = 0;
  u128 weight_bound = 0;  // upper bound of the live boundary's total weight (w64 certification)
};

// Boundary entries parked on the host (the seed, or a half split off under
// memory pressure), resuming at (row, site).
struct HostChunk {
  unsigned row = 0, site = 0;
  bool row_counted = false;  // site grain: this row's metrics already include these entries
  bool no_tail = false;      // entries that overflowed the slice tail: contract every row here
  u64 count = 0;
  u128 weight_bound = 0;      // upper bound of the chunk's total weight (w64 certification)
  std::vector<uint8_t> keys;
  std::vector<uint32_t> res;  // R planes of `count`
};

constexpr u64 kTermsUnknown = ~0ull;

struct StepOut {
  u64 in = 0, terms = 0, out = 0;
  u64 next_terms = kTermsUnknown;  // the output boundary's successor terms at the next row, if the merge counted them
  u64 exact_sum = 0;  // w64: exact total weight of the output boundary
  u64 weight[kMaxResidues] = {0, 0, 0, 0};
  u64 final_sum[kMaxResidues] = {0, 0, 0, 0};
};

enum class StepStatus { Ok, NeedSplit };

// Row steps of one contraction as launched, for CUDA-graph replay
// (qpeps_options.use_graph): every device batch's seed and, per row step, the
// partition configuration and the sizes the step saw.
struct GraphStepRec {
  PartitionCfg pc{};
  bool unit = false;  // class-grouped partitions: the plan is rebuilt on the device before the scatter
  UnitClassPlan ucp{};
  UnitPlanArgs upa{};
  u64 n_in = 0, terms = 0, out = 0, need_cap = 0;
  size_t region_bytes = 0, table_bytes = 0;
  bool final_step = false;
  u64 weight_sum[kMaxResidues] = {0, 0, 0, 0};  // raw device sums (not reduced)
  u64 final_sum[kMaxResidues] = {0, 0, 0, 0};
};

struct GraphChunkRec {
  u64 count = 0;
  std::vector<uint8_t> keys;
  std::vector<uint32_t> res;
  std::vector<GraphStepRec> steps;
};

struct GraphRecorder {
  bool ok = true;         // false once anything outside the capturable form ran
  bool compared = false;  // column-grouped or one-CTA rows ran: compared with the next run instead
  std::vector<GraphChunkRec> chunks;
};

static size_t key_bytes(const Plan& p) { return (size_t)p.key_bits / 8; }

// Grow front[0] to hold `need` entries, keeping the live ones. Returns false
// when the budget cannot hold the grown buffer next to `other_bytes`.
static bool ensure_front(Ctx& ctx, const Plan& p, DevFrontier& f, u64 need, size_t other_bytes, bool grows = true) {
  if (f.cap >= need) return true;
  const size_t eb = entry_bytes(p);
  // Grow in large steps (x3, capped where the step's scratch would no longer
  // fit next to the boundary) so that a growing frontier is copied rarely.
  const u64 step_cap = (u64)((double)p.budget / ((double)eb + 1.25 * (double)cand_bytes(p)));
  u64 want = grows ? std::max<u64>(need, std::min<u64>(need * 3, step_cap)) : need;
  const size_t live = ctx.front[0].bytes;
  if (live + want * eb + other_bytes > p.budget) want = need;
  if (live + want * eb + other_bytes > p.budget) return false;
  if (ctx.pool_bytes + want * eb + other_bytes > p.budget) group_release(ctx);
  DevBuf nb;
  cudaError_t e = cudaMalloc(&nb.ptr, want * eb);
  if (e != cudaSuccess && group_release(ctx)) {
    cudaGetLastError();
    e = cudaMalloc(&nb.ptr, want * eb);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  nb.bytes = want * eb;
  ctx.pool_bytes += nb.bytes;
  ++ctx.pool_gen;
  ctx.peak_pool_bytes = std::max(ctx.peak_pool_bytes, ctx.pool_bytes);
  if (f.count) {
    const size_t kb = key_bytes(p);
    char* src = static_cast<char*>(ctx.front[0].ptr);
    char* dst = static_cast<char*>(nb.ptr);
    cuda_check(cudaMemcpyAsync(dst, src, f.count * kb, cudaMemcpyDeviceToDevice, ctx.stream), "grow keys");
    for (int r = 0; r < p.R; ++r)
      cuda_check(cudaMemcpyAsync(dst + want * kb + (size_t)r * want * 4, src + f.cap * kb + (size_t)r * f.cap * 4,
                                 f.count * 4, cudaMemcpyDeviceToDevice, ctx.stream),
                 "grow residues");
    cuda_check(cudaStreamSynchronize(ctx.stream), "grow synchronize");
  }
  buf_release(ctx, ctx.front[0]);
  ctx.front[0] = nb;
  f.cap = want;
  return true;
}

// Give back what front[0] holds beyond `need` entries (a buffer of an earlier
// call, larger than a small budget can keep beside a step's scratch). The live
// entries move through the host, on the context's stream like everything that
// reads them: the two buffers together would pass the budget. False, with
// nothing changed, when the budget does not hold the smaller buffer beside the
// pool's others.
static bool shrink_front(Ctx& ctx, const Plan& p, DevFrontier& f, u64 need) {
  const size_t kb = key_bytes(p), eb = entry_bytes(p);
  const auto fits = [&] { return ctx.pool_bytes - ctx.front[0].bytes + need * eb <= p.budget; };
  if (!fits() && !(group_release(ctx) && fits())) return false;
  std::vector<char> live(f.count * eb);
  const auto move = [&](bool save) {
    char* const dev = static_cast<char*>(ctx.front[0].ptr);
    size_t at = 0;
    const auto part = [&](size_t off, size_t bytes) {
      char* const host = live.data() + at;
      cuda_check(save ? cudaMemcpyAsync(host, dev + off, bytes, cudaMemcpyDeviceToHost, ctx.stream)
                      : cudaMemcpyAsync(dev + off, host, bytes, cudaMemcpyHostToDevice, ctx.stream),
                 save ? "save boundary" : "restore boundary");
      at += bytes;
    };
    part(0, f.count * kb);
    for (int r = 0; r < p.R; ++r) part(f.cap * kb + (size_t)r * f.cap * 4, f.count * 4);
    cuda_check(cudaStreamSynchronize(ctx.stream), "shrink synchronize");
    (save ? ctx.d2h_bytes : ctx.h2d_bytes) += at;
  };
  move(true);
  buf_release(ctx, ctx.front[0]);
  buf_reserve(ctx, ctx.front[0], need * eb, p.budget, "boundary");
  f.cap = ctx.front[0].bytes / eb;
  move(false);
  return true;
}

static u64 count_terms(Ctx& ctx, const Plan& p, const DevFrontier& f, bool site, unsigned site_idx, RunStats& rs) {
  if (f.count == 0) return 0;
  LaunchCfg cfg{p.key_bits, p.R, p.threads, ctx.sms};
  FrontierView in = view_of(p, ctx.front[0], f.cap);
  cuda_check(cudaMemsetAsync(ctx.d_sc, 0, sizeof(StepScalars), ctx.stream), "clear step scalars");
  if (site)
    cuda_check(launch_site_count(cfg, in, f.count, p.n, site_idx, ctx.d_sc, ctx.stream), "site count kernel");
  else
    cuda_check(launch_row_count(cfg, in, f.count, p.n, ctx.d_sc, ctx.stream), "row count kernel");
  rs.launches += 1;
  sync_scalars(ctx);
  return ctx.h_sc->terms;
}

static double binom(unsigned n, unsigned k) {
  if (k > n) return 0;
  double v = 1;
  for (unsigned i = 1; i <= k; ++i) v = v * (double)(n - k + i) / (double)i;
  return v;
}

// Class plan of a row step with `terms` successors whose columns hold
// `filled` queens: the window width t puts about target / 2 candidates in a
// class, and the bucket count is about twice the class count.
static UnitClassPlan unit_class_plan(unsigned n, unsigned filled, u64 terms, u32 target) {
  UnitClassPlan c{};
  c.n = n;
  const double per_class = std::max(64.0, target / 2.0);
  const double groups = std::max(1.0, binom(n, std::min(filled, n)));
  const double want = (double)terms / (groups * per_class);
  unsigned t = want > 1.0 ? (unsigned)std::lround(std::log(want) / std::log(4.0)) : 0u;
  t = std::min(t, std::min(7u, n / 2));
  c.t = t;
  const double classes = std::max(1.0, (double)terms / per_class);
  unsigned lg = (unsigned)std::ceil(std::log2(classes)) + 1;
  lg = std::max(10u, std::min(24u, lg));
  c.lg = lg;
  return c;
}

// One merge step (a row in row grain, a site in site grain), in place.
// `known_terms`: the step's successor count when the previous row's merge
// counted it for exactly this boundary (no counting pass then).
static StepStatus merge_step(Ctx& ctx, const Plan& p, DevFrontier& f, bool site, unsigned site_idx, bool final_step,
                             RunStats& rs, unsigned row, StepOut* so_out, u64 known_terms = kTermsUnknown) {
  StepOut so;
  const u64 n_in = f.count;
  so.in = n_in;
  so.terms = (known_terms != kTermsUnknown && !site) ? known_terms : count_terms(ctx, p, f, site, site_idx, rs);
  if (so.terms == 0) {
    f.count = 0;
    *so_out = so;
    if (ctx.rec && !ctx.rec->chunks.empty()) ctx.rec->chunks.back().steps.push_back(GraphStepRec{});
    return StepStatus::Ok;
  }
  const bool partition = p.merge == QPEPS_MERGE_PARTITION && !site;
  if (ctx.rec && !partition) ctx.rec->ok = false;
  const size_t eb = entry_bytes(p);
  // Wide merge CTAs halve the number of open partition tails the scatter
  // keeps in L2; they pay off once the narrow partitions no longer fit there.
  const double narrow_parts = (double)so.terms / (ctx.partition_fill * partition_capacity(0));
  const bool want_wide = ctx.tune.wide_merge == 1 ||
                         (ctx.tune.wide_merge == 2 && narrow_parts > (double)ctx.tune.wide_above_parts);
  // Class-grouped partitions (16-byte candidates, narrow merge CTAs).
  // 128-bit keys: their own scatter and merge (one shape, 1024-candidate partitions).
  const bool wkeys = p.key_bits == 128;
  // (Its classes read the reference key layout: boards up to N = 21.)
  const bool unit = partition && !wkeys && ctx.tune.scatter_kind == 3 && unit_scatter_supported(p.R) &&
                    p.n <= kRefU64MaxN;
  const bool small = ctx.tune.wide_merge == 3;
  const u32 wide = (!unit && !wkeys && wide_merge_supported(p.R)) ? (small ? 2u : want_wide ? 1u : 0u) : 0u;
  const u32 pcap = wkeys ? wide_key_partition_capacity() : partition_capacity(wide);
  double mean = ctx.partition_fill * pcap;
  double unit_target = ctx.tune.unit_target;
  for (int attempt = 0;; ++attempt) {
    u32 parts = 0, cstride = 1;
    u64 slots = 0;
    size_t table_bytes, region_bytes = 0;
    PartitionCfg tl{};  // two-level scatter plan (tl.tl_nb = 0: one-level)
    UnitClassPlan ucp{};
    UnitPlanArgs upa{};
    UnitPlanDev upd{};
    if (unit) {
      // Plan on the device from a sampled histogram of this step's successors;
      // the host reads back the unit count to size the regions.
      ucp = unit_class_plan(p.n, row + 1, so.terms, (u32)unit_target);
      upa.lg = ucp.lg;
      upa.sample = ctx.tune.unit_sample;
      upa.target = (u64)unit_target;
      const size_t plan_bytes = unit_plan_scratch_bytes(upa.lg);
      if (ctx.plan.bytes < plan_bytes) {
        buf_release(ctx, ctx.plan);
        if (ctx.pool_bytes + plan_bytes > p.budget) buf_release(ctx, ctx.table);
        buf_reserve(ctx, ctx.plan, plan_bytes, p.budget, "partition plan");
      }
      cuda_check(cudaEventRecord(ctx.ev[3], ctx.stream), "event");
      cuda_check(launch_unit_plan(view_of(p, ctx.front[0], f.cap), n_in, ucp, upa, ctx.plan.ptr, ctx.sms, ctx.stream,
                                  &upd),
                 "partition plan kernels");
      cuda_check(cudaEventRecord(ctx.ev[4], ctx.stream), "event");
      UnitPlanTotals tot{};
      cuda_check(cudaMemcpyAsync(&tot, upd.totals, sizeof tot, cudaMemcpyDeviceToHost, ctx.stream), "plan totals");
      cuda_check(cudaStreamSynchronize(ctx.stream), "plan synchronize");
      ctx.d2h_bytes += sizeof tot;
      rs.launches += 4;
      if (tot.units == 0 || tot.units > 0xffffffffull)
        fail(QPEPS_ERR_CAPACITY, row_msg("partition plan out of range at row", row + 1));
      parts = (u32)tot.units;
      region_bytes = (size_t)parts * pcap * cand_bytes(p);
      cstride = (parts <= ctx.tune.spread_cursors_below) ? 8u : 1u;
      table_bytes = region_bytes + ((size_t)parts * 4 * cstride + 255) / 256 * 256;
    } else if (partition) {
      const u64 parts64 = std::max<u64>(1, (u64)((double)so.terms / mean) + 1);
      if (parts64 > 0xffffffffull) fail(QPEPS_ERR_CAPACITY, row_msg("too many partitions at row", row + 1));
      parts = (u32)parts64;
      if (!wkeys && ctx.tune.scatter_kind == 2 && two_level_plan(so.terms, parts, p.R, &tl)) parts = tl.parts;
      region_bytes = (size_t)parts * pcap * cand_bytes(p);
      cstride = (parts <= ctx.tune.spread_cursors_below) ? 8u : 1u;
      table_bytes = region_bytes + ((size_t)parts * 4 * cstride + 255) / 256 * 256;
      if (tl.tl_nb) {
        tl.cursor_stride = cstride;
        table_bytes += two_level_extra_bytes(tl);
      }
    } else {
      slots = pow2_at_least(std::max<u64>(1024, so.terms * 2));
      table_bytes = slots * slot_bytes(p.key_bits, p.R);
    }
    const u64 need_cap = final_step ? n_in : std::max<u64>(n_in, so.terms);
    // The pool's other buffers count: where they are in the way, those that this
    // step does not use go.
    const auto others = [&] { return ctx.pool_bytes - ctx.front[0].bytes - ctx.table.bytes; };
    const auto fits = [&](u64 cap) { return cap * eb + table_bytes + others() <= p.budget; };
    if (!fits(std::max<u64>(f.cap, need_cap))) idle_release(ctx, !unit);
    if (f.cap > need_cap && !fits(f.cap) && fits(need_cap * 5 / 4) && f.count <= need_cap) {
      buf_release(ctx, ctx.table);
      shrink_front(ctx, p, f, need_cap);
    }
    if (!fits(std::max<u64>(f.cap, need_cap))) {
      if (n_in <= 1) fail(QPEPS_ERR_CAPACITY, row_msg("device budget exceeded at row", row + 1));
      return StepStatus::NeedSplit;
    }
    if (ctx.table.bytes < table_bytes) buf_release(ctx, ctx.table);
    if (f.cap < need_cap) {
      if (ctx.pool_bytes + (need_cap - f.cap) * eb + table_bytes > p.budget) buf_release(ctx, ctx.table);
      if (!ensure_front(ctx, p, f, need_cap, ctx.table.ptr ? 0 : table_bytes)) {
        if (n_in <= 1) fail(QPEPS_ERR_CAPACITY, row_msg("device budget exceeded at row", row + 1));
        return StepStatus::NeedSplit;
      }
    }
    if (ctx.pool_bytes - ctx.table.bytes + table_bytes > p.budget) buf_release(ctx, ctx.table);
    // (A boundary that grew beyond its need, for rows to come, gives way.)
    const char* what = partition ? "partition regions" : "hash table";
    const auto scratch = [&] { return try_reserve(ctx, ctx.table, table_bytes, p.budget, what); };
    if (!scratch() && !(f.cap > need_cap && shrink_front(ctx, p, f, need_cap) && scratch())) {
      if (n_in <= 1) fail(QPEPS_ERR_CAPACITY, row_msg("device budget exceeded at row", row + 1));
      return StepStatus::NeedSplit;
    }

    LaunchCfg cfg{p.key_bits, p.R, p.threads, ctx.sms};
    FrontierView view = view_of(p, ctx.front[0], f.cap);
    const u64 terms = so.terms;
    cuda_check(cudaMemsetAsync(ctx.d_sc, 0, sizeof(StepScalars), ctx.stream), "clear step scalars");
    PartitionCfg pc{p.R, ctx.sms, parts, pcap, p.R == 1 ? 3 : p.R == 2 ? 2 : 1, cstride, ctx.tune.parents_per_lane,
                    wide, ctx.tune.scatter_kind, ctx.tune.merge_kind,
                    p.w64 ? 2u : (ctx.tune.fold_weights && p.R == 2 && p.free_rows <= 20) ? 1u : 0u};
    pc.merge_regs = ctx.tune.merge_compact;
    pc.scatter_block = ctx.tune.scatter_block;
    pc.key_bits = (uint32_t)p.key_bits;
    pc.tl_nb = tl.tl_nb;
    pc.tl_p2 = tl.tl_p2;
    pc.tl_bcap = tl.tl_bcap;
    void* regions = ctx.table.ptr;
    uint32_t* cursors = reinterpret_cast<uint32_t*>(static_cast<char*>(ctx.table.ptr) + region_bytes);
    if (partition)
      cuda_check(cudaMemsetAsync(cursors, 0, (size_t)parts * 4 * cstride, ctx.stream), "clear partition cursors");
    else
      cuda_check(cudaMemsetAsync(ctx.table.ptr, 0, table_bytes, ctx.stream), "clear hash table");
    cuda_check(cudaEventRecord(ctx.ev[0], ctx.stream), "event");
    if (unit)
      cuda_check(launch_unit_scatter(pc, view, n_in, ucp, upd.table, regions, cursors, ctx.d_sc, ctx.stream),
                 "class scatter kernel");
    else if (partition)
      cuda_check(launch_partition_scatter(pc, view, n_in, p.n, regions, cursors, ctx.d_sc, ctx.stream),
                 "partition scatter kernel");
    else if (site)
      cuda_check(launch_site_expand_insert(cfg, view, n_in, p.n, site_idx, ctx.table.ptr, slots, ctx.d_sc, ctx.stream),
                 "site expand-insert kernel");
    else
      cuda_check(launch_row_expand_insert(cfg, view, n_in, p.n, ctx.table.ptr, slots, ctx.d_sc, ctx.stream),
                 "row expand-insert kernel");
    cuda_check(cudaEventRecord(ctx.ev[1], ctx.stream), "event");
    if (partition)
      cuda_check(launch_partition_merge(pc, regions, cursors, view, p.n, !final_step, ctx.d_sc, ctx.stream),
                 "partition merge kernel");
    else
      cuda_check(launch_compact(cfg, ctx.table.ptr, slots, view, p.n, !final_step, ctx.d_sc, ctx.stream),
                 "compact kernel");
    cuda_check(cudaEventRecord(ctx.ev[2], ctx.stream), "event");
    rs.launches += 2;
    sync_scalars(ctx);
    if (ctx.h_sc->error & kErrBounds)
      fail(QPEPS_ERR_CUDA, row_msg("a kernel's bounds check failed (access skipped) at row", row + 1));
    if (partition && (ctx.h_sc->error & kErrOverflow)) {
      // The merge kernel saw the flag and wrote nothing: the input is intact.
      if (attempt >= 4) fail(QPEPS_ERR_CAPACITY, row_msg("partition overflow persists at row", row + 1));
      mean *= 0.6;
      unit_target = std::max(256.0, unit_target * 0.7);
      ctx.partition_fill = std::max(0.3, ctx.partition_fill * 0.8);  // keep a wider margin for this context
      (void)terms;
      continue;
    }
    if (ctx.h_sc->error & kErrProbeLimit) fail(QPEPS_ERR_CAPACITY, row_msg("hash probe bound exceeded at row", row + 1));
    if (ctx.h_sc->error) fail(QPEPS_ERR_CAPACITY, row_msg("device capacity error at row", row + 1));
    float ms_a = 0, ms_b = 0, ms_plan = 0;
    cudaEventElapsedTime(&ms_a, ctx.ev[0], ctx.ev[1]);
    cudaEventElapsedTime(&ms_b, ctx.ev[1], ctx.ev[2]);
    if (unit) {
      // The plan kernels belong to the scatter's side of the step (as in a
      // CUDA-graph replay, where they run back to back with it).
      cudaEventElapsedTime(&ms_plan, ctx.ev[3], ctx.ev[4]);
      ms_a += ms_plan;
    }
    so.out = ctx.h_sc->out_count;
    if (!final_step && ctx.h_sc->next_terms_ok) so.next_terms = ctx.h_sc->next_terms;
    so.exact_sum = ctx.h_sc->weight_sum[0];
    for (int r = 0; r < p.Rc; ++r) {
      // Exact weights: plane 0 carries the exact sums.
      so.weight[r] = ctx.h_sc->weight_sum[p.w64 ? 0 : r] % kPrimes[r];
      so.final_sum[r] = ctx.h_sc->final_sum[p.w64 ? 0 : r] % kPrimes[r];
    }
    if (ctx.rec) {
      if (ctx.rec->chunks.empty() || !partition) {
        ctx.rec->ok = false;
      } else {
        GraphStepRec g;
        g.pc = pc;
        g.unit = unit;
        g.ucp = ucp;
        g.upa = upa;
        g.n_in = n_in;
        g.terms = terms;
        g.out = so.out;
        g.need_cap = need_cap;
        g.region_bytes = region_bytes;
        g.table_bytes = table_bytes;
        g.final_step = final_step;
        for (int r = 0; r < p.R; ++r) {
          g.weight_sum[r] = ctx.h_sc->weight_sum[r];
          g.final_sum[r] = ctx.h_sc->final_sum[r];
        }
        ctx.rec->chunks.back().steps.push_back(g);
      }
    }
    rs.device_ms += ms_a + ms_b;
    rs.scatter_ms += ms_a;
    rs.merge_ms += ms_b;
    rs.merge_launches += 1;
    rs.forms |= QPEPS_ROWS_SINGLE;
    rs.merge_bytes += (n_in + so.out) * eb;
    rs.entries_in += n_in;
    rs.entries_out += so.out;
    rs.candidates += so.terms;
    f.count = final_step ? 0 : so.out;
    *so_out = so;
    return StepStatus::Ok;
  }
}

// Move the upper half of the live boundary to the host; the caller resumes it
// later at the same (row, site).
static void split_to_host(Ctx& ctx, const Plan& p, DevFrontier& f, unsigned row, unsigned site, bool row_counted,
                          bool no_tail, std::vector<HostChunk>& pending) {
  if (ctx.rec) ctx.rec->ok = false;
  const u64 keep = f.count / 2, moved = f.count - keep;
  HostChunk hc;
  hc.row = row;
  hc.site = site;
  hc.row_counted = row_counted;
  hc.no_tail = no_tail;
  hc.count = moved;
  hc.weight_bound = f.weight_bound;
  const size_t kb = key_bytes(p);
  hc.keys.resize(moved * kb);
  hc.res.resize((size_t)p.R * moved);
  const char* src = static_cast<const char*>(ctx.front[0].ptr);
  cuda_check(cudaMemcpyAsync(hc.keys.data(), src + keep * kb, moved * kb, cudaMemcpyDeviceToHost, ctx.stream),
             "spill keys");
  for (int r = 0; r < p.R; ++r)
    cuda_check(cudaMemcpyAsync(hc.res.data() + (size_t)r * moved, src + f.cap * kb + ((size_t)r * f.cap + keep) * 4,
                               moved * 4, cudaMemcpyDeviceToHost, ctx.stream),
               "spill residues");
  cuda_check(cudaStreamSynchronize(ctx.stream), "spill synchronize");
  ctx.d2h_bytes += moved * (kb + 4u * p.R);
  f.count = keep;
  pending.push_back(std::move(hc));
}

constexpr size_t kSeedStage = 64 << 10;

// Pooled buffers are dead between chunks; those of earlier calls go where they
// exceed this call's budget.
static void trim_pool(Ctx& ctx, const Plan& p) {
  if (!p.budget.known()) return;
  if (ctx.pool_bytes > p.budget) group_release(ctx);
  if (ctx.pool_bytes > p.budget) buf_release(ctx, ctx.table);
  if (ctx.front[0].bytes > p.budget) buf_release(ctx, ctx.front[0]);
}

static void upload_chunk(Ctx& ctx, const Plan& p, const HostChunk& hc, DevFrontier& f) {
  f.count = 0;
  trim_pool(ctx, p);
  if (!ctx.front[0].ptr || f.cap < hc.count) {
    buf_release(ctx, ctx.front[0]);
    f.cap = 0;
  }
  if (!ensure_front(ctx, p, f, std::max<u64>(hc.count, 1), 0))
    fail(QPEPS_ERR_CAPACITY, "device budget cannot hold the seed boundary");
  const size_t kb = key_bytes(p);
  char* dst = static_cast<char*>(ctx.front[0].ptr);
  // A small chunk goes through pinned memory, which the copies read while the
  // host goes on (the chunk's last row is waited for before the next upload).
  const size_t bytes = hc.count * (kb + 4u * p.R);
  const uint8_t* keys = hc.keys.data();
  const uint8_t* res = reinterpret_cast<const uint8_t*>(hc.res.data());
  const bool staged = bytes <= kSeedStage;
  if (staged) {
    if (!ctx.h_seed) cuda_check(cudaMallocHost(&ctx.h_seed, kSeedStage), "pinned seed staging");
    std::memcpy(ctx.h_seed, keys, hc.count * kb);
    std::memcpy(ctx.h_seed + hc.count * kb, res, hc.count * 4u * p.R);
    keys = ctx.h_seed;
    res = ctx.h_seed + hc.count * kb;
  }
  cuda_check(cudaMemcpyAsync(dst, keys, hc.count * kb, cudaMemcpyHostToDevice, ctx.stream), "upload keys");
  for (int r = 0; r < p.R; ++r)
    cuda_check(cudaMemcpyAsync(dst + f.cap * kb + (size_t)r * f.cap * 4, res + (size_t)r * hc.count * 4, hc.count * 4,
                               cudaMemcpyHostToDevice, ctx.stream),
               "upload residues");
  if (!staged) cuda_check(cudaStreamSynchronize(ctx.stream), "upload synchronize");
  ctx.h2d_bytes += hc.count * (kb + 4u * p.R);
  f.count = hc.count;
  f.weight_bound = hc.weight_bound;
  if (ctx.rec) {
    GraphChunkRec c;
    c.count = hc.count;
    c.keys = hc.keys;
    c.res = hc.res;
    ctx.rec->chunks.push_back(std::move(c));
  }
}

static HostChunk chunk_from_items(const Plan& p, const std::vector<Item>& items, unsigned row) {
  HostChunk hc;
  hc.row = row;
  hc.count = items.size();
  for (const Item& it : items) hc.weight_bound += it.weight;
  const size_t kb = key_bytes(p);
  hc.keys.resize(hc.count * kb);
  hc.res.resize((size_t)p.R * hc.count);
  for (u64 i = 0; i < hc.count; ++i) {
    if (kb == 8) {
      // Host items hold the reference layout in a u128; a u64 device key at
      // N = 22 takes the compact layout.
      const u64 mask = (1ull << p.n) - 1;
      const State st = unpack<u128>(items[i].key, p.n, mask);
      const u64 k = pack<u64>(st.cols, st.dr, st.dl, p.n);
      std::memcpy(&hc.keys[i * 8], &k, 8);
    } else {
      std::memcpy(&hc.keys[i * 16], &items[i].key, 16);
    }
    if (p.w64) {
      hc.res[i] = (uint32_t)items[i].weight;
      hc.res[hc.count + i] = (uint32_t)(items[i].weight >> 32);
    } else {
      for (int r = 0; r < p.R; ++r) hc.res[(size_t)r * hc.count + i] = (uint32_t)(items[i].weight % kPrimes[r]);
    }
  }
  return hc;
}

// Rows [row0, n) of every live boundary entry through the slice-tail kernel;
// entries that overflow its shared-memory capacity come back as a host chunk
// that the row engine contracts to the end.
static void run_tail(Ctx& ctx, const Plan& p, DevFrontier& f, unsigned row0, std::vector<RowAcc>& rows, RunStats& rs,
                     std::vector<HostChunk>& pending) {
  if (ctx.rec) ctx.rec->ok = false;
  const u64 items = f.count;
  const size_t ctl_bytes = (sizeof(TailControl) + 255) / 256 * 256;
  const size_t need = ctl_bytes + items * 8;
  if (ctx.tail.bytes < need) {
    buf_release(ctx, ctx.tail);
    if (ctx.pool_bytes + need > p.budget) buf_release(ctx, ctx.table);
    buf_reserve(ctx, ctx.tail, need, p.budget, "slice-tail control");
  }
  TailControl* d_ctl = static_cast<TailControl*>(ctx.tail.ptr);
  uint64_t* d_over = reinterpret_cast<uint64_t*>(static_cast<char*>(ctx.tail.ptr) + ctl_bytes);
  TailControl h{};
  h.overflow_cap = items;
  h.overflow_items = d_over;
  cuda_check(cudaMemcpyAsync(d_ctl, &h, sizeof h, cudaMemcpyHostToDevice, ctx.stream), "tail control");
  FrontierView view = view_of(p, ctx.front[0], f.cap);
  const auto t0 = std::chrono::steady_clock::now();
  cuda_check(cudaEventRecord(ctx.ev[0], ctx.stream), "event");
  cuda_check(launch_slice_tail(p.R, view, items, p.n, row0, d_ctl, ctx.sms, ctx.stream), "slice tail kernel");
  cuda_check(cudaEventRecord(ctx.ev[1], ctx.stream), "event");
  rs.launches += 1;
  cuda_check(cudaMemcpyAsync(&h, d_ctl, sizeof h, cudaMemcpyDeviceToHost, ctx.stream), "tail results");
  cuda_check(cudaStreamSynchronize(ctx.stream), "tail synchronize");
  if (h.error) fail(QPEPS_ERR_CAPACITY, "slice-tail overflow list exceeded");
  float ms = 0;
  cudaEventElapsedTime(&ms, ctx.ev[0], ctx.ev[1]);
  rs.tail_ms += ms;
  rs.device_ms += ms;
  rs.tail_items += items;
  rs.tail_overflow += h.overflow_count;
  for (int r = 0; r < p.R; ++r) rs.final_res[r] = (rs.final_res[r] + h.final_sum[r] % kPrimes[r]) % kPrimes[r];
  const double el = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
  for (unsigned row = row0; row < p.n; ++row) {
    const unsigned q = row - row0;
    RowAcc& acc = rows[row];
    acc.used = true;
    acc.device_row = true;
    acc.input_states += h.row_acc[q][0];
    acc.output_states += h.row_acc[q][1];
    acc.matched += h.row_acc[q][2];
    acc.completed += h.row_acc[q][2];
    acc.candidates += (u128)h.row_acc[q][0] * p.n;
    for (int r = 0; r < p.R; ++r) acc.weight_res[r] = (acc.weight_res[r] + h.row_acc[q][3 + r] % kPrimes[r]) % kPrimes[r];
    acc.elapsed += el / (p.n - row0);
    rs.entries_in += h.row_acc[q][0];
    rs.entries_out += h.row_acc[q][1];
    rs.candidates += h.row_acc[q][2];
  }
  if (h.overflow_count) {
    // Gather the overflowing entries (compact, plane stride = count) into the
    // table buffer, then park them on the host as a merged chunk.
    const u64 m = h.overflow_count;
    const size_t kb = key_bytes(p);
    const size_t bytes = m * (kb + 4u * p.R);
    if (ctx.table.bytes < bytes) {
      buf_release(ctx, ctx.table);
      buf_reserve(ctx, ctx.table, bytes, p.budget, "tail overflow gather");
    }
    uint64_t* gk = static_cast<uint64_t*>(ctx.table.ptr);
    uint32_t* gr = reinterpret_cast<uint32_t*>(static_cast<char*>(ctx.table.ptr) + m * kb);
    cuda_check(launch_gather_entries(p.R, view, d_over, m, gk, gr, ctx.sms, ctx.stream), "gather kernel");
    rs.launches += 1;
    HostChunk hc;
    hc.row = row0;
    hc.no_tail = true;
    hc.count = m;
    hc.keys.resize(m * kb);
    hc.res.resize((size_t)p.R * m);
    cuda_check(cudaMemcpyAsync(hc.keys.data(), gk, m * kb, cudaMemcpyDeviceToHost, ctx.stream), "overflow keys");
    cuda_check(cudaMemcpyAsync(hc.res.data(), gr, m * 4u * p.R, cudaMemcpyDeviceToHost, ctx.stream),
               "overflow residues");
    cuda_check(cudaStreamSynchronize(ctx.stream), "overflow synchronize");
    pending.push_back(std::move(hc));
  }
  f.count = 0;
}

// ---- queued rows ------------------------------------------------------------
//
// A small row's kernels take a few microseconds, the host's wait for its sizes
// several times that. While a boundary is expected to stay within kQueueTerms
// successor terms, its rows are queued as one chain: each row's kernels read
// the entry and term counts the row before left on the device (StepSource),
// the merges clear the partition cursors they read, and the host waits once
// for all of them. A row that does not fit the chain's buffers stops it with
// its input intact, and the host goes on from that row as before.
// Larger rows, from kQueueTerms to kLargeQueueTerms, are a chain of their own in
// the merge's 2048-candidate shape: a row that runs by itself waits about 25 us
// for its sizes. Beyond that a row runs for 2 ms and more, and its exact sizes
// save more memory than the wait costs.
constexpr u64 kQueueTerms = 4u << 20;
constexpr u64 kLargeQueueTerms = 64u << 20;

// Pinned scalars of `steps` steps and of the state before them ([0], which the
// caller fills), zero.
static StepScalars* pinned_scalars(Ctx& ctx, size_t steps) {
  const size_t n = steps + 1;
  if (ctx.h_queue_steps < n) {
    if (ctx.h_queue) cudaFreeHost(ctx.h_queue);
    ctx.h_queue = nullptr;
    ctx.h_queue_steps = 0;
    cuda_check(cudaMallocHost(&ctx.h_queue, n * sizeof(StepScalars)), "pinned step scalars");
    ctx.h_queue_steps = n;
  }
  std::memset(ctx.h_queue, 0, n * sizeof(StepScalars));
  return ctx.h_queue;
}

// The same with their copy on the device (chain_buffers has made its room).
static StepScalars* queue_scalars(Ctx& ctx, size_t steps) {
  pinned_scalars(ctx, steps);
  return static_cast<StepScalars*>(ctx.queue.ptr);
}

// Device times of a finished chain's kernels from their stamps (the host's
// time before the first launch is in neither: a kernel's first launch in a
// process takes 10 ms and more). A site step's compaction stamps its end in the
// last step only (242 stamps of N = 11 took 2 % of its time).
struct QueueTimes {
  std::vector<double> scatter, merge;  // ms per step
  double sum = 0;
};
static QueueTimes queue_times(const StepScalars* h, size_t steps, size_t queued) {
  QueueTimes t;
  for (size_t i = 1; i <= steps; ++i) {
    const StepScalars& a = h[i];
    t.scatter.push_back(a.t_merge > a.t_scatter ? (double)(a.t_merge - a.t_scatter) * 1e-6 : 0.0);
    const u64 end = a.t_end ? a.t_end : i < queued ? h[i + 1].t_scatter : 0;
    t.merge.push_back(end > a.t_merge ? (double)(end - a.t_merge) * 1e-6 : 0.0);
    t.sum += t.scatter.back() + t.merge.back();
  }
  return t;
}

// Room for a chain of `steps` steps: their scalars, a boundary of `most`
// entries and `table_bytes` of scratch, or false with the boundary and the
// scratch as they were (the rows that run instead use them; a scratch freed
// here and reserved there again, row by row, doubled the time of N = 16 in 280
// batches). Buffers that stand are not asked about again.
static bool chain_buffers(Ctx& ctx, const Plan& p, DevFrontier& f, u64 most, size_t table_bytes, size_t steps,
                          const char* what) {
  const size_t scalar_bytes = (steps + 1) * sizeof(StepScalars), eb = entry_bytes(p);
  if (!p.budget.known() && f.cap >= most && ctx.table.bytes >= table_bytes && ctx.queue.bytes >= scalar_bytes) return true;
  const auto others = [&] {
    const size_t scalars = std::max(ctx.queue.bytes, scalar_bytes);
    return ctx.pool_bytes - ctx.front[0].bytes - ctx.table.bytes - ctx.queue.bytes + scalars;
  };
  const size_t table = std::max(table_bytes, ctx.table.bytes);
  const size_t grown = f.cap < most ? most * eb : 0;  // a new boundary, beside the old one while that is copied
  const auto fits = [&](size_t boundary, size_t scratch) { return p.budget.holds(others() + boundary + scratch); };
  const auto room = [&] {
    return fits(std::max(ctx.front[0].bytes, grown), table_bytes) &&
           (!grown || fits(ctx.front[0].bytes + grown, ctx.table.bytes < table_bytes ? 0 : ctx.table.bytes));
  };
  if (!room() && !(group_release(ctx) && room())) return false;
  // The scalars come before the table, which takes what is left of the budget
  // up to a quarter more than it needs.
  if (!queue_reserve(ctx, scalar_bytes, p.budget)) return false;
  if (ctx.table.bytes < table_bytes || !fits(std::max(ctx.front[0].bytes, grown), table)) buf_release(ctx, ctx.table);
  // (A large chain's boundary is sized for its largest row, and one that leaves
  // the scratch no room when it grows ahead for what it needs.)
  const bool ahead = most <= kQueueTerms && fits(ctx.front[0].bytes + 3 * grown, table_bytes);
  return ensure_front(ctx, p, f, most, 0, ahead) && try_reserve(ctx, ctx.table, table_bytes, p.budget, what);
}

// Planned candidates per partition of a queued step. A partition that overflows
// ends the chain, and its row runs again by itself, so a fill meant for rows
// that stand alone is held six standard deviations (a partition's candidates
// are about Poisson) below the capacity: 849 of 1024 slots, where a fill of 0.9
// plans 922 and fails nearly every row of millions of terms (N = 14: 61
// launches instead of 27).
static double chain_mean(const Ctx& ctx, u32 pcap) {
  const double root = std::sqrt(9.0 + (double)pcap) - 3.0;  // mean + 6 sqrt(mean) = pcap
  return std::min(std::min(ctx.partition_fill, ctx.chain_fill) * pcap, root * root);
}

// What a chain learns from the step that ended it: a wider margin where one of
// its partitions overflowed all the same.
static void chain_ended(Ctx& ctx, const StepScalars& failed, double mean, u32 pcap) {
  if (failed.error & kErrOverflow) ctx.chain_fill = std::max(0.3, 0.8 * mean / pcap);
}

// A finished row's metrics: `in` entries with `terms` successors. `exact`:
// plane 0 carries exact sums.
static void add_row(const Plan& p, unsigned row, u64 in, u64 terms, const StepScalars& r, bool exact,
                    std::vector<RowAcc>& rows, RunStats& rs) {
  RowAcc& acc = rows[row];
  acc.used = true;
  acc.device_row = true;
  acc.input_states += in;
  acc.candidates += (u128)in * p.n;
  acc.matched += terms;
  acc.completed += terms;
  acc.output_states += r.out_count;
  for (int q = 0; q < p.Rc; ++q) {
    acc.weight_res[q] = (acc.weight_res[q] + r.weight_sum[exact ? 0 : q] % kPrimes[q]) % kPrimes[q];
    if (row + 1 == p.n) rs.final_res[q] = (rs.final_res[q] + r.final_sum[exact ? 0 : q] % kPrimes[q]) % kPrimes[q];
  }
  rs.peak_states = std::max<u64>(rs.peak_states, r.out_count);
  if (!terms) return;
  rs.merge_launches += 1;
  rs.merge_bytes += (in + r.out_count) * entry_bytes(p);
  rs.entries_in += in;
  rs.entries_out += r.out_count;
  rs.candidates += terms;
}

// A partly placed board whose boundary is expected to fit one CTA's shared
// memory, from its host entries to the last row in one launch that writes its
// scalars to pinned memory. (Whole boards report each row's time and run as
// chains.) False, with nothing added, where it does not apply or the boundary
// outgrew it.
static bool run_resident(Ctx& ctx, const Plan& p, const HostChunk& hc, std::vector<RowAcc>& rows, RunStats& rs) {
  if (!p.prefix || hc.count == 0 || hc.count > kResidentSeeds || hc.no_tail || hc.row >= p.n || p.tail_row < p.n ||
      p.batch_states <= 0 || p.batch_states > 0.5 * resident_capacity() || p.grain != QPEPS_GRAIN_ROW ||
      p.merge != QPEPS_MERGE_PARTITION || p.key_bits != 64 || p.free_rows > 20 || ctx.tune.merge_kind != 1 ||
      ctx.tune.scatter_kind != 1 || ctx.tune.fold_weights != 2 || !(p.w64 || p.R == 1))
    return false;
  const unsigned count = p.n - hc.row;
  StepScalars* h = pinned_scalars(ctx, count);
  ResidentArgs a{};
  a.n = p.n;
  a.row = hc.row;
  a.count = (u32)hc.count;
  a.out = h + 1;
  const u64 mask = (1ull << p.n) - 1;
  h[0].out_count = hc.count;
  for (u64 i = 0; i < hc.count; ++i) {
    std::memcpy(&a.key[i], &hc.keys[i * 8], 8);
    a.weight[i] = p.w64 ? (u64)hc.res[i] | ((u64)hc.res[hc.count + i] << 32) : hc.res[i];
    const State st = unpack<u64>(a.key[i], p.n, mask);
    h[0].next_terms += (u64)__builtin_popcountll(~(st.cols | st.dr | st.dl) & mask);
  }
  cuda_check(launch_resident_rows(a, ctx.stream), "resident rows kernel");
  cuda_check(cudaStreamSynchronize(ctx.stream), "resident rows");
  rs.launches += 1;
  if (h[1].error) return false;
  trim_pool(ctx, p);
  if (ctx.rec) ctx.rec->ok = false, ctx.rec->compared = true;
  ctx.h2d_bytes += sizeof a;
  ctx.d2h_bytes += count * sizeof(StepScalars);
  rs.batches += 1;
  rs.forms |= QPEPS_ROWS_ONE_CTA;
  const double ms = h[count].t_merge > h[1].t_scatter ? (double)(h[count].t_merge - h[1].t_scatter) * 1e-6 : 0.0;
  rs.device_ms += ms;
  rs.merge_ms += ms;
  rs.peak_states = std::max<u64>(rs.peak_states, hc.count);
  // (No row times: partly placed boards report none.)
  for (unsigned i = 0; i < count; ++i) add_row(p, hc.row + i, h[i].out_count, h[i].next_terms, h[i + 1], true, rows, rs);
  return true;
}

// Rows [row, stop) of the live boundary as a chain; returns how many were
// contracted (0: none, the boundary and the metrics are unchanged).
static unsigned run_queued_rows(Ctx& ctx, const Plan& p, DevFrontier& f, unsigned row, unsigned stop, u64& known_terms,
                                std::vector<RowAcc>& rows, RunStats& rs) {
  const bool wkeys = p.key_bits == 128;
  const u32 kind = ctx.tune.scatter_kind;
  if (p.grain != QPEPS_GRAIN_ROW || p.merge != QPEPS_MERGE_PARTITION || p.batch_states <= 0 || f.count == 0 ||
      row >= stop || ctx.tune.merge_kind != 1)
    return 0;
  if (!wkeys && ((kind != 0 && kind != 1 && kind != 4) || (ctx.tune.wide_merge & 1u))) return 0;
  // Terms a row may have, and those it is expected to have at most (the grids
  // are sized for these; a grid covers any number).
  // A chain of larger rows starts where a row is known to have more than a
  // chain of small ones holds.
  const bool large = known_terms != kTermsUnknown && known_terms > kQueueTerms;
  const u64 most = (u64)std::min((double)(large ? kLargeQueueTerms : kQueueTerms),
                                 std::max(1048576.0, 1.6 * p.batch_states));
  const double likely = std::min((double)most, std::max(65536.0, 1.6 * p.batch_states));
  if (f.count > most || (known_terms != kTermsUnknown && known_terms > most)) return 0;
  // Rows that may stay below that: an entry with r of n rows placed has about
  // n (1 - r / n)^2.3 successors (N = 17: 6.7 at r = 5, 3.6 at 8, 2.2 at 10, 1.3
  // at 12). Boards differ by a factor of four either way; a row too many costs
  // two launches that return at once, one too few a wait.
  unsigned count = 0;
  auto growth = [&](unsigned r) { return std::max(1.0, p.n * std::pow(1.0 - (double)r / p.n, 2.3)); };
  double expect = known_terms != kTermsUnknown ? (double)known_terms : (double)f.count * growth(row);
  while (row + count < stop &&
         (1.6 * p.batch_states <= (double)most || 2 * row > p.n || expect <= 4.0 * (double)most)) {
    ++count;
    expect *= growth(row + count);
  }
  if (count < 2) return 0;
  const size_t eb = entry_bytes(p);
  // Small merge CTAs (four an SM, 1024 candidates) where they exist: a chain's
  // scatter waits for its deepest partition cursor, and half the candidates a
  // partition halve that.
  // (Large rows scatter faster into half as many partitions.)
  const u32 shape = !wkeys && !large && wide_merge_supported(p.R) ? 2u : 0u;
  const u32 pcap = wkeys ? wide_key_partition_capacity() : partition_capacity(shape);
  const double mean = chain_mean(ctx, pcap);
  StepSource source{nullptr, mean, 0, (shape == 2 ? 8u : 2u) * (u32)ctx.sms};
  const u32 parts_cap = source.parts_cap = (u32)source.partitions(most);
  const u32 cstride = (parts_cap <= ctx.tune.spread_cursors_below) ? 8u : 1u;
  const size_t region_bytes = (size_t)parts_cap * pcap * cand_bytes(p);
  const size_t cursor_bytes = (size_t)parts_cap * 4 * cstride;
  const size_t table_bytes = region_bytes + (cursor_bytes + 255) / 256 * 256;
  if (!chain_buffers(ctx, p, f, most, table_bytes, count, "partition regions")) return 0;
  StepScalars* d = queue_scalars(ctx, count);
  StepScalars* h = ctx.h_queue;
  const auto t0 = std::chrono::steady_clock::now();
  h[0].out_count = f.count;
  if (known_terms != kTermsUnknown) h[0].next_terms = known_terms;
  void* regions = ctx.table.ptr;
  u32* cursors = reinterpret_cast<u32*>(static_cast<char*>(ctx.table.ptr) + region_bytes);
  const FrontierView view = view_of(p, ctx.front[0], f.cap);
  PartitionCfg pc{p.R, ctx.sms, parts_cap, pcap, p.R == 1 ? 3 : p.R == 2 ? 2 : 1, cstride, ctx.tune.parents_per_lane,
                  shape, kind, ctx.tune.merge_kind,
                  p.w64 ? 2u : (ctx.tune.fold_weights && p.R == 2 && p.free_rows <= 20) ? 1u : 0u};
  pc.merge_regs = ctx.tune.merge_compact;
  pc.scatter_block = ctx.tune.scatter_block;
  pc.key_bits = (uint32_t)p.key_bits;
  cuda_check(cudaMemcpyAsync(d, h, (count + 1) * sizeof(StepScalars), cudaMemcpyHostToDevice, ctx.stream),
             "queued step scalars");
  cuda_check(cudaMemsetAsync(cursors, 0, cursor_bytes, ctx.stream), "clear partition cursors");
  u64 launches = 0;
  if (known_terms == kTermsUnknown) {
    cuda_check(launch_row_count(LaunchCfg{p.key_bits, p.R, p.threads, ctx.sms}, view, f.count, p.n, d, ctx.stream),
               "row count kernel");
    launches += 1;
  }
  cuda_check(cudaEventRecord(ctx.ev[0], ctx.stream), "event");
  // Grid bounds: a row's entries are at most the terms of the row before.
  u64 entries = f.count;
  double terms = known_terms != kTermsUnknown ? (double)known_terms : (double)f.count * p.n;
  for (unsigned i = 0; i < count; ++i) {
    const double fits = std::min(likely, terms);
    pc.queued = source;
    pc.queued.prev = d + i;
    pc.parts = (u32)source.partitions((u64)fits);
    cuda_check(launch_partition_scatter(pc, view, entries, p.n, regions, cursors, d + i + 1, ctx.stream),
               "partition scatter kernel");
    cuda_check(launch_partition_merge(pc, regions, cursors, view, p.n, row + i + 1 < p.n, d + i + 1, ctx.stream),
               "partition merge kernel");
    launches += 2;
    entries = (u64)fits;
    terms = fits * (p.n - (row + i + 1));
  }
  cuda_check(cudaEventRecord(ctx.ev[1], ctx.stream), "event");
  cuda_check(cudaMemcpyAsync(h, d, (count + 1) * sizeof(StepScalars), cudaMemcpyDeviceToHost, ctx.stream),
             "read step scalars");
  cuda_check(cudaStreamSynchronize(ctx.stream), "queued rows");
  ctx.h2d_bytes += (count + 1) * sizeof(StepScalars);
  ctx.d2h_bytes += (count + 1) * sizeof(StepScalars);
  rs.launches += launches;
  float ms = 0;
  cudaEventElapsedTime(&ms, ctx.ev[0], ctx.ev[1]);
  rs.device_ms += ms;
  unsigned done = 0;
  while (done < count && !h[done + 1].error) ++done;
  if (done < count) chain_ended(ctx, h[done + 1], mean, pcap);
  if (done < count && (h[done + 1].error & kErrBounds))
    fail(QPEPS_ERR_CUDA, row_msg("a kernel's bounds check failed (access skipped) at row", row + done + 1));
  const QueueTimes times = queue_times(h, done, count);
  const double wall = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
  for (unsigned i = 0; i < done; ++i) {
    const StepScalars& r = h[i + 1];
    const u64 in = i ? h[i].out_count : f.count, tm = h[i].next_terms;
    const bool last = row + i + 1 == p.n;
    if (p.w64) {
      // The certificate of the row, as before a row that runs by itself.
      const u128 bound = f.weight_bound * (u128)(p.n - (row + i));
      if (bound >> 63) fail(QPEPS_ERR_OVERFLOW, row_msg("exact 64-bit weights are not certified at row", row + i + 1));
      f.weight_bound = r.weight_sum[0];
    }
    rows[row + i].elapsed += times.sum > 0 ? wall * (times.scatter[i] + times.merge[i]) / times.sum : 0.0;
    if (tm) {
      rs.scatter_ms += times.scatter[i];
      rs.merge_ms += times.merge[i];
    }
    add_row(p, row + i, in, tm, r, p.w64, rows, rs);
    if (ctx.rec) {
      // What the row would have recorded by itself.
      GraphStepRec g;
      if (tm) {
        g.pc = pc;
        g.pc.queued = StepSource{};
        g.pc.parts = (u32)source.partitions(tm);
        g.pc.cursor_stride = (g.pc.parts <= ctx.tune.spread_cursors_below) ? 8u : 1u;
        g.n_in = in;
        g.terms = tm;
        g.out = r.out_count;
        g.need_cap = last ? in : std::max(in, tm);
        g.region_bytes = (size_t)g.pc.parts * pcap * cand_bytes(p);
        g.table_bytes = g.region_bytes + ((size_t)g.pc.parts * 4 * g.pc.cursor_stride + 255) / 256 * 256;
        g.final_step = last;
        for (int q = 0; q < p.R; ++q) {
          g.weight_sum[q] = r.weight_sum[q];
          g.final_sum[q] = r.final_sum[q];
        }
      }
      if (ctx.rec->chunks.empty())
        ctx.rec->ok = false;
      else
        ctx.rec->chunks.back().steps.push_back(g);
    }
  }
  if (done) {
    rs.forms |= QPEPS_ROWS_CHAIN;
    const bool ended = row + done == p.n;
    f.count = ended ? 0 : h[done].out_count;
    known_terms = h[done].next_terms;
  } else if (known_terms == kTermsUnknown) {
    known_terms = h[0].next_terms;
  }
  return done;
}

// The per-site form's sites from (row, 0) on as a chain: two kernels a site
// (expand and insert, compact), each site's table sized on the device from the
// terms the compaction before counted. Returns the sites contracted; the row
// of the first one left has its counters added when it is not its first.
static u64 run_queued_sites_plain(Ctx& ctx, const Plan& p, DevFrontier& f, unsigned row, unsigned stop,
                                  std::vector<RowAcc>& rows, RunStats& rs) {
  if (p.grain != QPEPS_GRAIN_SITE || p.batch_states <= 0 || f.count == 0 || row >= stop) return 0;
  // A boundary inside a row holds the placed and the unplaced states.
  const double largest = 4.0 * p.batch_states;
  const u64 most = (u64)std::min((double)kQueueTerms, std::max(65536.0, largest));
  if (f.count > most / 2) return 0;
  unsigned count = 0;  // rows expected to stay below that
  double expect = (double)f.count;
  while (row + count < stop && (largest <= (double)most || 4.0 * expect <= (double)most)) {
    expect *= std::max(1.5, (double)p.n - 2.2 * (row + count));
    ++count;
  }
  if (count == 0) return 0;
  const size_t eb = entry_bytes(p);
  TableSource source;
  source.slots_cap = source.slots(most);
  const size_t table_bytes = source.slots_cap * slot_bytes(p.key_bits, p.R);
  const size_t sites = (size_t)count * p.n;
  if (!chain_buffers(ctx, p, f, most, table_bytes, sites, "hash table")) return 0;
  StepScalars* d = queue_scalars(ctx, sites);
  StepScalars* h = ctx.h_queue;
  const auto t0 = std::chrono::steady_clock::now();
  h[0].out_count = f.count;
  const LaunchCfg cfg{p.key_bits, p.R, p.threads, ctx.sms};
  const FrontierView view = view_of(p, ctx.front[0], f.cap);
  // The first site's terms are at most two an entry; its row's counters come
  // from a count of their own.
  h[0].next_terms = 2 * f.count;
  cuda_check(cudaMemcpyAsync(d, h, (sites + 1) * sizeof(StepScalars), cudaMemcpyHostToDevice, ctx.stream),
             "queued step scalars");
  cuda_check(cudaMemsetAsync(ctx.d_sc, 0, sizeof(StepScalars), ctx.stream), "clear step scalars");
  cuda_check(cudaMemsetAsync(ctx.table.ptr, 0, table_bytes, ctx.stream), "clear hash table");
  cuda_check(launch_row_count(cfg, view, f.count, p.n, ctx.d_sc, ctx.stream), "row count kernel");
  cuda_check(cudaEventRecord(ctx.ev[0], ctx.stream), "event");
  u64 entries = f.count;
  for (size_t i = 0; i < sites; ++i) {
    const unsigned r = row + (unsigned)(i / p.n), site = (unsigned)(i % p.n);
    const u64 fits = std::min<u64>(most, 2 * entries);
    source.prev = d + i;
    source.last = i + 1 == sites;
    const bool last = r + 1 == p.n && site + 1 == p.n;
    cuda_check(launch_site_expand_insert(cfg, view, entries, p.n, site, ctx.table.ptr, source.slots(fits), d + i + 1,
                                         ctx.stream, source),
               "site expand-insert kernel");
    cuda_check(launch_compact(cfg, ctx.table.ptr, source.slots(fits), view, p.n, !last, d + i + 1, ctx.stream, source,
                              site + 1 == p.n ? 0u : site + 1),
               "compact kernel");
    entries = fits;
  }
  cuda_check(cudaEventRecord(ctx.ev[1], ctx.stream), "event");
  cuda_check(cudaMemcpyAsync(h, d, (sites + 1) * sizeof(StepScalars), cudaMemcpyDeviceToHost, ctx.stream),
             "read step scalars");
  sync_scalars(ctx);
  ctx.h2d_bytes += (sites + 1) * sizeof(StepScalars);
  ctx.d2h_bytes += (sites + 1) * sizeof(StepScalars);
  rs.launches += 1 + 2 * sites;
  float ms = 0;
  cudaEventElapsedTime(&ms, ctx.ev[0], ctx.ev[1]);
  rs.device_ms += ms;
  size_t done = 0;
  while (done < sites && !h[done + 1].error) ++done;
  if (done < sites && (h[done + 1].error & kErrProbeLimit))
    fail(QPEPS_ERR_CAPACITY, row_msg("hash probe bound exceeded at row", row + (unsigned)(done / p.n) + 1));
  const QueueTimes times = queue_times(h, done, sites);
  const double wall = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
  if (ctx.rec) ctx.rec->ok = false;
  for (size_t i = 0; i < done; ++i) {
    const StepScalars& r = h[i + 1];
    const unsigned at = row + (unsigned)(i / p.n), site = (unsigned)(i % p.n);
    const u64 in = i ? h[i].out_count : f.count;
    RowAcc& acc = rows[at];
    acc.used = true;
    acc.device_row = true;
    if (site == 0) {
      const u64 examined = i ? h[i].sitewise_examined : ctx.h_sc->sitewise_examined;
      acc.input_states += in;
      acc.completed += i ? h[i].row_terms : ctx.h_sc->terms;
      acc.examined += examined;
      acc.tmatched += examined;
    }
    if (r.terms) {
      rs.scatter_ms += times.scatter[i];
      rs.merge_ms += times.merge[i];
      rs.merge_launches += 1;
      rs.merge_bytes += (in + r.out_count) * eb;
      rs.entries_in += in;
      rs.entries_out += r.out_count;
    }
    acc.elapsed += times.sum > 0 ? wall * (times.scatter[i] + times.merge[i]) / times.sum : 0.0;
    // (The first site's terms are a bound; what it merged is exact.)
    rs.candidates += i ? r.terms : r.out_count;
    if (site + 1 == p.n) {
      const bool last = at + 1 == p.n;
      acc.output_states += r.out_count;
      for (int q = 0; q < p.Rc; ++q) {
        acc.weight_res[q] = (acc.weight_res[q] + r.weight_sum[q] % kPrimes[q]) % kPrimes[q];
        if (last) rs.final_res[q] = (rs.final_res[q] + r.final_sum[q] % kPrimes[q]) % kPrimes[q];
      }
      rs.peak_states = std::max<u64>(rs.peak_states, r.out_count);
    }
  }
  if (done) rs.forms |= QPEPS_ROWS_CHAIN;
  if (done) f.count = row + done / p.n == p.n ? 0 : h[done].out_count;
  return done;
}

// ---- column-grouped rows (qpeps_group_kernels.cu) ---------------------------
//
// All rows of a device batch are queued at once: a row's plan and pull read
// the sizes they need from the previous row's scalars on the device, so the
// host waits once, at the end. A row whose output does not fit its buffer
// marks itself and the rows after it return at once; the host grows the buffer
// to the size the row counted and queues the rows again from there, the row's
// input being untouched.

struct GroupBinomials {
  u32 v[(kGroupMaxN + 2) * (kGroupMaxN + 2)];
  GroupBinomials() {
    constexpr unsigned d = kGroupMaxN + 2;
    for (unsigned i = 0; i < d; ++i)
      for (unsigned k = 0; k < d; ++k)
        v[i * d + k] = k == 0 ? 1u : i == 0 ? 0u : v[(i - 1) * d + k] + v[(i - 1) * d + k - 1];
  }
  u32 at(unsigned i, unsigned k) const { return v[i * (kGroupMaxN + 2) + k]; }
};
static const GroupBinomials kBinomials;

// A seed boundary in the grouped layout: packed entries and their buckets.
struct GroupSeed {
  std::vector<u32> keys, weights;
  std::vector<GroupSeedUnit> units;
  GroupRow row{};
};

// Host entries beyond this are not regrouped (halves of a boundary split off
// under memory pressure): they take the partitioned merge.
constexpr u64 kGroupMaxSeeds = 4096;

// Top u bits implied by the bucket, so that the stored diagonals fit 32 bits.
static unsigned group_implied_bits(unsigned n) { return 2 * n - 2 > 32 ? 2 * n - 2 - 32 : 0; }

// Expected largest boundary that column-grouped rows are to hold, 0 where the
// partitioned rows are faster. A row costs about 2 us a CTA and bucket besides
// its entries, so the line lies at 1200 expected entries a bucket: `states` over
// the column sets of the board's middle (C(N - k, (N - k) / 2) below k placed
// rows) and the buckets a set has at least. Device ms at N = 15 / 16 / 17 / 18
// (2.8, 8.2, 29 and 4.9 K entries a bucket): grouped 1.96 / 8.3 / 53.4 / 481,
// partitioned 2.4 / 15.6 / 117 / 821; N = 14 without the orbits (1.7 K) 0.90
// against 1.08, N = 16 below one row (2 K) 1.75 to 2.04 against 1.67 to 2.32;
// N = 14 (0.8 K) 0.70 against 0.53, N = 18 below two rows (0.6 K) 5.4 to 7.2
// against 3.8 to 8.2. Repeated contractions (use_graph) keep the rows that a
// graph can replay up to 200 M entries. `room`: the buffers' size over the
// expected one.
static double group_rows_states(unsigned n, unsigned placed, double states, double room, bool replay) {
  if (n > kGroupMaxN) return 0.0;
  const unsigned left = n - std::min(placed, n);
  const double buckets = (double)kBinomials.at(left, left / 2) * (1u << group_implied_bits(n));
  return states >= std::max(1200.0 * buckets, replay ? 200e6 : 0.0) ? states * room : 0.0;
}

static bool group_applies(const Ctx& ctx, const Plan& p, const HostChunk& hc) {
  // Exact weights: two words (w64; the seed's high words are zero), or one
  // residue below which every weight stays (R = 1: (N - k)! < p0). The
  // claim-list merge and the window scatter stand for the default row step;
  // other kinds of the tuning keep their own kernels.
  const bool exact = p.w64 || (p.R == 1 && ctx.tune.fold_weights == 2 && ctx.tune.merge_kind == 1);
  return p.group_states > 0 && exact && p.merge == QPEPS_MERGE_PARTITION && p.grain == QPEPS_GRAIN_ROW &&
         p.key_bits == 64 && p.tail_row >= p.n && p.n <= kGroupMaxN && p.free_rows <= 20 &&
         ctx.tune.scatter_kind == 1 && ctx.tune.merge_compact == 0 && hc.count > 0 && hc.count <= kGroupMaxSeeds &&
         !hc.no_tail && hc.row >= 1 && hc.row < p.n &&
         (p.R == 1 || std::all_of(hc.res.begin() + hc.count, hc.res.begin() + 2 * hc.count,
                                  [](u32 high) { return high == 0; }));
}

static GroupSeed group_seed(const Plan& p, const HostChunk& hc) {
  const unsigned n = p.n, rm = group_implied_bits(n), nu = n - 1 - rm;
  const u64 mask = (1ull << n) - 1;
  struct E {
    u64 cols;
    u32 bucket, quarter, key, w;
  };
  std::vector<E> es(hc.count);
  GroupSeed sd;
  for (u64 i = 0; i < hc.count; ++i) {
    u64 k;
    std::memcpy(&k, &hc.keys[i * 8], 8);
    const State st = unpack<u64>(k, n, mask);
    E& e = es[i];
    e.cols = st.cols;
    e.bucket = (u32)(st.dr >> (n - rm));
    e.quarter = (u32)(st.dr >> (n - 2 - rm)) & 3u;
    e.key = (u32)((st.dr >> 1) & ((1ull << nu) - 1)) | (u32)(st.dl << nu);
    e.w = hc.res[i];
    sd.row.next_terms += (u64)__builtin_popcountll(~(st.cols | st.dr | st.dl) & mask);
    sd.row.weight_sum += e.w;
    sd.row.weight_max = std::max<unsigned long long>(sd.row.weight_max, e.w);
  }
  std::sort(es.begin(), es.end(), [](const E& a, const E& b) {
    return a.cols != b.cols ? a.cols < b.cols : a.bucket != b.bucket ? a.bucket < b.bucket : a.quarter < b.quarter;
  });
  size_t group = 0;  // its first bucket in sd.units
  for (u64 i = 0; i < hc.count; ++i) {
    const E& e = es[i];
    if (i == 0 || es[i - 1].cols != e.cols) {
      u32 rank = 0, j = 0;
      for (u64 left = e.cols; left; left &= left - 1) rank += kBinomials.at((unsigned)__builtin_ctzll(left), ++j);
      group = sd.units.size();
      for (u32 q = 0; q < (1u << rm); ++q)
        sd.units.push_back(GroupSeedUnit{(u32)i, (u32)sd.units.size(), 0u, 0u, rank, rm, 0u});
    }
    GroupSeedUnit& un = sd.units[group + e.bucket];
    if (!(un.quarters01 | un.quarters23)) un.first = (u32)i;
    (e.quarter & 2u ? un.quarters23 : un.quarters01) += e.quarter & 1u ? 0x10000u : 1u;
    sd.units[group].total += 1;
    sd.keys.push_back(e.key);
    sd.weights.push_back(e.w);
  }
  sd.row.out_count = hc.count;
  sd.row.merge_rate = 1.f;
  return sd;
}

constexpr size_t kGroupEntryBytes = 8;  // key, weight

// Layout of Ctx::grp_dir.
struct GroupDirs {
  u32 groups = 0, unit_cap = 0;
  size_t off_gdir[2], off_udir[2], off_units, off_rows, off_bin, off_list, bytes;
};
static GroupDirs group_dirs(unsigned n, unsigned row0, u64 cap, u64 seed_units) {
  GroupDirs d;
  for (unsigned m = row0; m <= n; ++m) d.groups = std::max(d.groups, kBinomials.at(n, m));
  // A group takes 2^rm buckets at least; beyond that buckets are cut so that
  // more than half the target is expected in each, and cut units add pieces.
  const u64 most = ((u64)d.groups << group_implied_bits(n)) + (u64)(4.0 * (double)cap / group_unit_target()) + 65536 +
                   seed_units;
  d.unit_cap = (u32)std::min<u64>(most, 0x7fffffffu);
  size_t o = 0;
  auto take = [&](size_t b) {
    const size_t at = o;
    o += (b + 255) / 256 * 256;
    return at;
  };
  for (int i = 0; i < 2; ++i) d.off_gdir[i] = take((size_t)d.groups * sizeof(GroupDir));
  for (int i = 0; i < 2; ++i) d.off_udir[i] = take((size_t)d.unit_cap * sizeof(uint4));
  d.off_units = take((size_t)d.unit_cap * sizeof(uint2));
  d.off_rows = take((kGroupMaxN + 1) * sizeof(GroupRow));
  d.off_bin = take(sizeof kBinomials.v);
  d.off_list = take((size_t)std::max<u64>(seed_units, 1) * sizeof(GroupSeedUnit));
  d.bytes = o;
  return d;
}

// Grow-only, exact when the budget is near; false when it does not fit.
static bool group_reserve(Ctx& ctx, DevBuf& b, size_t bytes, const Budget& budget) {
  if (b.bytes >= bytes) return true;
  if (ctx.pool_bytes - b.bytes + bytes > budget) buf_release(ctx, ctx.table);
  if (ctx.pool_bytes - b.bytes + bytes > budget) buf_release(ctx, ctx.front[0]);
  if (ctx.pool_bytes - b.bytes + bytes > budget) return false;
  buf_release(ctx, b);
  if (cudaMalloc(&b.ptr, bytes) != cudaSuccess) {
    cudaGetLastError();
    b.ptr = nullptr;
    return false;
  }
  b.bytes = bytes;
  ctx.pool_bytes += bytes;
  ctx.peak_pool_bytes = std::max(ctx.peak_pool_bytes, ctx.pool_bytes);
  ++ctx.pool_gen;
  return true;
}

// The row step's arguments from the buffers as they stand: boundaries
// alternate sides, the seed (m = row0) on side 0.
static GroupStepArgs group_args(const Ctx& ctx, const Plan& p, const GroupDirs& d, unsigned row0, unsigned m) {
  char* base = static_cast<char*>(ctx.grp_dir.ptr);
  auto side = [&](unsigned i) {
    GroupSide s{};
    s.cap = std::min<u64>(ctx.grp_side[i].bytes / kGroupEntryBytes, 0xfffffff0ull);
    s.keys = static_cast<u32*>(ctx.grp_side[i].ptr);
    s.lo = s.keys + s.cap;
    s.gdir = reinterpret_cast<GroupDir*>(base + d.off_gdir[i]);
    s.udir = reinterpret_cast<uint4*>(base + d.off_udir[i]);
    s.unit_cap = d.unit_cap;
    return s;
  };
  GroupStepArgs a{};
  a.in = side((m - 1 - row0) & 1u);
  a.out = side((m - row0) & 1u);
  GroupRow* rows = reinterpret_cast<GroupRow*>(base + d.off_rows);
  a.prev = rows + (m - 1);
  a.row = rows + m;
  a.units = reinterpret_cast<uint2*>(base + d.off_units);
  a.binomials = reinterpret_cast<const u32*>(base + d.off_bin);
  a.n = p.n;
  a.m = m;
  a.rm = group_implied_bits(p.n);
  a.max_bits = std::min(12u, p.n - 4);
  a.write_out = m < p.n;
  a.block = group_block(p.group_states, ctx.sms);
  a.target = group_unit_target();
  a.share = group_unit_share(ctx.sms);
  return a;
}

static void* group_pinned(Ctx& ctx, size_t bytes) {
  if (ctx.grp_pin_bytes < bytes) {
    if (ctx.grp_pin) cudaFreeHost(ctx.grp_pin);
    ctx.grp_pin = nullptr;
    ctx.grp_pin_bytes = 0;
    cuda_check(cudaMallocHost(&ctx.grp_pin, bytes + bytes / 2), "pinned row scalars");
    ctx.grp_pin_bytes = bytes + bytes / 2;
  }
  return ctx.grp_pin;
}

// Contract one batch with column-grouped rows. False (and nothing added to
// the metrics) where they do not apply or the budget does not hold them.
static bool run_chunk_grouped(Ctx& ctx, const Plan& p, const HostChunk& hc, std::vector<RowAcc>& rows, RunStats& rs) {
  if (!group_applies(ctx, p, hc)) return false;
  const unsigned n = p.n, row0 = hc.row;
  const auto t0 = std::chrono::steady_clock::now();
  const GroupSeed sd = group_seed(p, hc);
  const u64 cap = std::max<u64>(group_capacity(p.group_states, ctx.sms), hc.count);
  if (cap > 0xfffffff0ull) return false;
  const GroupDirs d = group_dirs(n, row0, std::max<u64>(cap, ctx.grp_side[0].bytes / kGroupEntryBytes), sd.units.size());
  size_t others = ctx.pool_bytes - ctx.front[0].bytes - ctx.table.bytes;  // what stays beside the two sides
  for (const DevBuf* b : {&ctx.grp_side[0], &ctx.grp_side[1], &ctx.grp_dir}) others -= b->bytes;
  if (2 * cap * kGroupEntryBytes + d.bytes + others > p.budget) return false;
  if (ctx.pool_bytes > p.budget) {
    buf_release(ctx, ctx.table);
    buf_release(ctx, ctx.front[0]);
    if (ctx.pool_bytes > p.budget) group_release(ctx);
  }
  for (int i = 0; i < 2; ++i)
    if (!group_reserve(ctx, ctx.grp_side[i], cap * kGroupEntryBytes, p.budget)) return false;
  if (!group_reserve(ctx, ctx.grp_dir, d.bytes, p.budget)) return false;
  // Upload the seed: one pinned image, its parts copied to their places.
  const size_t ns = sd.keys.size();
  const size_t seed_bytes = ns * 8 + sd.units.size() * sizeof(GroupSeedUnit);
  const size_t rows_bytes = (kGroupMaxN + 1) * sizeof(GroupRow);
  char* pin = static_cast<char*>(group_pinned(ctx, 2 * rows_bytes + sizeof kBinomials.v + seed_bytes + 256));
  GroupRow* h_rows = reinterpret_cast<GroupRow*>(pin);  // read back
  size_t o = rows_bytes;
  uint64_t h2d = 0;
  char* base = static_cast<char*>(ctx.grp_dir.ptr);
  auto put = [&](void* dst, const void* src, size_t bytes, const char* what) {
    std::memcpy(pin + o, src, bytes);
    cuda_check(cudaMemcpyAsync(dst, pin + o, bytes, cudaMemcpyHostToDevice, ctx.stream), what);
    o += (bytes + 15) / 16 * 16;
    h2d += bytes;
  };
  cuda_check(cudaEventRecord(ctx.ev[0], ctx.stream), "event");
  const GroupStepArgs a0 = group_args(ctx, p, d, row0, row0 + 1);
  std::vector<GroupRow> init(kGroupMaxN + 1);
  init[row0] = sd.row;
  put(base + d.off_rows, init.data(), rows_bytes, "row scalars");
  put(base + d.off_bin, kBinomials.v, sizeof kBinomials.v, "binomials");
  put(a0.in.keys, sd.keys.data(), ns * 4, "seed keys");
  put(a0.in.lo, sd.weights.data(), ns * 4, "seed weights");
  put(base + d.off_list, sd.units.data(), sd.units.size() * sizeof(GroupSeedUnit), "seed buckets");
  cuda_check(cudaMemsetAsync(a0.in.gdir, 0, (size_t)kBinomials.at(n, row0) * sizeof(GroupDir), ctx.stream),
             "clear seed directory");
  cuda_check(launch_group_seed(reinterpret_cast<const GroupSeedUnit*>(base + d.off_list), (u32)sd.units.size(), a0.in,
                               ctx.stream),
             "group seed kernel");
  uint64_t launches = 1;

  unsigned from = row0 + 1;
  for (int attempt = 0;; ++attempt) {
    for (unsigned m = from; m <= n; ++m) {
      const GroupStepArgs a = group_args(ctx, p, d, row0, m);
      cuda_check(launch_group_plan(a, kBinomials.at(n, m), ctx.stream), "group plan kernel");
      cuda_check(launch_group_pull(a, ctx.sms, ctx.stream), "group pull kernel");
      launches += 2;
    }
    cuda_check(cudaEventRecord(ctx.ev[1], ctx.stream), "event");
    cuda_check(cudaMemcpyAsync(h_rows, base + d.off_rows, rows_bytes, cudaMemcpyDeviceToHost, ctx.stream),
               "read row scalars");
    cuda_check(cudaStreamSynchronize(ctx.stream), "grouped rows");
    ctx.d2h_bytes += rows_bytes;
    unsigned bad = 0;
    for (unsigned m = from; m <= n && !bad; ++m)
      if (h_rows[m].error) bad = m;
    if (!bad) break;
    // Run again from the row that failed; its input stands.
    const GroupRow& r = h_rows[bad];
    if (attempt >= 40 || (r.error & kErrBounds)) return false;
    // (More units or pieces than the directory holds, or weights beyond 32 bits:
    // the partitioned rows take the batch.)
    if ((r.error & kErrNeedWide) || r.units + r.pieces > d.unit_cap) return false;
    const unsigned side = (bad - row0) & 1u;
    const u64 need = (u64)r.alloc + r.alloc / 8 + 4096;
    if (need > 0xfffffff0ull || !group_reserve(ctx, ctx.grp_side[side], need * kGroupEntryBytes, p.budget)) return false;
    cuda_check(cudaMemsetAsync(base + d.off_rows + bad * sizeof(GroupRow), 0, (n + 1 - bad) * sizeof(GroupRow),
                               ctx.stream),
               "clear row scalars");
    from = bad;
  }
  float ms = 0;
  cudaEventElapsedTime(&ms, ctx.ev[0], ctx.ev[1]);

  // Certify the weights as the row-by-row path does: a row's output total is
  // at most its input total times its free columns.
  u128 total = 0;
  for (u64 i = 0; i < hc.count; ++i) total += p.R == 1 ? hc.res[i] : (u64)hc.res[i] | ((u64)hc.res[hc.count + i] << 32);
  for (unsigned m = row0 + 1; m <= n; ++m) {
    if ((total * (u128)(n - m + 1)) >> 63)
      fail(QPEPS_ERR_OVERFLOW, row_msg("exact 64-bit weights are not certified at row", m));
    total = h_rows[m].weight_sum;
  }
  if (ctx.rec) ctx.rec->ok = false, ctx.rec->compared = true;
  ctx.h2d_bytes += h2d;
  rs.batches += 1;
  rs.forms |= QPEPS_ROWS_GROUPED;
  rs.launches += launches;
  rs.device_ms += ms;
  rs.peak_states = std::max<u64>(rs.peak_states, hc.count);
  u64 in = hc.count, terms = sd.row.next_terms;
  u64 ns_all = 0;
  for (unsigned m = row0 + 1; m <= n; ++m) ns_all += h_rows[m].t_end > h_rows[m].t_plan ? h_rows[m].t_end - h_rows[m].t_plan : 0;
  const double wall = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
  for (unsigned m = row0 + 1; m <= n; ++m) {
    const GroupRow& r = h_rows[m];
    RowAcc& acc = rows[m - 1];
    acc.used = true;
    acc.device_row = true;
    acc.input_states += in;
    acc.candidates += (u128)in * n;
    acc.matched += terms;
    acc.completed += terms;
    acc.output_states += r.out_count;
    for (int q = 0; q < p.Rc; ++q) acc.weight_res[q] = (acc.weight_res[q] + r.weight_sum % kPrimes[q]) % kPrimes[q];
    if (m == n)
      for (int q = 0; q < p.Rc; ++q) rs.final_res[q] = (rs.final_res[q] + r.weight_sum % kPrimes[q]) % kPrimes[q];
    const u64 t = r.t_end > r.t_plan ? r.t_end - r.t_plan : 0;
    acc.elapsed += ns_all ? wall * (double)t / (double)ns_all : 0.0;
    if (terms) {
      rs.scatter_ms += r.t_pull > r.t_plan ? (double)(r.t_pull - r.t_plan) * 1e-6 : 0.0;
      rs.merge_ms += r.t_end > r.t_pull ? (double)(r.t_end - r.t_pull) * 1e-6 : 0.0;
      rs.merge_launches += 1;
      rs.merge_bytes += (in + r.out_count) * kGroupEntryBytes;
      rs.entries_in += in;
      rs.entries_out += r.out_count;
      rs.candidates += terms;
    }
    rs.peak_states = std::max<u64>(rs.peak_states, r.out_count);
    in = r.out_count;
    terms = r.next_terms;
  }
  return true;
}


// Contract every pending chunk to the last row. Each chunk is one merged
// device boundary; under memory pressure a boundary is halved and the upper
// half parked on the host (exact: the contraction is linear in the boundary).
static void run_chunks(Ctx& ctx, const Plan& p, std::vector<HostChunk> pending, std::vector<RowAcc>& rows,
                       RunStats& rs) {
  DevFrontier f;
  buf_release(ctx, ctx.front[1]);
  // The boundary buffer persists across calls; its plane stride follows this
  // plan's entry size.
  f.cap = ctx.front[0].ptr ? ctx.front[0].bytes / entry_bytes(p) : 0;
  while (!pending.empty()) {
    HostChunk hc = std::move(pending.back());
    pending.pop_back();
    if (run_resident(ctx, p, hc, rows, rs)) continue;
    if (run_chunk_grouped(ctx, p, hc, rows, rs)) continue;
    f.cap = ctx.front[0].ptr ? ctx.front[0].bytes / entry_bytes(p) : 0;  // (it may have been given back)
    upload_chunk(ctx, p, hc, f);
    rs.batches += 1;
    rs.peak_states = std::max<u64>(rs.peak_states, f.count);
    unsigned site0 = hc.site;
    bool counted = hc.row_counted;
    u64 known_terms = kTermsUnknown;  // successor count of the live boundary, when a merge counted it
    const unsigned stop = hc.no_tail ? p.n : std::max(p.tail_row, hc.row);
    for (unsigned row = hc.row; row < stop; ++row) {
      if (const unsigned queued = run_queued_rows(ctx, p, f, row, stop, known_terms, rows, rs)) {
        row += queued - 1;
        continue;
      }
      if (site0 == 0 && !counted)
        if (const u64 sites = run_queued_sites_plain(ctx, p, f, row, stop, rows, rs)) {
          row += (unsigned)(sites / p.n);
          site0 = (unsigned)(sites % p.n);
          counted = site0 != 0;
          if (row >= stop) break;
        }
      const auto t0 = std::chrono::steady_clock::now();
      const bool last_row = row + 1 == p.n;
      RowAcc& acc = rows[row];
      acc.used = true;
      acc.device_row = true;
      StepOut so;
      if (p.grain == QPEPS_GRAIN_SITE) {
        if (!counted) {
          // The sitewise backend's counters: C entries matched per parent
          // (counted on the device from the row's input keys), no row
          // operator counts.
          const u64 row_terms = count_terms(ctx, p, f, false, 0, rs);
          acc.input_states += f.count;
          acc.completed += row_terms;
          if (f.count) {  // count_terms ran the count kernel
            acc.examined += ctx.h_sc->sitewise_examined;
            acc.tmatched += ctx.h_sc->sitewise_examined;
          }
        }
        for (unsigned site = site0; site < p.n; ++site) {
          const bool fin = last_row && site + 1 == p.n;
          while (merge_step(ctx, p, f, true, site, fin, rs, row, &so) == StepStatus::NeedSplit)
            split_to_host(ctx, p, f, row, site, true, hc.no_tail, pending);
          if (fin)
            for (int r = 0; r < p.Rc; ++r) rs.final_res[r] = (rs.final_res[r] + so.final_sum[r]) % kPrimes[r];
        }
        site0 = 0;
        counted = false;
      } else {
        if (p.w64) {
          // Every entry has at most n - row successors, so the output's
          // weights and per-key sums are at most (input total) * (n - row);
          // the words hold them exactly while that stays below 2^63.
          const u128 bound = f.weight_bound * (u128)(p.n - row);
          if (bound >> 63) fail(QPEPS_ERR_OVERFLOW, row_msg("exact 64-bit weights are not certified at row", row + 1));
        }
        while (merge_step(ctx, p, f, false, 0, last_row, rs, row, &so, known_terms) == StepStatus::NeedSplit) {
          split_to_host(ctx, p, f, row, 0, false, hc.no_tail, pending);
          known_terms = kTermsUnknown;  // the boundary was halved
        }
        known_terms = so.next_terms;
        if (p.w64) f.weight_bound = so.exact_sum;
        acc.input_states += so.in;
        acc.candidates += (u128)so.in * p.n;
        acc.matched += so.terms;
        acc.completed += so.terms;
        if (last_row)
          for (int r = 0; r < p.Rc; ++r) rs.final_res[r] = (rs.final_res[r] + so.final_sum[r]) % kPrimes[r];
      }
      acc.output_states += last_row ? so.out : f.count;
      for (int r = 0; r < p.Rc; ++r) acc.weight_res[r] = (acc.weight_res[r] + so.weight[r]) % kPrimes[r];
      rs.peak_states = std::max<u64>(rs.peak_states, last_row ? so.out : f.count);
      acc.elapsed += std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    }
    if (stop < p.n && f.count > 0) run_tail(ctx, p, f, stop, rows, rs, pending);
  }
}

// Host expansion of one row over a merged item list (used for the first
// row(s) that seed slices): compiled successor + optional orbit weights,
// merged by key (checked u128).
// With `sitewise` (site granularity) the row's counters are those of the
// reference's sitewise backend: C entries matched per parent, and no row
// operator counts (src/lib.rs:5633-5750).
static std::vector<Item> host_expand(unsigned n, const std::vector<Item>& in, unsigned row, bool orbit, RowAcc& acc,
                                     bool sitewise) {
  const u64 mask = (n >= 64) ? ~0ull : ((1ull << n) - 1);
  std::map<u128, u128> next;
  acc.used = true;
  acc.input_states = in.size();
  for (const Item& it : in) {
    State s = unpack<u128>(it.key, n, mask);
    u64 fr = ~(s.cols | s.dr | s.dl) & mask;
    if (sitewise) {
      acc.examined += sitewise_entries(fr, n);
      acc.tmatched += sitewise_entries(fr, n);
    } else {
      acc.candidates += n;
    }
    while (fr) {
      const u64 b = fr & (~fr + 1);
      fr &= fr - 1;
      if (!sitewise) acc.matched += 1;
      u128 w = it.weight;
      if (row == 0 && orbit) {
        const unsigned c = (unsigned)__builtin_ctzll(b), mirror = n - 1 - c;
        if (c > mirror) continue;
        if (c < mirror && !mul_u128(w, 2, &w)) fail(QPEPS_ERR_OVERFLOW, "coefficient overflow in D4 orbit weighting");
      }
      acc.completed += 1;
      u128& dst = next[row_successor<u128>(s, b, n, mask)];
      if (!add_u128(dst, w, &dst)) fail(QPEPS_ERR_OVERFLOW, row_msg("coefficient overflow after row", row + 1));
    }
  }
  std::vector<Item> out;
  out.reserve(next.size());
  for (auto& kv : next) {
    out.push_back(Item{kv.first, kv.second});
    if (!add_u128(acc.weight_exact, kv.second, &acc.weight_exact))
      fail(QPEPS_ERR_OVERFLOW, row_msg("coefficient sum overflow after row", row + 1));
  }
  acc.output_states = out.size();
  return out;
}

struct Contraction {
  u128 count = 0;
  uint64_t h2d_bytes = 0, d2h_bytes = 0;
  u64 peak_states = 1;
  std::vector<RowAcc> rows;
  RunStats rs;
  Plan plan{};
  unsigned slice_depth = 0;
  double elapsed = 0;
};

static Plan make_plan(Ctx& ctx, unsigned n, const qpeps_options& o, unsigned free_rows) {
  Plan p;
  p.n = n;
  p.grain = o.granularity == QPEPS_GRAIN_SITE ? QPEPS_GRAIN_SITE : QPEPS_GRAIN_ROW;
  p.free_rows = free_rows;
  p.R = o.residues ? (int)o.residues : crt_plan(free_rows);
  if (p.R < 1 || p.R > kMaxResidues) fail(QPEPS_ERR_INVALID, "residue count must be in 1..=4");
  if (o.residues && p.R < crt_plan(free_rows))
    fail(QPEPS_ERR_RANGE, "forced residue count does not certify N! for this N");
  // Row keys fit a u64 up to N = 22 (the compact layout at 22); the per-site
  // form's mid-row key carries one more bit, the row signal at bit 3N.
  const unsigned narrow_max = p.grain == QPEPS_GRAIN_SITE ? 20 : kU64MaxN;
  if (o.key_bits == 0)
    p.key_bits = n <= narrow_max ? 64 : 128;
  else if (o.key_bits == 64 || o.key_bits == 128)
    p.key_bits = (int)o.key_bits;
  else
    fail(QPEPS_ERR_INVALID, "key_bits must be 0, 64 or 128");
  if (p.key_bits == 64 && n > narrow_max) fail(QPEPS_ERR_RANGE, "packed boundary does not fit a u64 key for this N");
  p.budget = o.device_budget_bytes ? Budget((size_t)o.device_budget_bytes) : Budget(ctx);
  p.threads = o.block_threads ? (int)o.block_threads : 256;
  const bool partition_ok = (p.key_bits == 64 || p.key_bits == 128) && p.grain == QPEPS_GRAIN_ROW;
  if (o.merge == QPEPS_MERGE_PARTITION && !partition_ok)
    fail(QPEPS_ERR_INVALID, "the partitioned merge needs row granularity");
  if (o.merge == QPEPS_MERGE_HASH)
    p.merge = QPEPS_MERGE_HASH;
  else if (o.merge == QPEPS_MERGE_PARTITION)
    p.merge = partition_ok ? QPEPS_MERGE_PARTITION : QPEPS_MERGE_HASH;
  else if (o.merge == QPEPS_MERGE_AUTO)
    p.merge = (partition_ok && ctx.tune.merge_auto == QPEPS_MERGE_PARTITION) ? QPEPS_MERGE_PARTITION : QPEPS_MERGE_HASH;
  else
    fail(QPEPS_ERR_INVALID, "unknown merge strategy");
  // The slice tail needs u64 keys and the compiled row operator.
  const bool tail_ok = p.key_bits == 64 && p.grain == QPEPS_GRAIN_ROW && n >= 2 && n <= kRefU64MaxN;
  if (o.tail_row == 0)
    p.tail_row = n;  // auto: the merged row engine for every row (fastest measured through N=18)
  else
    p.tail_row = (tail_ok && o.tail_row < n) ? o.tail_row : n;
  // Exact 64-bit weights (only the partitioned row merge reads the planes):
  // two u32 planes carry each weight's words and the host derives the Rc
  // residues of the CRT bookkeeping from exact sums. Every row is certified
  // before it runs from the exact total of its input (run_chunks); with at
  // most 20 free rows that holds by 20! < 2^63; with 21 or 22 it is checked
  // (a row's total is at most its partial placements, for Q(22) far below
  // 2^63 / 22).
  p.Rc = p.R;
  if (ctx.tune.fold_weights == 2 && ctx.tune.merge_kind == 1 && p.R >= 2 && p.free_rows <= 22 &&
      p.merge == QPEPS_MERGE_PARTITION && p.grain == QPEPS_GRAIN_ROW && p.key_bits == 64 && p.tail_row >= n) {
    p.w64 = true;
    p.R = 2;
  }
  return p;
}

// Contract rows from a list of seed items at depth row0 (rows already applied).
static void contract_items(Ctx& ctx, Contraction& out, const std::vector<Item>& items, unsigned row0) {
  const Plan& p = out.plan;
  if (items.empty()) return;
  if (row0 >= p.n) {
    // Fully placed boards.
    const u64 mask = (p.n >= 64) ? ~0ull : ((1ull << p.n) - 1);
    for (const Item& it : items)
      if (((u64)it.key & mask) == mask)
        for (int r = 0; r < p.Rc; ++r)
          out.rs.final_res[r] = (out.rs.final_res[r] + (u64)(it.weight % kPrimes[r])) % kPrimes[r];
    return;
  }
  std::vector<HostChunk> pending;
  pending.push_back(chunk_from_items(p, items, row0));
  run_chunks(ctx, p, std::move(pending), out.rows, out.rs);
}

// Measured peak merged frontier (orbit path) per N (N=19: measured with
// slicing; N >= 20: extrapolated by the x6.3 per-N growth of N=13..19).
static double serve_peak_states(unsigned n) {
  static const double peaks[20] = {1,        1,        2,        3,        6,         10,        21,
                                   46,       130,      371,      4510,     22253,     98939,     541745,
                                   2847130,  18178233, 105530452, 705792694, 4275565705.0, 2.7e10};
  if (n < 20) return peaks[n];
  double e = peaks[19];
  for (unsigned i = 19; i < n; ++i) e *= 6.3;
  return e;
}

// Estimated peak frontier of a request with k placed rows: each placed row
// divides the orbit path's frontier by roughly the number of choices it made.
static double serve_estimate(unsigned n, unsigned k) {
  double e = serve_peak_states(n);
  if (k >= 1) e *= 2.0 / std::max(1u, n);
  for (unsigned i = 1; i < k; ++i) e /= std::max(1.0, (double)n - 3.0);
  return std::max(e, 1.0);
}

static void contract_impl(Ctx& ctx, unsigned n, const qpeps_options& o, const uint32_t* prefix, unsigned k,
                          Contraction& out);

// ---- Explicit-C generic site frontier (src/lib.rs:940-967, 1419-1711) ------
//
// Each site has eight legs (column, row, down-right and down-left diagonal,
// in and out). A leg is a virtual bond shared with the neighbouring site, or
// an open board-edge leg with its allowed values: incoming legs carry 0,
// outgoing column and row legs must carry 1 (one queen per column and row),
// outgoing diagonals are free. Bond ids follow the reference's numbering
// (row bonds, column bonds, down-right, down-left), so the sorted open-bond
// list and with it every key bit position and the counters match its run.

struct FrontierLegH {
  bool bond;
  unsigned id;
  uint8_t allowed;  // open leg: bit v set = value v allowed
};

struct FrontierSiteH {
  unsigned row, column;
  FrontierLegH legs[8];  // column in/out, row in/out, dr in/out, dl in/out
};

static std::vector<FrontierSiteH> frontier_sites(unsigned n) {
  const unsigned span = n - 1, col0 = n * span, dr0 = col0 + n * span, dl0 = dr0 + span * span;
  auto b = [](unsigned id) { return FrontierLegH{true, id, 0}; };
  auto e = [](uint8_t allowed) { return FrontierLegH{false, 0, allowed}; };
  std::vector<FrontierSiteH> out;
  for (unsigned r = 0; r < n; ++r)
    for (unsigned c = 0; c < n; ++c) {
      FrontierSiteH st{r, c, {}};
      const bool top = r == 0, bottom = r + 1 == n, left = c == 0, right = c + 1 == n;
      st.legs[0] = top ? e(1) : b(col0 + (r - 1) * n + c);
      st.legs[1] = bottom ? e(2) : b(col0 + r * n + c);
      st.legs[2] = left ? e(1) : b(r * span + c - 1);
      st.legs[3] = right ? e(2) : b(r * span + c);
      st.legs[4] = (top || left) ? e(1) : b(dr0 + (r - 1) * span + c - 1);
      st.legs[5] = (bottom || right) ? e(3) : b(dr0 + r * span + c);
      st.legs[6] = (top || right) ? e(1) : b(dl0 + (r - 1) * span + c);
      st.legs[7] = (bottom || left) ? e(3) : b(dl0 + r * span + c - 1);
      out.push_back(st);
    }
  return out;
}

struct ExplicitRun {
  unsigned n = 0, order = 0;
  bool complete = false;
  u128 count = 0;
  double elapsed = 0, device_ms = 0;
  u64 peak_states = 1, peak_open_bonds = 0, contracted_sites = 0, launches = 0;
  u128 examined = 0, accepted = 0;
  uint32_t merge = QPEPS_MERGE_PARTITION;
};

// One explicit-C frontier step through the 128-bit partitions, in place:
// count the (entry, matching transition) pairs, size the partitions from
// that count, scatter, merge. Returns the count; the merged boundary's
// scalars are left in ctx.h_sc. An overflowing partition makes the merge
// write nothing, so the step is retried with smaller partitions.
// `known_terms`: the step's match count when the previous step's merge
// counted it (kTermsUnknown otherwise); on return, this step's merge count of
// the next step's matches, if `next_dev` (the next step on the device) was
// given and the merge counted them.
static u64 explicit_partition_step(Ctx& ctx, const Plan& p, DevFrontier& f, const FrontierStepDev& st,
                                   const FrontierStepDev* st_dev, const FrontierStepDev* next_dev, u64& known_terms, ExplicitRun& out) {
  float ms = 0;
  u64 terms = known_terms;
  known_terms = kTermsUnknown;
  if (terms == kTermsUnknown) {
    cuda_check(cudaMemsetAsync(ctx.d_sc, 0, sizeof(StepScalars), ctx.stream), "clear step scalars");
    cuda_check(cudaEventRecord(ctx.ev[0], ctx.stream), "event");
    cuda_check(launch_frontier_count(view_of(p, ctx.front[0], f.cap), f.count, st, ctx.sms, ctx.d_sc, ctx.stream),
               "frontier count kernel");
    cuda_check(cudaEventRecord(ctx.ev[1], ctx.stream), "event");
    out.launches += f.count ? 1 : 0;
    sync_scalars(ctx);
    cudaEventElapsedTime(&ms, ctx.ev[0], ctx.ev[1]);
    out.device_ms += ms;
    terms = ctx.h_sc->terms;
  }
  if (terms == 0) {  // no entries, zero weight: what the caller reads back
    std::memset(ctx.h_sc, 0, sizeof(StepScalars));
    return 0;
  }
  const u32 pcap = wide_key_partition_capacity();
  double mean = ctx.partition_fill * pcap;
  for (int attempt = 0;; ++attempt) {
    const u64 parts64 = std::max<u64>(1, (u64)((double)terms / mean) + 1);
    if (parts64 > 0xffffffffull) fail(QPEPS_ERR_CAPACITY, "explicit-C frontier needs too many partitions");
    const u32 parts = (u32)parts64;
    const u32 cstride = (parts <= ctx.tune.spread_cursors_below) ? 8u : 1u;
    const size_t region_bytes = (size_t)parts * pcap * cand_bytes(p);
    const size_t table_bytes = region_bytes + ((size_t)parts * 4 * cstride + 255) / 256 * 256;
    if (ctx.table.bytes < table_bytes) buf_release(ctx, ctx.table);
    if (!ensure_front(ctx, p, f, std::max<u64>(f.count, terms), ctx.table.ptr ? 0 : table_bytes))
      fail(QPEPS_ERR_CAPACITY, "device budget exceeded by the explicit-C frontier");
    buf_reserve(ctx, ctx.table, table_bytes, p.budget, "explicit-C frontier partitions");
    const FrontierView view = view_of(p, ctx.front[0], f.cap);
    void* regions = ctx.table.ptr;
    u32* cursors = reinterpret_cast<u32*>(static_cast<char*>(ctx.table.ptr) + region_bytes);
    PartitionCfg pc{};
    pc.residues = p.R;
    pc.sms = ctx.sms;
    pc.parts = parts;
    pc.cap = pcap;
    pc.merge_blocks_per_sm = 2;
    pc.cursor_stride = cstride;
    pc.key_bits = 128;
    cuda_check(cudaMemsetAsync(ctx.d_sc, 0, sizeof(StepScalars), ctx.stream), "clear step scalars");
    cuda_check(cudaMemsetAsync(cursors, 0, (size_t)parts * 4 * cstride, ctx.stream), "clear partition cursors");
    cuda_check(cudaEventRecord(ctx.ev[0], ctx.stream), "event");
    cuda_check(launch_frontier_partition_scatter(pc, view, f.count, st_dev, regions, cursors, ctx.d_sc, ctx.stream),
               "frontier scatter kernel");
    cuda_check(launch_wide_partition_merge(pc, regions, cursors, view, 0, true, ctx.d_sc, ctx.stream, next_dev),
               "frontier merge kernel");
    cuda_check(cudaEventRecord(ctx.ev[1], ctx.stream), "event");
    out.launches += 2;
    sync_scalars(ctx);
    cudaEventElapsedTime(&ms, ctx.ev[0], ctx.ev[1]);
    out.device_ms += ms;
    if (ctx.h_sc->error & kErrBounds)
      fail(QPEPS_ERR_CUDA, "explicit-C frontier: a kernel's bounds check failed (access skipped)");
    if (ctx.h_sc->error & kErrOverflow) {
      if (attempt >= 4) fail(QPEPS_ERR_CAPACITY, "explicit-C frontier: partition overflow persists");
      mean *= 0.6;
      continue;
    }
    if (ctx.h_sc->error) fail(QPEPS_ERR_CAPACITY, "explicit-C frontier: device capacity error");
    if (next_dev && ctx.h_sc->next_terms_ok) known_terms = ctx.h_sc->next_terms;
    return terms;
  }
}

// Steps of a chain that may stop at the support limit, at most: the launches
// queued behind the site that passes it return at once, but take 2 us each all
// the same (N = 20 in one chain: 10.5 ms for a limit of one entry). Fewer where
// the boundary is near the limit: a site at most doubles it, and grows it by
// half that in the logarithm on average.
constexpr size_t kLimitedChain = 16;

// Site steps [first, end) of the explicit-C frontier as a chain
// (run_queued_rows above has the idea), fewer where the support limit may stop
// it; `known_terms`: the first step's matches, kTermsUnknown to count them.
// Returns the steps contracted, the one that passes the limit included; their
// scalars are in ctx.h_queue[1 ..], the first step's matches in [0]. Fewer than
// `queued` (the steps the chain had): the next one did not fit its buffers.
static size_t run_queued_sites(Ctx& ctx, const Plan& p, DevFrontier& f, const std::vector<FrontierStepDev>& steps,
                               const FrontierStepDev* d_steps, const std::vector<size_t>& open_after, size_t first,
                               size_t end, u64 support_limit, u64 known_terms, ExplicitRun& out, size_t& queued) {
  // Largest boundaries: 1.3 M entries at N = 12 (diamond), times about 5.8 per
  // size; at most two matches an entry, of which at most `support_limit` stand.
  const double states = 1.4e6 * std::pow(5.8, (double)p.n - 12.0);
  const double limit = (double)support_limit;
  const u64 most = (u64)std::min({(double)kQueueTerms, std::max(65536.0, 1.8 * states), 2.0 * limit + 1024.0});
  size_t count = end - first;
  if (limit < 2.0 * states) {
    const double doublings = std::log2(limit / (double)std::max<u64>(f.count, 1));
    count = std::min({count, kLimitedChain, (size_t)(2.0 + 2.0 * doublings)});
  }
  queued = count;
  const u32 pcap = wide_key_partition_capacity();
  const double mean = chain_mean(ctx, pcap);
  StepSource source{nullptr, mean, 0, 2 * (u32)ctx.sms, support_limit};
  const u32 parts_cap = source.parts_cap = (u32)source.partitions(most);
  const u32 cstride = (parts_cap <= ctx.tune.spread_cursors_below) ? 8u : 1u;
  const size_t region_bytes = (size_t)parts_cap * pcap * cand_bytes(p);
  const size_t cursor_bytes = (size_t)parts_cap * 4 * cstride;
  const size_t table_bytes = region_bytes + (cursor_bytes + 255) / 256 * 256;
  if (count < 2 || f.count > most || !chain_buffers(ctx, p, f, most, table_bytes, count, "partition regions")) return 0;
  StepScalars* d = queue_scalars(ctx, count);
  StepScalars* h = ctx.h_queue;
  h[0].out_count = f.count;
  if (known_terms != kTermsUnknown) h[0].next_terms = known_terms;
  void* regions = ctx.table.ptr;
  u32* cursors = reinterpret_cast<u32*>(static_cast<char*>(ctx.table.ptr) + region_bytes);
  const FrontierView view = view_of(p, ctx.front[0], f.cap);
  PartitionCfg pc{};
  pc.residues = p.R;
  pc.sms = ctx.sms;
  pc.cap = pcap;
  pc.merge_blocks_per_sm = 2;
  pc.cursor_stride = cstride;
  pc.key_bits = 128;
  cuda_check(cudaMemcpyAsync(d, h, (count + 1) * sizeof(StepScalars), cudaMemcpyHostToDevice, ctx.stream),
             "queued step scalars");
  cuda_check(cudaMemsetAsync(cursors, 0, cursor_bytes, ctx.stream), "clear partition cursors");
  cuda_check(cudaEventRecord(ctx.ev[0], ctx.stream), "event");
  if (known_terms == kTermsUnknown) {
    cuda_check(launch_frontier_count(view, f.count, steps[first], ctx.sms, d, ctx.stream), "frontier count kernel");
    out.launches += 1;
  }
  u64 entries = f.count;
  for (size_t i = 0; i < count; ++i) {
    const u64 fits = std::min(most, 2 * entries);  // at most two matches an entry
    pc.queued = source;
    pc.queued.prev = d + i;
    pc.parts = (u32)source.partitions(fits);
    // The merge counts the next step's matches, for the chain or the step that
    // follows it.
    const size_t after = first + i + 1;
    const bool next = after < steps.size() && open_after[after] < 128;
    cuda_check(launch_frontier_partition_scatter(pc, view, entries, d_steps + first + i, regions, cursors, d + i + 1,
                                                 ctx.stream),
               "frontier scatter kernel");
    cuda_check(launch_wide_partition_merge(pc, regions, cursors, view, 0, true, d + i + 1, ctx.stream,
                                           next ? d_steps + after : nullptr),
               "frontier merge kernel");
    entries = fits;
  }
  cuda_check(cudaEventRecord(ctx.ev[1], ctx.stream), "event");
  cuda_check(cudaMemcpyAsync(h, d, (count + 1) * sizeof(StepScalars), cudaMemcpyDeviceToHost, ctx.stream),
             "read step scalars");
  cuda_check(cudaStreamSynchronize(ctx.stream), "queued sites");
  ctx.h2d_bytes += (count + 1) * sizeof(StepScalars);
  ctx.d2h_bytes += (count + 1) * sizeof(StepScalars);
  out.launches += 2 * count;
  float ms = 0;
  cudaEventElapsedTime(&ms, ctx.ev[0], ctx.ev[1]);
  out.device_ms += ms;
  size_t done = 0;
  while (done < count && !h[done + 1].error) ++done;
  if (done < count) chain_ended(ctx, h[done + 1], mean, pcap);
  if (done < count && (h[done + 1].error & kErrBounds))
    fail(QPEPS_ERR_CUDA, "explicit-C frontier: a kernel's bounds check failed (access skipped)");
  return done;
}

static void explicit_frontier(Ctx& ctx, unsigned n, unsigned order, u64 support_limit, ExplicitRun& out) {
  const auto t0 = std::chrono::steady_clock::now();
  if (n > 21) fail(QPEPS_ERR_RANGE, "explicit-C frontier key supports N <= 21");
  if (support_limit == 0) fail(QPEPS_ERR_INVALID, "explicit-C frontier support limit must be positive");
  if (order > 1) fail(QPEPS_ERR_INVALID, "order must be QPEPS_ORDER_ROW_MAJOR or QPEPS_ORDER_TOP_LEFT_DIAMOND");
  out = ExplicitRun{};
  out.n = n;
  out.order = order;
  if (n == 0) {
    out.complete = true;
    out.count = 1;
    return;
  }
  certify_c(ctx.c);
  if (ctx.c.size() != 17) fail(QPEPS_ERR_INVALID, "explicit-C frontier requires the Sec. VI 17-entry tensor");
  cuda_check(cudaSetDevice(ctx.device), "cudaSetDevice");
  const std::vector<FrontierSiteH> sites = frontier_sites(n);
  std::vector<unsigned> ordering((size_t)n * n);
  for (unsigned i = 0; i < ordering.size(); ++i) ordering[i] = i;
  if (order == QPEPS_ORDER_TOP_LEFT_DIAMOND)
    std::stable_sort(ordering.begin(), ordering.end(), [n](unsigned a, unsigned b) {
      const unsigned da = a / n + a % n, db = b / n + b % n;
      return da != db ? da < db : a / n < b / n;
    });

  Plan p{};
  p.n = n;
  p.free_rows = n;
  p.R = crt_plan(n);
  p.Rc = p.R;
  p.key_bits = 128;
  p.grain = QPEPS_GRAIN_SITE;
  p.merge = QPEPS_MERGE_HASH;
  p.budget = Budget(ctx);
  p.threads = 256;
  p.tail_row = n;
  const size_t eb = entry_bytes(p);
  DevFrontier f;
  buf_release(ctx, ctx.front[1]);
  f.cap = ctx.front[0].ptr ? ctx.front[0].bytes / eb : 0;
  if (!ensure_front(ctx, p, f, 1024, 0)) fail(QPEPS_ERR_CAPACITY, "device budget cannot hold the seed boundary");
  {
    // Seed: the empty boundary (key 0) with weight 1.
    char* base = static_cast<char*>(ctx.front[0].ptr);
    cuda_check(cudaMemsetAsync(base, 0, 16, ctx.stream), "seed key");
    const uint32_t one = 1;
    for (int r = 0; r < p.R; ++r)
      cuda_check(cudaMemcpyAsync(base + f.cap * 16 + (size_t)r * f.cap * 4, &one, 4, cudaMemcpyHostToDevice,
                                 ctx.stream),
                 "seed weight");
    cuda_check(cudaStreamSynchronize(ctx.stream), "seed");
    ctx.h2d_bytes += 4u * p.R;
    f.count = 1;
  }
  LaunchCfg cfg{128, p.R, 256, ctx.sms};
  // Pass 1 (host only): every site step's transitions and open-bond count, so
  // that each step's merge can count the next step's matches on the device.
  // An error found here is raised when the contraction reaches its step.
  const size_t total = ordering.size();
  std::vector<FrontierStepDev> steps(total);
  std::vector<size_t> open_after(total, 0);
  size_t fail_step = total;
  int fail_code = QPEPS_OK;
  std::string fail_msg;
  std::vector<unsigned> open;
  for (size_t step = 0; step < total && fail_step == total; ++step) {
    const FrontierSiteH& site = sites[ordering[step]];
    auto pos_in = [](const std::vector<unsigned>& v, unsigned id) -> int {
      auto it = std::lower_bound(v.begin(), v.end(), id);
      return (it != v.end() && *it == id) ? (int)(it - v.begin()) : -1;
    };
    std::vector<unsigned> incident;
    for (const FrontierLegH& l : site.legs)
      if (l.bond) incident.push_back(l.id);
    std::vector<unsigned> next;
    for (unsigned id : open)
      if (std::find(incident.begin(), incident.end(), id) == incident.end()) next.push_back(id);
    for (unsigned id : incident)
      if (pos_in(open, id) < 0) next.push_back(id);
    std::sort(next.begin(), next.end());
    if (next.size() > 128) {
      char buf[96];
      std::snprintf(buf, sizeof buf, "explicit-C frontier exceeds 128 open bonds at site (%u,%u)", site.row,
                    site.column);
      fail_step = step;
      fail_code = QPEPS_ERR_RANGE;
      fail_msg = buf;
      break;
    }
    // Bonds that stay open keep their order: group them into runs that move
    // by one shift each.
    FrontierStepDev st;
    std::memset(&st, 0, sizeof st);
    int prev_old = -2, prev_new = -2;
    for (unsigned i = 0; i < open.size(); ++i) {
      const int j = pos_in(next, open[i]);
      if (j < 0) continue;
      if ((int)i == prev_old + 1 && j == prev_new + 1 && st.n_runs > 0) {
        st.run_mask[st.n_runs - 1] |= (u128)1 << i;
      } else {
        if (st.n_runs == (uint32_t)kFrontierMaxRuns) {
          fail_step = step;
          fail_code = QPEPS_ERR_CAPACITY;
          fail_msg = "explicit-C frontier: too many bond runs";
          break;
        }
        st.run_mask[st.n_runs] = (u128)1 << i;
        st.run_shift[st.n_runs] = j - (int)i;
        ++st.n_runs;
      }
      prev_old = (int)i;
      prev_new = j;
    }
    for (const CEntryH& e : ctx.c) {
      const Legs lg = legs_from_key(e.legs);
      const uint8_t values[8] = {lg.ci, lg.co, lg.ri, lg.ro, lg.dri, lg.dro, lg.dli, lg.dlo};
      u128 req_mask = 0, req_value = 0, added = 0;
      bool keep = true;
      for (int l = 0; l < 8 && keep; ++l) {
        const FrontierLegH& leg = site.legs[l];
        if (!leg.bond) {
          keep = (leg.allowed >> values[l]) & 1;
        } else if (const int i = pos_in(open, leg.id); i >= 0) {
          req_mask |= (u128)1 << i;
          req_value |= (u128)values[l] << i;
        } else {
          added |= (u128)values[l] << pos_in(next, leg.id);
        }
      }
      if (!keep) continue;
      st.req_mask[st.n_trans] = req_mask;
      st.req_value[st.n_trans] = req_value;
      st.added[st.n_trans] = added;
      ++st.n_trans;
    }
    if (fail_step < total) break;
    steps[step] = st;
    open_after[step] = next.size();
    open.swap(next);
  }
  const bool ends_closed = open.empty();
  // The partitioned merge unless the tuning asks for the global table, or a
  // key could set all 128 bits (the partition tables' empty marker).
  const bool partitioned = ctx.tune.merge_auto != QPEPS_MERGE_HASH;
  out.merge = partitioned ? QPEPS_MERGE_PARTITION : QPEPS_MERGE_HASH;
  FrontierStepDev* d_steps = nullptr;
  if (partitioned) {
    buf_reserve(ctx, ctx.plan, total * sizeof(FrontierStepDev), p.budget, "explicit-C frontier steps");
    d_steps = static_cast<FrontierStepDev*>(ctx.plan.ptr);
    cuda_check(cudaMemcpyAsync(d_steps, steps.data(), total * sizeof(FrontierStepDev), cudaMemcpyHostToDevice,
                               ctx.stream),
               "frontier steps");
    ctx.h2d_bytes += total * sizeof(FrontierStepDev);
  }
  // Pass 2: the device steps.
  u64 weight_res[kMaxResidues] = {0, 0, 0, 0};
  u64 known_terms = kTermsUnknown;
  auto merged_step = [&](size_t step, const StepScalars& sc) {  // false: the support limit stops here
    const u64 merged = sc.out_count;
    out.peak_open_bonds = std::max<u64>(out.peak_open_bonds, open_after[step]);
    if (merged > support_limit) {
      out.peak_states = std::max<u64>(out.peak_states, support_limit + 1);
      out.contracted_sites = step;
      out.elapsed = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
      return false;
    }
    f.count = merged;
    for (int r = 0; r < p.R; ++r) weight_res[r] = sc.weight_sum[r] % kPrimes[r];
    out.peak_states = std::max<u64>(out.peak_states, merged);
    return true;
  };
  // Leading steps that can be queued run as chains, until one does not fit.
  size_t chainable = 0, step = 0;
  if (partitioned && d_steps)
    while (chainable < total && chainable != fail_step && open_after[chainable] < 128) ++chainable;
  for (size_t queued = 0, done = 0; step < chainable && done == queued;) {
    done = run_queued_sites(ctx, p, f, steps, d_steps, open_after, step, chainable, support_limit, known_terms, out,
                            queued);
    for (size_t i = 0; i < done; ++i, ++step) {
      const StepScalars& sc = ctx.h_queue[i + 1];
      out.examined += (u128)f.count * 17;
      out.accepted += ctx.h_queue[i].next_terms;
      if (!merged_step(step, sc)) return;
      known_terms = sc.next_terms_ok ? sc.next_terms : kTermsUnknown;
    }
  }
  for (; step < total; ++step) {
    if (step == fail_step) fail(fail_code, fail_msg);
    const FrontierStepDev& st = steps[step];
    const size_t next_open = open_after[step];
    out.examined += (u128)f.count * 17;
    if (partitioned && next_open < 128) {
      const bool next_partitioned = step + 1 < total && step + 1 != fail_step && open_after[step + 1] < 128;
      const FrontierStepDev* next_dev = next_partitioned ? d_steps + step + 1 : nullptr;
      const u64 terms = explicit_partition_step(ctx, p, f, st, d_steps + step, next_dev, known_terms, out);
      out.accepted += terms;
      if (!merged_step(step, *ctx.h_sc)) return;
      continue;
    }
    known_terms = kTermsUnknown;
    // Every incoming leg of a site is a bond of an earlier site or a board
    // edge in both orders, so at most two C entries match a key.
    const u64 need = std::max<u64>(f.count * 2, 1);
    const u64 slots = pow2_at_least(std::max<u64>(1024, need * 2));
    const size_t table_bytes = slots * slot_bytes(128, p.R);
    if (ctx.table.bytes < table_bytes) buf_release(ctx, ctx.table);
    if (!ensure_front(ctx, p, f, need, ctx.table.ptr ? 0 : table_bytes))
      fail(QPEPS_ERR_CAPACITY, "device budget exceeded by the explicit-C frontier");
    buf_reserve(ctx, ctx.table, table_bytes, p.budget, "explicit-C frontier table");
    FrontierView view = view_of(p, ctx.front[0], f.cap);
    cuda_check(upload_frontier_step(st, ctx.stream), "frontier step");
    cuda_check(cudaMemsetAsync(ctx.d_sc, 0, sizeof(StepScalars), ctx.stream), "clear step scalars");
    cuda_check(cudaMemsetAsync(ctx.table.ptr, 0, table_bytes, ctx.stream), "clear table");
    cuda_check(cudaEventRecord(ctx.ev[0], ctx.stream), "event");
    cuda_check(launch_frontier_expand_insert(cfg, view, f.count, ctx.table.ptr, slots, ctx.d_sc, ctx.stream),
               "frontier expand-insert kernel");
    cuda_check(launch_compact(cfg, ctx.table.ptr, slots, view, 0, true, ctx.d_sc, ctx.stream), "compact kernel");
    cuda_check(cudaEventRecord(ctx.ev[1], ctx.stream), "event");
    out.launches += 2;
    sync_scalars(ctx);
    if (ctx.h_sc->error) fail(QPEPS_ERR_CAPACITY, "explicit-C frontier table probe bound exceeded");
    float ms = 0;
    cudaEventElapsedTime(&ms, ctx.ev[0], ctx.ev[1]);
    out.device_ms += ms;
    out.accepted += ctx.h_sc->terms;
    if (!merged_step(step, *ctx.h_sc)) return;
  }
  if (!ends_closed) fail(QPEPS_ERR_INVALID, "explicit-C contraction ended with uncontracted virtual bonds");
  // No bond is open: the boundary is the single key 0 (or empty) and its
  // weight is the count.
  if (f.count > 1) fail(QPEPS_ERR_INVALID, "explicit-C contraction ended with more than one closed boundary");
  out.count = f.count ? crt_reconstruct(weight_res, p.R) : 0;
  if (out.count > factorial(n)) fail(QPEPS_ERR_CRT_BOUND, "CRT reconstruction exceeds certified N! count bound");
  out.complete = true;
  out.contracted_sites = (u64)n * n;
  out.elapsed = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
}

// ---- CUDA-graph replay (qpeps_options.use_graph) ---------------------------
//
// A contraction's device work is fixed by N, the prefix, the options and the
// tuning: the same seeds, the same per-row successor counts and the same
// partition sizes every time. With use_graph, an eager run records its row
// steps (GraphRecorder); if it ran as whole device batches with the
// partitioned merge (no host spill, no tail kernel), the steps are captured
// once into a graph: per batch a copy of the batch's seed from pinned host
// memory, then per row the cursor clear, the scatter and the merge, each row's
// scalars into its own slot, and one copy of all scalars to pinned memory at
// the end. A later identical contraction on the same context, while the
// context's buffers are unchanged, replays it: one graph launch and one
// synchronisation instead of three launches and two synchronisations per row.
// The replay checks every row's output count, weight sums and final sums
// against the recorded run before it answers; on any difference it drops the
// graph and contracts eagerly. Column-grouped and one-CTA rows are queued
// without the host already and are not captured: each run is compared with the
// recorded one in the same figures.

// Device batches are independent sub-contractions (their results add), so
// the graph runs them on `batch_lanes` streams at once: each lane has its own
// boundary, partition regions and plan scratch (lane 0 borrows the context's)
// and takes whole batches, balanced by their recorded successor counts; the
// kernels of different lanes overlap on the device. The start event, the
// lanes' fork and join and the read-back of all scalars stay on the context's
// stream.
struct GraphLane {
  cudaStream_t stream = nullptr;  // lane 0: the context's stream
  DevBuf front, table, plan;      // owned by lanes >= 1
  u64 cap = 0;                    // boundary capacity (entries)
  cudaEvent_t join = nullptr;
  std::vector<size_t> chunks;     // indices into GraphPlan::chunks, in launch order
};

struct GraphPlan {
  unsigned n = 0;
  std::vector<uint32_t> prefix;
  qpeps_options opt{};
  Ctx::Tune tune{};
  uint64_t pool_gen = 0;
  Contraction base;
  std::vector<GraphChunkRec> chunks;
  std::vector<size_t> step_base;  // first scalars slot of each chunk
  cudaGraphExec_t exec = nullptr;
  void* h_seeds = nullptr;  // pinned: every batch's seed keys and residue planes, packed
  std::vector<size_t> seed_off;
  size_t seed_bytes = 0;
  StepScalars* d_scal = nullptr;
  StepScalars* h_scal = nullptr;
  size_t nsteps = 0;
  uint64_t launches = 0;
  size_t lane_bytes = 0;          // device memory held by lanes >= 1
  std::vector<GraphLane> lanes;
  cudaEvent_t fork = nullptr;
  std::vector<cudaEvent_t> ev;    // three per step with work: start, after the scatter, after the merge
};

static void graph_free(Ctx& ctx) {
  GraphPlan* g = ctx.graph;
  if (!g) return;
  if (g->exec) cudaGraphExecDestroy(g->exec);
  if (g->h_seeds) cudaFreeHost(g->h_seeds);
  if (g->d_scal) cudaFree(g->d_scal);
  if (g->h_scal) cudaFreeHost(g->h_scal);
  for (cudaEvent_t e : g->ev)
    if (e) cudaEventDestroy(e);
  if (g->fork) cudaEventDestroy(g->fork);
  for (size_t l = 0; l < g->lanes.size(); ++l) {
    GraphLane& L = g->lanes[l];
    if (L.join) cudaEventDestroy(L.join);
    if (l == 0) continue;
    for (DevBuf* b : {&L.front, &L.table, &L.plan})
      if (b->ptr) cudaFree(b->ptr);
    if (L.stream) cudaStreamDestroy(L.stream);
  }
  delete g;
  ctx.graph = nullptr;
}

static qpeps_options graph_key_options(const qpeps_options& o) {
  qpeps_options k = o;
  k.use_graph = 0;
  k.reserved = 0;
  return k;
}

// Whether the context's record is of this call.
static bool same_call(const Ctx& ctx, unsigned n, const qpeps_options& o, const uint32_t* prefix, unsigned k) {
  const GraphPlan* g = ctx.graph;
  if (!g || g->n != n || g->prefix.size() != k) return false;
  for (unsigned i = 0; i < k; ++i)
    if (g->prefix[i] != prefix[i]) return false;
  const qpeps_options a = graph_key_options(o), b = graph_key_options(g->opt);
  if (std::memcmp(&a, &b, sizeof a) != 0) return false;
  return std::memcmp(&g->tune, &ctx.tune, sizeof g->tune) == 0;
}

// Whether a captured graph of this call can replay in the buffers as they stand.
static bool graph_matches(const Ctx& ctx, unsigned n, const qpeps_options& o, const uint32_t* prefix, unsigned k) {
  return same_call(ctx, n, o, prefix, k) && ctx.graph->exec && ctx.graph->pool_gen == ctx.pool_gen;
}

// A run that is not captured, as the record that the next one is compared with.
static void record_rows(Ctx& ctx, unsigned n, const qpeps_options& o, const uint32_t* prefix, unsigned k,
                        const Contraction& done) {
  graph_free(ctx);
  GraphPlan* g = ctx.graph = new GraphPlan();
  g->n = n;
  g->prefix.assign(prefix, prefix + k);
  g->opt = o;
  g->tune = ctx.tune;
  g->base = done;
}

// The figures that a replay checks, of two whole runs.
static bool same_rows(const Contraction& a, const Contraction& b) {
  bool same = a.count == b.count && a.rows.size() == b.rows.size();
  for (size_t i = 0; same && i < a.rows.size(); ++i) {
    const RowAcc &x = a.rows[i], &y = b.rows[i];
    same = x.input_states == y.input_states && x.output_states == y.output_states && x.matched == y.matched;
    for (int r = 0; r < kMaxResidues; ++r) same = same && x.weight_res[r] == y.weight_res[r];
  }
  return same;
}

// Capture the recorded steps. Best effort: any failure leaves no graph.
static void graph_build(Ctx& ctx, unsigned n, const qpeps_options& o, const uint32_t* prefix, unsigned k,
                        const Contraction& done, GraphRecorder& rec) {
  graph_free(ctx);
  const Plan& p = done.plan;
  if (!rec.ok || rec.chunks.empty() || p.merge != QPEPS_MERGE_PARTITION || p.grain != QPEPS_GRAIN_ROW ||
      !ctx.front[0].ptr || !ctx.table.ptr)
    return;
  const size_t eb = entry_bytes(p), kb = key_bytes(p);
  const u64 cap0 = ctx.front[0].bytes / eb;
  size_t seed_bytes = 0, nsteps = 0;
  // Per chunk: boundary capacity, region and plan bytes it needs, and its work.
  const size_t nc = rec.chunks.size();
  std::vector<u64> need_cap(nc, 0), work(nc, 0);
  std::vector<size_t> need_table(nc, 0), need_plan(nc, 0);
  for (size_t i = 0; i < nc; ++i) {
    const GraphChunkRec& c = rec.chunks[i];
    need_cap[i] = std::max<u64>(c.count, 1);
    seed_bytes += c.count * eb;
    for (const GraphStepRec& st : c.steps) {
      ++nsteps;
      if (!st.terms) continue;
      need_cap[i] = std::max(need_cap[i], st.need_cap);
      need_table[i] = std::max(need_table[i], st.table_bytes);
      if (st.unit) need_plan[i] = std::max(need_plan[i], unit_plan_scratch_bytes(st.upa.lg));
      work[i] += st.terms;
    }
    if (need_cap[i] > cap0 || need_table[i] > ctx.table.bytes || (need_plan[i] && need_plan[i] > ctx.plan.bytes))
      return;  // lane 0 runs in the context's buffers
  }
  // Lanes: whole batches, heaviest first to the least loaded lane; a lane
  // beyond the first is kept only while the device budget holds its buffers.
  // Several lanes are used only with the window and direct scatters, the
  // combinations run and checked at Q(18) on GB300. (An autotuning run that
  // replayed Q(18) on two lanes stopped on an illegal address; the likely
  // cause is the class-grouped replay described below, which wrote through
  // partition indices beyond its regions before the bounds check existed.)
  bool lanes_ok = true;
  for (const GraphChunkRec& c : rec.chunks)
    for (const GraphStepRec& st : c.steps)
      if (st.terms && st.pc.scatter_kind != 1 && st.pc.scatter_kind != 4) lanes_ok = false;
  // Class-grouped partitions are not captured: in one replay of Q(17) the plan
  // rebuilt on the device at a later row named more partitions than the
  // recorded run had (caught by the class scatter's bounds check, the access
  // skipped), so an earlier replayed row had left a different boundary; the
  // cause is not found. Those contractions run eagerly, where every row's
  // plan is read back before its scatter.
  for (const GraphChunkRec& c : rec.chunks)
    for (const GraphStepRec& st : c.steps)
      if (st.terms && st.unit) return;
  unsigned nl = lanes_ok ? (unsigned)std::max<u64>(1, std::min<u64>(ctx.tune.batch_lanes, nc)) : 1u;
  std::vector<size_t> order(nc);
  for (size_t i = 0; i < nc; ++i) order[i] = i;
  std::stable_sort(order.begin(), order.end(), [&](size_t a, size_t b) { return work[a] > work[b]; });
  std::vector<std::vector<size_t>> assign;
  std::vector<size_t> lane_bytes;
  for (;; --nl) {
    assign.assign(nl, {});
    std::vector<u64> load(nl, 0);
    for (size_t i : order) {
      const size_t l = (size_t)(std::min_element(load.begin(), load.end()) - load.begin());
      assign[l].push_back(i);
      load[l] += work[i] + 1;
    }
    lane_bytes.assign(nl, 0);
    size_t extra = 0;
    for (unsigned l = 1; l < nl; ++l) {
      u64 cap = 1;
      size_t tb = 0, pb = 0;
      for (size_t i : assign[l]) {
        cap = std::max(cap, need_cap[i]);
        tb = std::max(tb, need_table[i]);
        pb = std::max(pb, need_plan[i]);
      }
      lane_bytes[l] = cap * eb + tb + pb;
      extra += lane_bytes[l];
    }
    if (nl == 1 || ctx.pool_bytes + extra <= p.budget) break;
  }
  for (auto& a : assign) std::sort(a.begin(), a.end());  // recorded order within a lane
  GraphPlan* g = new GraphPlan();
  ctx.graph = g;
  g->n = n;
  g->prefix.assign(prefix, prefix + k);
  g->opt = o;
  g->tune = ctx.tune;
  g->base = done;
  g->chunks = std::move(rec.chunks);
  g->nsteps = nsteps;
  bool capturing = false;
  cudaGraph_t graph = nullptr;
  auto ok = [&](cudaError_t e) {
    if (e != cudaSuccess) throw Failure{QPEPS_ERR_CUDA, cudaGetErrorString(e)};
  };
  try {
    g->lanes.resize(nl);
    for (unsigned l = 0; l < nl; ++l) {
      GraphLane& L = g->lanes[l];
      L.chunks = assign[l];
      ok(cudaEventCreateWithFlags(&L.join, cudaEventDisableTiming));
      if (l == 0) {
        L.stream = ctx.stream;
        L.front = ctx.front[0];
        L.table = ctx.table;
        L.plan = ctx.plan;
        L.cap = cap0;
        continue;
      }
      ok(cudaStreamCreateWithFlags(&L.stream, cudaStreamNonBlocking));
      u64 cap = 1;
      size_t tb = 0, pb = 0;
      for (size_t i : L.chunks) {
        cap = std::max(cap, need_cap[i]);
        tb = std::max(tb, need_table[i]);
        pb = std::max(pb, need_plan[i]);
      }
      L.cap = cap;
      ok(cudaMalloc(&L.front.ptr, cap * eb));
      L.front.bytes = cap * eb;
      ok(cudaMalloc(&L.table.ptr, std::max<size_t>(tb, 256)));
      L.table.bytes = std::max<size_t>(tb, 256);
      if (pb) {
        ok(cudaMalloc(&L.plan.ptr, pb));
        L.plan.bytes = pb;
      }
      g->lane_bytes += L.front.bytes + L.table.bytes + L.plan.bytes;
    }
    ok(cudaEventCreateWithFlags(&g->fork, cudaEventDisableTiming));
    ok(cudaMallocHost(&g->h_seeds, std::max<size_t>(seed_bytes, 16)));
    g->seed_bytes = seed_bytes;
    ok(cudaMalloc(&g->d_scal, std::max<size_t>(nsteps, 1) * sizeof(StepScalars)));
    ok(cudaMallocHost(&g->h_scal, std::max<size_t>(nsteps, 1) * sizeof(StepScalars)));
    // Seeds: each batch's keys then its residue planes, packed in pinned
    // memory; every replay uploads them again (the graph's copy nodes).
    size_t off = 0, si = 0, nev = 0;
    g->seed_off.resize(g->chunks.size());
    g->step_base.resize(g->chunks.size());
    for (size_t i = 0; i < g->chunks.size(); ++i) {
      const GraphChunkRec& c = g->chunks[i];
      g->seed_off[i] = off;
      g->step_base[i] = si;
      std::memcpy(static_cast<char*>(g->h_seeds) + off, c.keys.data(), c.count * kb);
      std::memcpy(static_cast<char*>(g->h_seeds) + off + c.count * kb, c.res.data(), c.count * 4u * p.R);
      off += c.count * eb;
      si += c.steps.size();
      for (const GraphStepRec& st : c.steps) nev += st.terms ? 3 : 0;
    }
    g->ev.assign(nev, nullptr);
    for (cudaEvent_t& e : g->ev) ok(cudaEventCreate(&e));
    // Events of step j of chunk i: 3 * (rank of the step among steps with work).
    std::vector<size_t> ev_base(g->chunks.size());
    size_t ecount = 0;
    for (size_t i = 0; i < g->chunks.size(); ++i) {
      ev_base[i] = ecount;
      for (const GraphStepRec& st : g->chunks[i].steps) ecount += st.terms ? 3 : 0;
    }

    ok(cudaStreamBeginCapture(ctx.stream, cudaStreamCaptureModeRelaxed));
    capturing = true;
    ok(cudaMemsetAsync(g->d_scal, 0, std::max<size_t>(nsteps, 1) * sizeof(StepScalars), ctx.stream));
    ok(cudaEventRecord(g->fork, ctx.stream));
    for (unsigned l = 1; l < nl; ++l) ok(cudaStreamWaitEvent(g->lanes[l].stream, g->fork, 0));
    for (GraphLane& L : g->lanes) {
      cudaStream_t st_ = L.stream;
      char* front = static_cast<char*>(L.front.ptr);
      DevBuf lane_front = L.front;
      const FrontierView view = view_of(p, lane_front, L.cap);
      for (size_t i : L.chunks) {
        const GraphChunkRec& c = g->chunks[i];
        const char* sd = static_cast<const char*>(g->h_seeds) + g->seed_off[i];
        size_t ei = ev_base[i];
        size_t sj = g->step_base[i];
        bool first = true;
        for (const GraphStepRec& st : c.steps) {
          StepScalars* sc = g->d_scal + sj++;
          if (!st.terms) continue;
          ok(cudaEventRecordWithFlags(g->ev[ei], st_, cudaEventRecordExternal));
          if (first) {
            ok(cudaMemcpyAsync(front, sd, c.count * kb, cudaMemcpyHostToDevice, st_));
            for (int r = 0; r < p.R; ++r)
              ok(cudaMemcpyAsync(front + L.cap * kb + (size_t)r * L.cap * 4,
                                 sd + c.count * kb + (size_t)r * c.count * 4, c.count * 4, cudaMemcpyHostToDevice,
                                 st_));
            first = false;
          }
          void* regions = L.table.ptr;
          uint32_t* cursors = reinterpret_cast<uint32_t*>(static_cast<char*>(L.table.ptr) + st.region_bytes);
          ok(cudaMemsetAsync(cursors, 0, (size_t)st.pc.parts * 4 * st.pc.cursor_stride, st_));
          if (st.unit) {
            // The plan is a function of the boundary's keys only: the replay
            // rebuilds the recorded one.
            UnitPlanDev upd{};
            ok(launch_unit_plan(view, st.n_in, st.ucp, st.upa, L.plan.ptr, ctx.sms, st_, &upd, sc));
            ok(launch_unit_scatter(st.pc, view, st.n_in, st.ucp, upd.table, regions, cursors, sc, st_));
            g->launches += 4;
          } else {
            ok(launch_partition_scatter(st.pc, view, st.n_in, p.n, regions, cursors, sc, st_));
          }
          ok(cudaEventRecordWithFlags(g->ev[ei + 1], st_, cudaEventRecordExternal));
          PartitionCfg mpc = st.pc;
          mpc.count_next = 0;  // a replay's sizes are recorded: no next-row count
          ok(launch_partition_merge(mpc, regions, cursors, view, p.n, !st.final_step, sc, st_));
          ok(cudaEventRecordWithFlags(g->ev[ei + 2], st_, cudaEventRecordExternal));
          ei += 3;
          g->launches += 2;
        }
      }
      if (st_ != ctx.stream) {
        ok(cudaEventRecord(L.join, st_));
        ok(cudaStreamWaitEvent(ctx.stream, L.join, 0));
      }
    }
    ok(cudaMemcpyAsync(g->h_scal, g->d_scal, std::max<size_t>(nsteps, 1) * sizeof(StepScalars),
                       cudaMemcpyDeviceToHost, ctx.stream));
    capturing = false;
    ok(cudaStreamEndCapture(ctx.stream, &graph));
    ok(cudaGraphInstantiate(&g->exec, graph, 0));
    cudaGraphDestroy(graph);
    graph = nullptr;
    g->pool_gen = ctx.pool_gen;
    ctx.peak_pool_bytes = std::max(ctx.peak_pool_bytes, ctx.pool_bytes + g->lane_bytes);
  } catch (const Failure&) {
    if (capturing) {
      cudaGraph_t dead = nullptr;
      cudaStreamEndCapture(ctx.stream, &dead);
      if (dead) cudaGraphDestroy(dead);
    }
    if (graph) cudaGraphDestroy(graph);
    cudaGetLastError();
    graph_free(ctx);
  }
}

// Replay the captured contraction into `out`; false when there is no matching
// graph or the replay's scalars differ from the recorded run.
static bool graph_replay(Ctx& ctx, unsigned n, const qpeps_options& o, const uint32_t* prefix, unsigned k,
                         Contraction& out) {
  if (!graph_matches(ctx, n, o, prefix, k)) return false;
  GraphPlan* g = ctx.graph;
  const auto t0 = std::chrono::steady_clock::now();
  cuda_check(cudaSetDevice(ctx.device), "cudaSetDevice");
  cuda_check(cudaEventRecord(ctx.ev[0], ctx.stream), "event");
  cuda_check(cudaGraphLaunch(g->exec, ctx.stream), "graph launch");
  cuda_check(cudaEventRecord(ctx.ev[1], ctx.stream), "event");
  cuda_check(cudaStreamSynchronize(ctx.stream), "graph synchronize");
  ctx.d2h_bytes += std::max<size_t>(g->nsteps, 1) * sizeof(StepScalars);
  ctx.h2d_bytes += g->seed_bytes;
  const int R = g->base.plan.R;
  size_t si = 0;
  bool same = true;
  std::string trail;  // per step: recorded / replayed output entries and plan units, error bits
  for (size_t ci = 0; ci < g->chunks.size(); ++ci)
    for (size_t sj = 0; sj < g->chunks[ci].steps.size(); ++sj) {
      const GraphStepRec& st = g->chunks[ci].steps[sj];
      const StepScalars& h = g->h_scal[si++];
      if (st.terms && trail.size() < 1500) {
        char buf[128];
        std::snprintf(buf, sizeof buf, " [%zu.%zu out %llu/%llu units %u/%llu err %u]", ci, sj,
                      (unsigned long long)st.out, h.out_count, st.pc.parts, h.plan_units, h.error);
        trail += buf;
      }
      if (h.error & kErrBounds) {
        char msg[200];
        std::snprintf(msg, sizeof msg,
                      "a kernel's bounds check failed (access skipped) in the graph replay, batch %zu step %zu "
                      "(scatter kind %u, %u partitions); steps:",
                      ci, sj, st.pc.scatter_kind, st.pc.parts);
        graph_free(ctx);
        fail(QPEPS_ERR_CUDA, std::string(msg) + trail);
      }
      if (!st.terms) continue;
      same = same && h.error == 0 && h.out_count == st.out;
      for (int r = 0; r < R; ++r) same = same && h.weight_sum[r] == st.weight_sum[r] && h.final_sum[r] == st.final_sum[r];
    }
  if (!same) {
    graph_free(ctx);
    return false;
  }
  out = g->base;
  float ms = 0;
  cudaEventElapsedTime(&ms, ctx.ev[0], ctx.ev[1]);
  out.rs.device_ms = ms;
  // Kernel times per step (with several lanes they overlap in time, so their
  // sum can exceed device_ms).
  out.rs.scatter_ms = out.rs.merge_ms = 0;
  for (size_t ei = 0; ei + 2 < g->ev.size(); ei += 3) {
    float a = 0, b = 0;
    cudaEventElapsedTime(&a, g->ev[ei], g->ev[ei + 1]);
    cudaEventElapsedTime(&b, g->ev[ei + 1], g->ev[ei + 2]);
    out.rs.scatter_ms += a;
    out.rs.merge_ms += b;
  }
  out.rs.launches = g->launches;
  out.rs.forms = QPEPS_ROWS_REPLAY;
  out.elapsed = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
  return true;
}

// Contraction plus the host<->device bytes it moved.
static void contract(Ctx& ctx, unsigned n, const qpeps_options& o, const uint32_t* prefix, unsigned k,
                     Contraction& out) {
  const uint64_t h0 = ctx.h2d_bytes, d0 = ctx.d2h_bytes;
  if (!(o.use_graph && graph_replay(ctx, n, o, prefix, k, out))) {
    GraphRecorder rec;
    if (o.use_graph) ctx.rec = &rec;
    try {
      contract_impl(ctx, n, o, prefix, k, out);
    } catch (...) {
      ctx.rec = nullptr;
      throw;
    }
    ctx.rec = nullptr;
    if (rec.compared && same_call(ctx, n, o, prefix, k) && !ctx.graph->exec) {
      if (!same_rows(ctx.graph->base, out)) {
        // As after a replay that differs: the record goes, and a run of its own
        // answers.
        graph_free(ctx);
        Contraction again;
        contract_impl(ctx, n, o, prefix, k, again);
        out = std::move(again);
        record_rows(ctx, n, o, prefix, k, out);
      } else {
        out.rs.forms |= QPEPS_ROWS_CHECKED;
      }
    } else if (rec.compared) {
      record_rows(ctx, n, o, prefix, k, out);
    } else if (o.use_graph) {
      graph_build(ctx, n, o, prefix, k, out, rec);
    }
  }
  out.h2d_bytes = ctx.h2d_bytes - h0;
  out.d2h_bytes = ctx.d2h_bytes - d0;
}

static void contract_impl(Ctx& ctx, unsigned n, const qpeps_options& o, const uint32_t* prefix, unsigned k,
                          Contraction& out) {
  auto t0 = std::chrono::steady_clock::now();
  if (n > 42) fail(QPEPS_ERR_RANGE, "the packed u128 virtual-boundary backend supports N <= 42");
  out.rows.assign(n, RowAcc());
  if (n == 0) {
    out.count = 1;
    out.peak_states = 1;
    return;
  }
  cuda_check(cudaSetDevice(ctx.device), "cudaSetDevice");
  certify_c(ctx.c);
  if (!ctx.c_uploaded) {
    cuda_check(upload_c_table(ctx.c_dev, ctx.stream), "upload C table");
    ctx.c_uploaded = true;
  }
  // Completions of a k-row prefix place n - k queens in distinct columns:
  // the count and every row weight are at most (n - k)!.
  out.plan = make_plan(ctx, n, o, n - std::min(k, n));
  const u64 mask = (1ull << n) - 1;
  std::vector<Item> items;
  unsigned row0 = 0;
  if (k > 0) {
    if (k > n) fail(QPEPS_ERR_RANGE, "prefix longer than the board");
    State s{0, 0, 0};
    bool legal = true;
    for (unsigned r = 0; r < k; ++r) {
      if (prefix[r] >= n) fail(QPEPS_ERR_RANGE, "prefix column out of range");
      const u64 b = 1ull << prefix[r];
      if ((s.cols | s.dr | s.dl) & b) {
        legal = false;
        break;
      }
      const u128 key = row_successor<u128>(s, b, n, mask);
      s = unpack<u128>(key, n, mask);
    }
    if (!legal) {
      out.count = 0;
      out.peak_states = 1;
      return;
    }
    items.push_back(Item{pack<u128>(s.cols, s.dr, s.dl, n), 1});
    row0 = k;
  } else {
    items.push_back(Item{0, 1});
  }
  // Seed rows on the host: the first row applies the orbit weights
  // (src/lib.rs:721-749); further rows only when a slice depth is requested.
  const bool orbit = (k == 0) && o.symmetry;
  const unsigned depth =
      std::max<unsigned>(o.slice_depth ? o.slice_depth : std::max(1u, ctx.tune.slice_rows), row0 == 0 ? 1 : row0);
  while (row0 < depth && row0 < n) {
    RowAcc& acc = out.rows[row0];
    items = host_expand(n, items, row0, orbit && row0 == 0, acc, out.plan.grain == QPEPS_GRAIN_SITE);
    acc.device_row = false;
    out.peak_states = std::max<u64>(out.peak_states, items.size());
    ++row0;
  }
  // (Known for a whole board with the orbits, about twice that without them,
  // estimated below a prefix.)
  out.plan.batch_states = serve_estimate(n, k) * (k ? 3.0 : o.symmetry ? 1.0 : 2.0);
  out.plan.prefix = k > 0;
  out.plan.group_states =
      group_rows_states(n, k, out.plan.batch_states / (k ? 3.0 : 1.0), k ? 3.0 : 1.01, o.use_graph);
  // Predictive slicing: when the merged frontier is estimated not to fit the
  // device budget, contract groups of slices (first-row orbit slices, or
  // deeper prefix slices) one chunk at a time instead of halving a live
  // frontier at its peak and spilling it to the host.
  if (o.slice_depth == 0 && out.plan.grain == QPEPS_GRAIN_ROW && row0 < n && !items.empty()) {
    const double per_state = 2.0 * (double)entry_bytes(out.plan) + 1.25 * (double)cand_bytes(out.plan);
    // A placed prefix's frontier is estimated from the average over all
    // prefixes of its depth; central prefixes run to several times that (N=22:
    // 1.8-2.6x at depth 3), and an underestimate costs host spills at the peak
    // rows, so prefixes are sliced on four times the estimate.
    double est_total = serve_estimate(n, k) * (k ? 4.0 : 1.0);
    const bool fits = out.plan.budget.holds((size_t)std::min(1e18, est_total * per_state / 0.8));
    const double cap_states = fits ? est_total : 0.8 * (double)(size_t)out.plan.budget / per_state;
    while (!fits && est_total > cap_states && row0 + 2 < n) {
      // Slices are uneven (centre columns carry more states): tuned margin.
      const double est_item = est_total / (double)items.size() * ctx.tune.slice_margin;
      if (est_item <= cap_states) {
        const size_t per_chunk = std::max<size_t>(1, (size_t)(cap_states / est_item));
        std::vector<HostChunk> chunks;
        for (size_t lo = 0; lo < items.size(); lo += per_chunk) {
          std::vector<Item> part(items.begin() + lo, items.begin() + std::min(items.size(), lo + per_chunk));
          chunks.push_back(chunk_from_items(out.plan, part, row0));
        }
        out.slice_depth = row0;
        out.plan.batch_states = std::min(est_item * (double)per_chunk, cap_states);
        out.plan.group_states = group_rows_states(n, k, est_total / (double)items.size() * (double)per_chunk,
                                                  std::min(2.5, ctx.tune.slice_margin), o.use_graph);
        run_chunks(ctx, out.plan, std::move(chunks), out.rows, out.rs);
        items.clear();
        break;
      }
      RowAcc& acc = out.rows[row0];
      items = host_expand(n, items, row0, false, acc, out.plan.grain == QPEPS_GRAIN_SITE);
      acc.device_row = false;
      ++row0;
    }
  }
  if (!items.empty()) {
    out.slice_depth = std::max(out.slice_depth, row0);
    contract_items(ctx, out, items, row0);
  }
  out.peak_states = std::max<u64>(out.peak_states, out.rs.peak_states);
  // Count: host-finished boards plus device final sums, then CRT.
  u64 res[kMaxResidues];
  for (int r = 0; r < out.plan.Rc; ++r) res[r] = out.rs.final_res[r];
  out.count = crt_reconstruct(res, out.plan.Rc);
  if (out.count > factorial(out.plan.free_rows))
    fail(QPEPS_ERR_CRT_BOUND, "CRT reconstruction exceeds certified N! count bound");
  out.elapsed = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
}

static u128 row_weight(const Contraction& c, const RowAcc& a) {
  if (!a.device_row) return a.weight_exact;
  u64 res[kMaxResidues];
  for (int r = 0; r < c.plan.Rc; ++r) res[r] = a.weight_res[r];
  return crt_reconstruct(res, c.plan.Rc);
}

static void fill_result(const Ctx& ctx, const Contraction& c, unsigned n, qpeps_result* r, qpeps_layer* layers,
                        uint32_t cap) {
  std::memset(r, 0, sizeof *r);
  r->n = n;
  r->row_forms = c.rs.forms;
  r->count = to_abi(c.count);
  r->elapsed_s = c.elapsed;
  r->peak_states = c.peak_states;
  u128 cand = 0, matched = 0;
  uint32_t nl = 0;
  for (unsigned row = 0; row < c.rows.size(); ++row) {
    const RowAcc& a = c.rows[row];
    if (!a.used) continue;
    cand += a.candidates;
    matched += a.matched;
    if (layers && nl < cap) {
      qpeps_layer& L = layers[nl];
      std::memset(&L, 0, sizeof L);
      L.row = row;
      L.input_states = a.input_states;
      L.tensor_entries_examined = to_abi(a.examined);
      L.tensor_entries_matched = to_abi(a.tmatched);
      L.row_operator_candidates = to_abi(a.candidates);
      L.row_operator_matched = to_abi(a.matched);
      L.completed_row_terms = to_abi(a.completed);
      L.output_states = a.output_states;
      L.output_weight = to_abi(row_weight(c, a));
      L.elapsed_s = a.elapsed;
      L.peak_rss_bytes = ctx.pool_bytes;
    }
    ++nl;
  }
  r->n_layers = nl;
  // The compiled row operator examines the 17 C entries once (src/lib.rs:5654-5655);
  // the sitewise backend reports the entries its per-parent site kernel matched.
  u128 examined = 0, tmatched = 0;
  for (const RowAcc& a : c.rows) {
    examined += a.examined;
    tmatched += a.tmatched;
  }
  const bool sitewise = n && c.plan.grain == QPEPS_GRAIN_SITE;
  r->tensor_entries_examined = to_abi(sitewise ? examined : (n ? 17 : 0));
  r->tensor_entries_matched = to_abi(sitewise ? tmatched : (n ? 17 : 0));
  r->row_operator_candidates = to_abi(cand);
  r->row_operator_matched = to_abi(matched);
  r->peak_rss_bytes = ctx.peak_pool_bytes;
  r->residues = n ? (uint32_t)c.plan.Rc : 0;
  r->key_bits = n ? (uint32_t)c.plan.key_bits : 0;
  r->slice_depth = c.slice_depth;
  r->batches = c.rs.batches;
  r->merge = n ? (uint32_t)c.plan.merge : 0;
  r->entries_in = c.rs.entries_in;
  r->entries_out = c.rs.entries_out;
  r->candidates = c.rs.candidates;
  r->gpu_launches = c.rs.launches;
  r->peak_device_bytes = ctx.peak_pool_bytes;
  r->device_ms = c.rs.device_ms;
  r->merge_kernel_ms = c.rs.merge_ms;
  r->scatter_kernel_ms = c.rs.scatter_ms;
  r->merge_kernel_launches = c.rs.merge_launches;
  r->merge_kernel_bytes = c.rs.merge_bytes;
  r->tail_row = n ? c.plan.tail_row : 0;
  r->exact_weights = (n && c.plan.w64) ? 1u : 0u;
  r->tail_items = c.rs.tail_items;
  r->tail_overflow = c.rs.tail_overflow;
  r->tail_kernel_ms = c.rs.tail_ms;
  r->h2d_bytes = c.h2d_bytes;
  r->d2h_bytes = c.d2h_bytes;
  for (int i = 0; i < kMaxResidues; ++i) {
    r->residue_primes[i] = i < (n ? c.plan.Rc : 0) ? kPrimes[i] : 0;
    r->count_residues[i] = i < (n ? c.plan.Rc : 0) ? (uint64_t)(c.count % kPrimes[i]) : 0;
  }
}

static void set_err(char* err, size_t len, const std::string& msg) {
  if (err && len) std::snprintf(err, len, "%s", msg.c_str());
}

template <typename F>
static int guarded(char* err, size_t err_len, F&& f) {
  try {
    f();
    if (err && err_len) err[0] = 0;
    return QPEPS_OK;
  } catch (const Failure& e) {
    set_err(err, err_len, e.msg);
    return e.code;
  } catch (const std::bad_alloc&) {
    set_err(err, err_len, "host allocation failed");
    return QPEPS_ERR_OOM;
  } catch (const std::exception& e) {
    set_err(err, err_len, e.what());
    return QPEPS_ERR_INVALID;
  }
}

static qpeps_options effective_options(const qpeps_options* opt) {
  qpeps_options o;
  qpeps_options_default(&o);
  if (opt) {
    if (opt->struct_size != sizeof(qpeps_options)) fail(QPEPS_ERR_INVALID, "qpeps_options.struct_size mismatch");
    o = *opt;
  }
  return o;
}


// ===========================================================================
// Serving: continuous batching of counting requests.
//
// A request is (N, placed prefix of k rows). Small requests share one device
// boundary in a context of their own: keys carry the request's slot
// (SlotLayout), every step contracts one row of every admitted request with
// one count + scatter + merge launch triple, a request whose last row has
// been contracted frees its slot, and queued requests are admitted between
// steps while slots and the batch's device budget allow (an admitted
// request's estimated peak frontier is reserved until it finishes). Requests
// whose estimated frontier is too large for the shared batch run one at a
// time through the row engine on a second context and stream, so their
// kernels overlap with the batch's on the device. Repeated requests (equal N
// and prefix, or its mirror image) can be answered from an exact result cache.

using ServeClock = std::chrono::steady_clock;

struct ServeRequest {
  uint64_t tag = 0;
  uint32_t n = 0;
  std::vector<uint32_t> prefix;
  ServeClock::time_point t_submit;
  std::string cache_key;
  double est_states = 0;
};

struct ServeSlot {
  bool used = false;
  uint64_t tag = 0;
  uint32_t n = 0, k = 0;
  std::vector<uint32_t> prefix;
  unsigned rows_left = 0;
  ServeClock::time_point t_submit, t_admit;
  std::string cache_key;
  double est_states = 0;
};

static std::string serve_cache_key(unsigned n, const std::vector<uint32_t>& prefix) {
  std::vector<uint32_t> mir(prefix.size());
  for (size_t i = 0; i < prefix.size(); ++i) mir[i] = n - 1 - prefix[i];
  const std::vector<uint32_t>& key = std::min(prefix, mir);  // vertical reflection preserves the count
  std::string s = std::to_string(n) + ":";
  for (uint32_t c : key) s += std::to_string(c) + ",";
  return s;
}

// An identical request (same N and prefix, or its mirror) that arrived while
// the first was queued or running.
struct ServeWaiter {
  uint64_t tag = 0;
  uint32_t n = 0, k = 0;
  ServeClock::time_point t_submit;
};

struct Server {
  int device = 0;
  qpeps_serve_config cfg{};
  Ctx* batch = nullptr;
  std::vector<Ctx*> large;  // one context (own stream, own pool) per large-request worker
  std::mutex mu;
  std::condition_variable cv;
  std::deque<ServeRequest> q_small, q_large;
  std::vector<qpeps_serve_completion> done;
  std::condition_variable cv_done;
  bool stop = false;
  std::thread t_batch;
  std::vector<std::thread> t_large;
  std::map<std::string, u128> cache;
  std::map<std::string, std::vector<ServeWaiter>> inflight;  // queued or running keys (cache on)
  qpeps_serve_stats stats{};
  std::string fatal;
  int fatal_code = QPEPS_OK;
  // batch state (owned by the batch thread)
  ServeSlot slots[kServeMaxSlots];
  double reserved_states = 0;
  DevBuf slot_buf;  // u64 slot_mask[64] + u64 slot_final[64][4]
  DevFrontier f;
};

// Complete a request; with `key`, also every identical request that arrived
// while it was queued or running (they waited on it instead of running again).
static void serve_complete(Server& sv, uint64_t tag, uint32_t n, uint32_t k, u128 count, int status, uint32_t path,
                           ServeClock::time_point t_submit, ServeClock::time_point t_admit,
                           const std::string* key = nullptr) {
  const auto now = ServeClock::now();
  qpeps_serve_completion c{};
  c.tag = tag;
  c.count = to_abi(count);
  c.status = status;
  c.n = n;
  c.k = k;
  c.path = path;
  c.latency_s = std::chrono::duration<double>(now - t_submit).count();
  c.queue_s = std::chrono::duration<double>(t_admit - t_submit).count();
  {
    std::lock_guard<std::mutex> lk(sv.mu);
    sv.done.push_back(c);
    sv.stats.completed += 1;
    if (key) {
      auto it = sv.inflight.find(*key);
      if (it != sv.inflight.end()) {
        for (const ServeWaiter& w : it->second) {
          qpeps_serve_completion d = c;
          d.tag = w.tag;
          d.n = w.n;
          d.k = w.k;
          d.path = 4;
          d.latency_s = std::chrono::duration<double>(now - w.t_submit).count();
          d.queue_s = std::max(0.0, std::chrono::duration<double>(t_admit - w.t_submit).count());
          sv.done.push_back(d);
          sv.stats.completed += 1;
        }
        sv.inflight.erase(it);
      }
    }
  }
  sv.cv_done.notify_all();
}

// Host-side seed boundary of a request: the prefix boundary (weight 1), or
// for k = 0 the first-row orbit states (weights 2/1). Returns false for an
// attacked prefix.
static bool serve_seeds(unsigned n, const std::vector<uint32_t>& prefix, std::vector<std::pair<State, u64>>& out,
                        unsigned* row0) {
  const u64 mask = (1ull << n) - 1;
  out.clear();
  if (prefix.empty()) {
    for (unsigned c = 0; c < n; ++c) {
      const unsigned mirror = n - 1 - c;
      if (c > mirror) continue;
      const u64 b = 1ull << c;
      State s{b, (b << 1) & mask, b >> 1};
      out.push_back({s, c == mirror ? 1ull : 2ull});
    }
    *row0 = 1;
    return true;
  }
  State s{0, 0, 0};
  for (uint32_t c : prefix) {
    const u64 b = 1ull << c;
    if ((s.cols | s.dr | s.dl) & b) return false;
    s = State{s.cols | b, ((s.dr | b) << 1) & mask, (s.dl | b) >> 1};
  }
  out.push_back({s, 1});
  *row0 = (unsigned)prefix.size();
  return true;
}

// A request's frontier can exceed its estimate (centre-column prefixes carry
// more states); admission reserves this multiple of the estimate.
constexpr double kAdmitMargin = 2.5;

// Steps a shared batch takes between looking at its queue: new requests wait
// for a chain's end, so a chain is short.
constexpr unsigned kServeChain = 6;

// Up to `want` rows of the shared boundary (f, with `terms` successor terms,
// both updated): a chain of queued steps while it is small, one step with the
// host's sizes otherwise. Returns the rows contracted (at least one).
static unsigned serve_steps(Ctx& ctx, const Plan& p, DevFrontier& f, u64& terms, unsigned want, const u64* d_mask,
                            unsigned long long* d_final) {
  if (terms == 0) {  // no state has a successor: nothing is left to add
    f.count = 0;
    cuda_check(cudaStreamSynchronize(ctx.stream), "serve synchronize");  // (seeds may still be on their way)
    return want;
  }
  const u32 shape = 2;  // small merge CTAs, as in run_queued_rows
  const u32 pcap = partition_capacity(shape);
  double mean = chain_mean(ctx, pcap);
  StepSource source{nullptr, mean, 0, 8 * (u32)ctx.sms};
  if (want > 1 && terms <= kQueueTerms) {
    // A row multiplies the terms by less than 4 on average once three rows are
    // placed; a chain that outgrows its buffers stops and is sized below.
    const u64 most = std::min<u64>(kQueueTerms, std::max<u64>(1u << 20, 4 * terms));
    const u32 parts_cap = source.parts_cap = (u32)source.partitions(most);
    const size_t region_bytes = (size_t)parts_cap * pcap * cand_bytes(p);
    const size_t cursor_bytes = (size_t)parts_cap * 4 * 8;
    const size_t table_bytes = region_bytes + (cursor_bytes + 255) / 256 * 256;
    if (chain_buffers(ctx, p, f, most, table_bytes, want, "serve partitions")) {
      StepScalars* d = queue_scalars(ctx, want);
      StepScalars* h = ctx.h_queue;
      h[0].out_count = f.count;
      h[0].next_terms = terms;
      u32* cursors = reinterpret_cast<u32*>(static_cast<char*>(ctx.table.ptr) + region_bytes);
      const FrontierView view = view_of(p, ctx.front[0], f.cap);
      PartitionCfg pc{2, ctx.sms, parts_cap, pcap, 2, 8, ctx.tune.parents_per_lane, shape, 1, 1, 2u};
      cuda_check(cudaMemcpyAsync(d, h, (want + 1) * sizeof(StepScalars), cudaMemcpyHostToDevice, ctx.stream),
                 "queued step scalars");
      cuda_check(cudaMemsetAsync(cursors, 0, cursor_bytes, ctx.stream), "clear cursors");
      u64 entries = f.count;
      double likely = (double)terms;
      for (unsigned i = 0; i < want; ++i) {
        const u64 fits = (u64)std::min((double)most, likely);
        pc.queued = source;
        pc.queued.prev = d + i;
        pc.parts = (u32)source.partitions(fits);
        cuda_check(launch_serve_scatter(pc, view, std::max<u64>(entries, 1), d_mask, ctx.table.ptr, cursors, d + i + 1,
                                        ctx.stream),
                   "serve scatter");
        cuda_check(launch_serve_merge(pc, ctx.table.ptr, cursors, view, d_mask, d_final, d + i + 1, ctx.stream),
                   "serve merge");
        entries = fits;
        likely *= 4;
      }
      cuda_check(cudaMemcpyAsync(h, d, (want + 1) * sizeof(StepScalars), cudaMemcpyDeviceToHost, ctx.stream),
                 "read step scalars");
      cuda_check(cudaStreamSynchronize(ctx.stream), "serve chain");
      unsigned done = 0;
      while (done < want && !h[done + 1].error) ++done;
      if (done) {
        f.count = h[done].out_count;
        terms = h[done].next_terms;
      }
      if (done < want) chain_ended(ctx, h[done + 1], mean, pcap);
      if (done < want && (h[done + 1].error & kErrBounds)) fail(QPEPS_ERR_CUDA, "serving: a bounds check failed");
      if (done) return done;
    }
  }
  for (int attempt = 0;; ++attempt) {
    const u32 parts = (u32)std::max<u64>(1, (u64)((double)terms / mean) + 1);
    const size_t region_bytes = (size_t)parts * pcap * cand_bytes(p);
    const size_t table_bytes = region_bytes + ((size_t)parts * 4 + 255) / 256 * 256;
    if (ctx.table.bytes < table_bytes) buf_release(ctx, ctx.table);
    if (!ensure_front(ctx, p, f, std::max<u64>(f.count, terms), ctx.table.ptr ? 0 : table_bytes))
      fail(QPEPS_ERR_CAPACITY, "serving batch budget exceeded");
    buf_reserve(ctx, ctx.table, table_bytes, p.budget, "serve partitions");
    const FrontierView view = view_of(p, ctx.front[0], f.cap);
    u32* cursors = reinterpret_cast<u32*>(static_cast<char*>(ctx.table.ptr) + region_bytes);
    PartitionCfg pc{2, ctx.sms, parts, pcap, 2, 1, ctx.tune.parents_per_lane, shape, 1, 1, 2u};
    cuda_check(cudaMemsetAsync(cursors, 0, (size_t)parts * 4, ctx.stream), "clear cursors");
    cuda_check(cudaMemsetAsync(ctx.d_sc, 0, sizeof(StepScalars), ctx.stream), "clear scalars");
    cuda_check(launch_serve_scatter(pc, view, f.count, d_mask, ctx.table.ptr, cursors, ctx.d_sc, ctx.stream),
               "serve scatter");
    cuda_check(launch_serve_merge(pc, ctx.table.ptr, cursors, view, d_mask, d_final, ctx.d_sc, ctx.stream),
               "serve merge");
    sync_scalars(ctx);
    if (ctx.h_sc->error & kErrOverflow) {
      if (attempt >= 4) fail(QPEPS_ERR_CAPACITY, "serving partition overflow persists");
      chain_ended(ctx, *ctx.h_sc, mean, pcap);
      mean *= 0.6;
      continue;
    }
    if (ctx.h_sc->error) fail(QPEPS_ERR_CAPACITY, "serving device capacity error");
    f.count = ctx.h_sc->out_count;
    terms = ctx.h_sc->next_terms;
    return 1;
  }
}

static void serve_batch_loop(Server& sv) {
  Ctx& ctx = *sv.batch;
  cuda_check(cudaSetDevice(sv.device), "cudaSetDevice");
  Plan p{};
  p.n = 19;
  p.free_rows = 19;
  p.R = 2;
  p.Rc = 2;
  p.key_bits = 64;
  p.grain = QPEPS_GRAIN_ROW;
  p.merge = QPEPS_MERGE_PARTITION;
  p.budget = Budget((size_t)sv.cfg.batch_budget_bytes);
  p.threads = 256;
  p.tail_row = p.n;
  p.w64 = true;  // N <= 19: exact weights (19! < 2^63)
  const size_t eb = entry_bytes(p);
  buf_reserve(ctx, sv.slot_buf, kServeMaxSlots * 5 * sizeof(u64), p.budget, "serve slots");
  u64* d_mask = static_cast<u64*>(sv.slot_buf.ptr);
  unsigned long long* d_final = reinterpret_cast<unsigned long long*>(d_mask + kServeMaxSlots);
  u64 h_mask[kServeMaxSlots] = {0};
  cuda_check(cudaMemsetAsync(sv.slot_buf.ptr, 0, kServeMaxSlots * 5 * sizeof(u64), ctx.stream), "clear slots");
  const double budget_states = (double)p.budget / (2.4 * (double)eb);
  std::vector<u64> seed_keys, seed_weights;
  std::vector<std::pair<State, u64>> seeds;
  u64 seed_terms = 0;
  u64 next_terms = 0;  // successor terms of the shared boundary
  // Finished boards' sums on the device grow on; a request's count is what its
  // slot's sum grew by.
  unsigned long long h_base[kServeMaxSlots] = {0};
  unsigned long long* h_final = nullptr;  // pinned: the sums, then seed staging
  uint8_t* h_stage = nullptr;
  struct Pinned {
    void* p = nullptr;
    ~Pinned() {
      if (p) cudaFreeHost(p);
    }
  } pinned;
  cuda_check(cudaMallocHost(&pinned.p, kServeMaxSlots * 4 * sizeof(u64) + kSeedStage), "pinned serve buffers");
  h_final = static_cast<unsigned long long*>(pinned.p);
  h_stage = reinterpret_cast<uint8_t*>(h_final + kServeMaxSlots * 4);
  std::memset(h_final, 0, kServeMaxSlots * 4 * sizeof(u64));
  while (true) {
    // Admission.
    seed_keys.clear();
    seed_weights.clear();
    seed_terms = 0;
    bool mask_dirty = false;
    {
      std::unique_lock<std::mutex> lk(sv.mu);
      bool any = false;
      for (const ServeSlot& sl : sv.slots) any = any || sl.used;
      if (!any && sv.q_small.empty()) {
        if (sv.stop) break;
        sv.cv.wait_for(lk, std::chrono::milliseconds(50));
        continue;
      }
      while (!sv.q_small.empty()) {
        ServeRequest& rq = sv.q_small.front();
        int free_slot = -1;
        for (unsigned i = 0; i < std::min<unsigned>(sv.cfg.max_slots, kServeMaxSlots); ++i)
          if (!sv.slots[i].used) {
            free_slot = (int)i;
            break;
          }
        if (free_slot < 0) break;
        if (any && sv.reserved_states + kAdmitMargin * rq.est_states > budget_states) break;
        unsigned row0 = 0;
        ServeRequest r = std::move(rq);
        sv.q_small.pop_front();
        lk.unlock();
        const auto t_admit = ServeClock::now();
        if (!serve_seeds(r.n, r.prefix, seeds, &row0)) {
          serve_complete(sv, r.tag, r.n, (uint32_t)r.prefix.size(), 0, QPEPS_OK, 3, r.t_submit, t_admit,
                         &r.cache_key);
        } else if (row0 >= r.n) {
          serve_complete(sv, r.tag, r.n, (uint32_t)r.prefix.size(), 1, QPEPS_OK, 3, r.t_submit, t_admit,
                         &r.cache_key);
        } else {
          ServeSlot& sl = sv.slots[free_slot];
          sl.used = true;
          sl.tag = r.tag;
          sl.n = r.n;
          sl.k = (uint32_t)r.prefix.size();
          sl.prefix = r.prefix;
          sl.rows_left = r.n - row0;
          sl.t_submit = r.t_submit;
          sl.t_admit = t_admit;
          sl.cache_key = r.cache_key;
          sl.est_states = kAdmitMargin * r.est_states;
          sv.reserved_states += sl.est_states;
          h_mask[free_slot] = (1ull << r.n) - 1;
          mask_dirty = true;
          for (auto& sd : seeds) {
            const State& st = sd.first;
            seed_keys.push_back(serve_key((unsigned)free_slot, st.cols, st.dr, st.dl));
            seed_weights.push_back(sd.second);
            seed_terms += (u64)__builtin_popcountll(~(st.cols | st.dr | st.dl) & h_mask[free_slot]);
          }
          any = true;
        }
        lk.lock();
      }
    }
    unsigned steps = 0;
    try {
      if (mask_dirty)
        cuda_check(cudaMemcpyAsync(d_mask, h_mask, sizeof h_mask, cudaMemcpyHostToDevice, ctx.stream), "slot masks");
      if (!seed_keys.empty()) {
        // Append the seeds to the shared boundary.
        const u64 m = seed_keys.size();
        if (!ensure_front(ctx, p, sv.f, sv.f.count + m, ctx.table.bytes))
          fail(QPEPS_ERR_CAPACITY, "serving batch budget cannot hold the admitted seeds");
        // (At most 64 requests of at most 19 seeds: the staging holds them.)
        char* base = static_cast<char*>(ctx.front[0].ptr);
        u64* st_key = reinterpret_cast<u64*>(h_stage);
        u32* st_word = reinterpret_cast<u32*>(st_key + m);
        static_assert(kServeMaxSlots * 19 * 16 <= kSeedStage, "seed staging");
        for (u64 i = 0; i < m; ++i) {
          st_key[i] = seed_keys[i];
          st_word[i] = (u32)seed_weights[i];
          st_word[m + i] = (u32)(seed_weights[i] >> 32);
        }
        cuda_check(cudaMemcpyAsync(base + sv.f.count * 8, st_key, m * 8, cudaMemcpyHostToDevice, ctx.stream),
                   "seed keys");
        for (int r = 0; r < 2; ++r)
          cuda_check(cudaMemcpyAsync(base + sv.f.cap * 8 + ((size_t)r * sv.f.cap + sv.f.count) * 4, st_word + r * m,
                                     m * 4, cudaMemcpyHostToDevice, ctx.stream),
                     "seed weights");
        sv.f.count += m;
        next_terms += seed_terms;
      }
      bool active = false;
      unsigned first_end = ~0u;  // rows until the first request ends
      for (const ServeSlot& sl : sv.slots)
        if (sl.used) {
          active = true;
          first_end = std::min(first_end, sl.rows_left);
        }
      if (!active) continue;
      steps = serve_steps(ctx, p, sv.f, next_terms, std::min(first_end, kServeChain), d_mask, d_final);
      if (steps == first_end) {
        cuda_check(cudaMemcpyAsync(h_final, d_final, kServeMaxSlots * 4 * sizeof(u64), cudaMemcpyDeviceToHost, ctx.stream),
                   "slot finals");
        cuda_check(cudaStreamSynchronize(ctx.stream), "slot finals");
      }
    } catch (const Failure& e) {
      if (e.code != QPEPS_ERR_CAPACITY) throw;
      // The shared batch outgrew its device budget: every admitted request
      // restarts from its prefix on the large-request context, and the batch
      // starts empty.
      std::vector<ServeRequest> moved;
      for (unsigned i = 0; i < kServeMaxSlots; ++i) {
        ServeSlot& sl = sv.slots[i];
        if (!sl.used) continue;
        ServeRequest r;
        r.tag = sl.tag;
        r.n = sl.n;
        r.prefix = sl.prefix;
        r.t_submit = sl.t_submit;
        r.cache_key = sl.cache_key;
        r.est_states = sl.est_states / kAdmitMargin;
        moved.push_back(std::move(r));
        sl.used = false;
        h_mask[i] = 0;
      }
      sv.f.count = 0;
      next_terms = 0;
      std::memset(h_base, 0, sizeof h_base);
      buf_release(ctx, ctx.table);
      cuda_check(cudaMemsetAsync(sv.slot_buf.ptr, 0, kServeMaxSlots * 5 * sizeof(u64), ctx.stream), "clear slots");
      cuda_check(cudaStreamSynchronize(ctx.stream), "clear slots");
      {
        std::lock_guard<std::mutex> lk(sv.mu);
        sv.reserved_states = 0;
        sv.stats.batch_requeued += moved.size();
        for (ServeRequest& r : moved) sv.q_large.push_back(std::move(r));
      }
      sv.cv.notify_all();
      continue;
    }
    {
      std::lock_guard<std::mutex> lk(sv.mu);
      sv.stats.batch_steps += steps;
    }
    // Finished requests.
    bool any_done = false;
    for (ServeSlot& sl : sv.slots)
      if (sl.used && (sl.rows_left -= steps) == 0) any_done = true;
    if (!any_done) continue;
    for (unsigned i = 0; i < kServeMaxSlots; ++i) {
      ServeSlot& sl = sv.slots[i];
      if (!sl.used || sl.rows_left != 0) continue;
      const u128 count = h_final[i * 4] - h_base[i];
      h_base[i] = h_final[i * 4];
      h_mask[i] = 0;
      sl.used = false;
      {
        std::lock_guard<std::mutex> lk(sv.mu);
        sv.reserved_states -= sl.est_states;
        if (sv.cfg.use_cache) sv.cache[sl.cache_key] = count;
      }
      serve_complete(sv, sl.tag, sl.n, sl.k, count, QPEPS_OK, 0, sl.t_submit, sl.t_admit, &sl.cache_key);
    }
  }
}

// One large-request worker: takes the oldest queued large request and
// contracts it alone on its own context and stream; several workers overlap
// their requests on the device, each within an equal share of the large
// budget, so a long request no longer holds up every other large one.
static void serve_large_loop(Server& sv, size_t w) {
  cuda_check(cudaSetDevice(sv.device), "cudaSetDevice");
  while (true) {
    ServeRequest r;
    {
      std::unique_lock<std::mutex> lk(sv.mu);
      sv.cv.wait(lk, [&] { return sv.stop || !sv.q_large.empty(); });
      if (sv.q_large.empty()) break;
      r = std::move(sv.q_large.front());
      sv.q_large.pop_front();
    }
    const auto t_admit = ServeClock::now();
    qpeps_options o;
    qpeps_options_default(&o);
    o.device_budget_bytes = sv.cfg.large_budget_bytes / std::max<size_t>(1, sv.large.size());
    Contraction con;
    int status = QPEPS_OK;
    u128 count = 0;
    try {
      contract(*sv.large[w], r.n, o, r.prefix.empty() ? nullptr : r.prefix.data(), (unsigned)r.prefix.size(), con);
      count = con.count;
    } catch (const Failure& e) {
      status = e.code;
    }
    {
      std::lock_guard<std::mutex> lk(sv.mu);
      sv.stats.large_runs += 1;
      if (status == QPEPS_OK && sv.cfg.use_cache) sv.cache[r.cache_key] = count;
    }
    serve_complete(sv, r.tag, r.n, (uint32_t)r.prefix.size(), count, status, 1, r.t_submit, t_admit, &r.cache_key);
  }
}

static void serve_thread_main(Server& sv, bool large, size_t w) {
  try {
    if (large)
      serve_large_loop(sv, w);
    else
      serve_batch_loop(sv);
  } catch (const Failure& e) {
    std::lock_guard<std::mutex> lk(sv.mu);
    sv.fatal = e.msg;
    sv.fatal_code = e.code;
    sv.stop = true;
  } catch (const std::exception& e) {
    std::lock_guard<std::mutex> lk(sv.mu);
    sv.fatal = e.what();
    sv.fatal_code = QPEPS_ERR_INVALID;
    sv.stop = true;
  }
  sv.cv.notify_all();
  sv.cv_done.notify_all();
}
}  // namespace qpeps

using namespace qpeps;

// ---- tuning --------------------------------------------------------------

static qpeps_tuning tuning_of(const Ctx::Tune& t) {
  qpeps_tuning q;
  std::memset(&q, 0, sizeof q);
  q.struct_size = sizeof(qpeps_tuning);
  q.scatter_kind = t.scatter_kind;
  q.parents_per_lane = t.parents_per_lane;
  q.merge_kind = t.merge_kind;
  q.wide_merge = t.wide_merge;
  q.wide_above_parts = t.wide_above_parts;
  q.spread_cursors_below = t.spread_cursors_below;
  q.fold_weights = t.fold_weights;
  q.partition_fill = t.partition_fill;
  q.slice_margin = t.slice_margin;
  q.unit_target = t.unit_target;
  q.unit_sample = t.unit_sample;
  q.batch_lanes = t.batch_lanes;
  q.merge_compact = t.merge_compact;
  q.scatter_block = t.scatter_block;
  q.merge_auto = t.merge_auto;
  q.slice_rows = t.slice_rows;
  return q;
}

static Ctx::Tune tune_from(const qpeps_tuning& q) {
  if (q.struct_size != sizeof(qpeps_tuning)) fail(QPEPS_ERR_INVALID, "qpeps_tuning.struct_size mismatch");
  if (q.scatter_kind > 4) fail(QPEPS_ERR_INVALID, "scatter_kind must be 0..4");
  if (q.unit_target < 256 || q.unit_target > 2048) fail(QPEPS_ERR_INVALID, "unit_target must be in [256, 2048]");
  if (q.unit_sample < 1 || q.unit_sample > 64 || (q.unit_sample & (q.unit_sample - 1)))
    fail(QPEPS_ERR_INVALID, "unit_sample must be a power of two in [1, 64]");
  if (q.batch_lanes < 1 || q.batch_lanes > 8) fail(QPEPS_ERR_INVALID, "batch_lanes must be in [1, 8]");
  if (q.merge_compact > 1) fail(QPEPS_ERR_INVALID, "merge_compact must be 0 or 1");
  if (q.scatter_block != 128 && q.scatter_block != 256 && q.scatter_block != 512)
    fail(QPEPS_ERR_INVALID, "scatter_block must be 128, 256 or 512");
  if (q.merge_auto != QPEPS_MERGE_PARTITION && q.merge_auto != QPEPS_MERGE_HASH)
    fail(QPEPS_ERR_INVALID, "merge_auto must be QPEPS_MERGE_PARTITION or QPEPS_MERGE_HASH");
  if (q.slice_rows < 1 || q.slice_rows > 4) fail(QPEPS_ERR_INVALID, "slice_rows must be in [1, 4]");
  if (q.parents_per_lane != 2 && q.parents_per_lane != 4) fail(QPEPS_ERR_INVALID, "parents_per_lane must be 2 or 4");
  if (q.merge_kind > 1) fail(QPEPS_ERR_INVALID, "merge_kind must be 0 or 1");
  if (q.wide_merge > 3) fail(QPEPS_ERR_INVALID, "wide_merge must be 0, 1, 2 or 3");
  if (q.fold_weights > 2) fail(QPEPS_ERR_INVALID, "fold_weights must be 0, 1 or 2");
  if (!(q.partition_fill >= 0.3 && q.partition_fill <= 0.95))
    fail(QPEPS_ERR_INVALID, "partition_fill must be in [0.3, 0.95]");
  if (!(q.slice_margin >= 1.0 && q.slice_margin <= 64.0)) fail(QPEPS_ERR_INVALID, "slice_margin must be in [1, 64]");
  Ctx::Tune t;
  t.scatter_kind = q.scatter_kind;
  t.parents_per_lane = q.parents_per_lane;
  t.merge_kind = q.merge_kind;
  t.wide_merge = q.wide_merge;
  t.wide_above_parts = q.wide_above_parts;
  t.spread_cursors_below = q.spread_cursors_below;
  t.fold_weights = q.fold_weights;
  t.partition_fill = q.partition_fill;
  t.slice_margin = q.slice_margin;
  t.unit_target = q.unit_target;
  t.unit_sample = q.unit_sample;
  t.batch_lanes = q.batch_lanes;
  t.merge_compact = q.merge_compact;
  t.scatter_block = q.scatter_block;
  t.merge_auto = q.merge_auto;
  t.slice_rows = q.slice_rows;
  return t;
}

static void apply_tune(Ctx& c, const Ctx::Tune& t) {
  c.tune = t;
  c.partition_fill = t.partition_fill;
  c.chain_fill = 1.0;
}

// Autotuner: coordinate descent over the knobs of a contraction, starting
// from the context's tuning. Each pass tries, one dimension at a time, every
// value of that dimension with the others at their best so far and keeps the
// fastest (device time of a replay, best of `repeats` after one untimed warm-up
// run; every count is checked against known_count); passes repeat until one
// changes nothing (at most three). A candidate whose warm-up run takes more
// than three times the best so far is not timed further. A value is kept only
// if it gains half a percent and 5 us (at N = 17, where most knobs reach nothing
// that runs, the best of two runs differs by 0.2 %, at N = 11 by 3 us) and calls without use_graph do
// not get 2 % slower by it: some values turn chains, column-grouped rows or
// one-CTA boards off (N = 11, replays 0.200 -> 0.188 ms by the global table, but
// other calls 0.102 -> 0.192).
//   scatter kind (not the class-grouped one, which is not graph-captured),
//   parents per lane, scatter block size, merge kind, merge CTA
//   shape (wide), partition fill, weight accumulator (fold), merge strategy
//   (partitioned or global table) and batch sizing (slice margin, host rows
//   before slicing). Concurrent batch lanes are left as set (graph_build).
static double autotune(Ctx& c, unsigned n, unsigned repeats, Ctx::Tune* best) {
  if (n < 8 || n > 19) fail(QPEPS_ERR_RANGE, "autotune probe N must be in [8, 19]");
  repeats = std::max(1u, std::min(repeats, 16u));
  u128 known = 0;
  known_count(n, &known);
  qpeps_options o;
  qpeps_options_default(&o);
  o.collect_layers = 0;
  const Ctx::Tune saved = c.tune;
  Ctx::Tune cur = saved;
  double best_ms = 1e300, best_eager = 1e300;
  auto measure = [&](const Ctx::Tune& t, double cap_ms, uint32_t use_graph) {
    apply_tune(c, t);
    o.use_graph = use_graph;
    double ms = 1e300;
    for (unsigned r = 0; r <= repeats; ++r) {
      Contraction con;
      contract(c, n, o, nullptr, 0, con);
      if (con.count != known) fail(QPEPS_ERR_INVALID, "autotune: count differs from known_count");
      if (r == 0 && con.rs.device_ms > cap_ms) return 1e300;  // far slower than the best: not timed further
      if (r) ms = std::min(ms, con.rs.device_ms);
    }
    return ms;
  };
  using Setter = void (*)(Ctx::Tune&, double);
  struct Dim {
    std::vector<double> values;
    Setter set;
  };
  const std::vector<Dim> dims = {
      {{1, 0, 2, 4}, [](Ctx::Tune& t, double v) { t.scatter_kind = (uint32_t)v; }},
      {{4, 2}, [](Ctx::Tune& t, double v) { t.parents_per_lane = (uint32_t)v; }},
      {{256, 128, 512}, [](Ctx::Tune& t, double v) { t.scatter_block = (uint32_t)v; }},
      {{1, 0}, [](Ctx::Tune& t, double v) { t.merge_kind = (uint32_t)v; }},
      {{2, 0, 1, 3}, [](Ctx::Tune& t, double v) { t.wide_merge = (uint32_t)v; }},
      {{0.83, 0.9, 0.75}, [](Ctx::Tune& t, double v) { t.partition_fill = v; }},
      {{2, 1, 0}, [](Ctx::Tune& t, double v) { t.fold_weights = (uint32_t)v; }},
      {{QPEPS_MERGE_PARTITION, QPEPS_MERGE_HASH}, [](Ctx::Tune& t, double v) { t.merge_auto = (uint32_t)v; }},
      {{5, 3, 8}, [](Ctx::Tune& t, double v) { t.slice_margin = v; }},
      {{1, 2}, [](Ctx::Tune& t, double v) { t.slice_rows = (uint32_t)v; }},
      // Concurrent batch lanes of the graph replay (used with the window and
      // direct scatters only; other scatter kinds replay on one lane).
      {{1, 2}, [](Ctx::Tune& t, double v) { t.batch_lanes = (uint32_t)v; }},
  };
  try {
    best_ms = measure(cur, 1e300, 1);
    best_eager = measure(cur, 1e300, 0);
    for (int pass = 0; pass < 3; ++pass) {
      bool changed = false;
      for (const Dim& d : dims)
        for (double v : d.values) {
          Ctx::Tune t = cur;
          d.set(t, v);
          if (std::memcmp(&t, &cur, sizeof t) == 0) continue;
          const double ms = measure(t, 3.0 * best_ms, 1);
          if (ms >= std::min(0.995 * best_ms, best_ms - 0.005)) continue;
          const double eager = measure(t, 3.0 * best_eager, 0);
          if (eager <= 1.02 * best_eager) {
            best_ms = ms;
            best_eager = std::min(best_eager, eager);
            cur = t;
            changed = true;
          }
        }
      if (!changed) break;
    }
  } catch (...) {
    apply_tune(c, saved);
    throw;
  }
  apply_tune(c, cur);
  *best = cur;
  return best_ms;
}

extern "C" {

const char* qpeps_version(void) { return "qpeps-gb300 0.2.0 (sm_103a)"; }

void qpeps_options_default(qpeps_options* opt) {
  std::memset(opt, 0, sizeof *opt);
  opt->struct_size = sizeof(qpeps_options);
  opt->granularity = QPEPS_GRAIN_ROW;
  opt->merge = QPEPS_MERGE_AUTO;
  opt->symmetry = 1;
  opt->collect_layers = 1;
}

int qpeps_known_count(uint32_t n, qpeps_u128* out) {
  u128 v;
  if (!known_count(n, &v)) return QPEPS_ERR_RANGE;
  *out = to_abi(v);
  return QPEPS_OK;
}

int qpeps_ctx_create(int device, void** ctx_out, char* err, size_t err_len) {
  return guarded(err, err_len, [&] { *ctx_out = ctx_create(device); });
}

void qpeps_ctx_destroy(void* ctx) { ctx_free(static_cast<Ctx*>(ctx)); }

int qpeps_contract_rows(void* ctx, uint32_t n, const qpeps_options* opt, qpeps_result* result, qpeps_layer* layers,
                        uint32_t layers_cap, char* err, size_t err_len) {
  return guarded(err, err_len, [&] {
    if (!ctx || !result) fail(QPEPS_ERR_INVALID, "null context or result");
    Ctx& c = *static_cast<Ctx*>(ctx);
    qpeps_options o = effective_options(opt);
    Contraction con;
    contract(c, n, o, nullptr, 0, con);
    fill_result(c, con, n, result, layers, layers_cap);
  });
}

int qpeps_count(void* ctx, uint32_t n, const uint32_t* prefix, uint32_t k, const qpeps_options* opt,
                qpeps_u128* count_out, qpeps_result* stats_out, char* err, size_t err_len) {
  return guarded(err, err_len, [&] {
    if (!ctx || !count_out) fail(QPEPS_ERR_INVALID, "null context or output");
    if (k > 0 && !prefix) fail(QPEPS_ERR_INVALID, "null prefix with k > 0");
    Ctx& c = *static_cast<Ctx*>(ctx);
    qpeps_options o = effective_options(opt);
    Contraction con;
    contract(c, n, o, prefix, k, con);
    *count_out = to_abi(con.count);
    if (stats_out) fill_result(c, con, n, stats_out, nullptr, 0);
  });
}

int qpeps_count_batch(void* ctx, uint32_t num, const uint32_t* n, const uint32_t* k, const uint32_t* prefix_offset,
                      const uint32_t* prefix_cols, const qpeps_options* opt, qpeps_u128* counts, char* err,
                      size_t err_len) {
  return guarded(err, err_len, [&] {
    if (!ctx || (num && (!n || !k || !counts))) fail(QPEPS_ERR_INVALID, "null argument");
    Ctx& c = *static_cast<Ctx*>(ctx);
    qpeps_options o = effective_options(opt);
    for (uint32_t i = 0; i < num; ++i) {
      Contraction con;
      const uint32_t* pre = k[i] ? prefix_cols + prefix_offset[i] : nullptr;
      contract(c, n[i], o, pre, k[i], con);
      counts[i] = to_abi(con.count);
    }
  });
}

void qpeps_tuning_default(qpeps_tuning* t) { *t = tuning_of(Ctx::Tune{}); }

int qpeps_ctx_get_tuning(void* ctx, qpeps_tuning* out) {
  if (!ctx || !out) return QPEPS_ERR_INVALID;
  Ctx& c = *static_cast<Ctx*>(ctx);
  *out = tuning_of(c.tune);
  out->partition_fill = c.partition_fill;
  return QPEPS_OK;
}

int qpeps_ctx_set_tuning(void* ctx, const qpeps_tuning* t, char* err, size_t err_len) {
  return guarded(err, err_len, [&] {
    if (!ctx || !t) fail(QPEPS_ERR_INVALID, "null context or tuning");
    apply_tune(*static_cast<Ctx*>(ctx), tune_from(*t));
  });
}

int qpeps_probe_append(void* ctx, uint32_t mode, uint64_t candidates, uint32_t parts, uint32_t repeats,
                       double* best_ms, char* err, size_t err_len) {
  return guarded(err, err_len, [&] {
    if (!ctx) fail(QPEPS_ERR_INVALID, "null context");
    if (mode > QPEPS_PROBE_APPEND_PLAIN) fail(QPEPS_ERR_INVALID, "probe mode must be 0..4");
    if (parts == 0 || candidates == 0) fail(QPEPS_ERR_INVALID, "probe needs at least one partition and record");
    Ctx& c = *static_cast<Ctx*>(ctx);
    cuda_check(cudaSetDevice(c.device), "cudaSetDevice");
    const u32 cap = partition_capacity(0);
    const u32 cstride = (parts <= c.tune.spread_cursors_below) ? 8u : 1u;
    const size_t region_bytes = (size_t)parts * cap * 16;
    const size_t cursor_bytes = (size_t)parts * cstride * 4;
    size_t fr = 0, tot = 0;
    cuda_check(cudaMemGetInfo(&fr, &tot), "cudaMemGetInfo");
    if (region_bytes + cursor_bytes + (1u << 20) > fr) fail(QPEPS_ERR_CAPACITY, "probe regions exceed free device memory");
    void* regions = nullptr;
    u32* cursors = nullptr;
    unsigned long long* sink = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    auto release = [&] {
      if (regions) cudaFree(regions);
      if (cursors) cudaFree(cursors);
      if (sink) cudaFree(sink);
      if (e0) cudaEventDestroy(e0);
      if (e1) cudaEventDestroy(e1);
    };
    try {
      cuda_check(cudaMalloc(&regions, region_bytes), "probe regions");
      cuda_check(cudaMalloc(reinterpret_cast<void**>(&cursors), cursor_bytes), "probe cursors");
      cuda_check(cudaMalloc(reinterpret_cast<void**>(&sink), sizeof(unsigned long long)), "probe sink");
      cuda_check(cudaEventCreate(&e0), "event");
      cuda_check(cudaEventCreate(&e1), "event");
      double best = 1e300;
      for (uint32_t r = 0; r <= std::max(1u, repeats); ++r) {
        cuda_check(cudaMemsetAsync(cursors, 0, cursor_bytes, c.stream), "clear probe cursors");
        cuda_check(cudaEventRecord(e0, c.stream), "event");
        cuda_check(launch_append_probe(mode, candidates, parts, cap, regions, cursors, cstride, c.sms, 0x9e37ull * (r + 1),
                                       sink, c.stream),
                   "probe kernel");
        cuda_check(cudaEventRecord(e1, c.stream), "event");
        cuda_check(cudaStreamSynchronize(c.stream), "probe synchronize");
        float ms = 0;
        cuda_check(cudaEventElapsedTime(&ms, e0, e1), "event time");
        if (r) best = std::min(best, (double)ms);
      }
      if (best_ms) *best_ms = best;
    } catch (...) {
      release();
      throw;
    }
    release();
  });
}

int qpeps_autotune(void* ctx, uint32_t n, uint32_t repeats, qpeps_tuning* best, double* best_device_ms, char* err,
                   size_t err_len) {
  return guarded(err, err_len, [&] {
    if (!ctx) fail(QPEPS_ERR_INVALID, "null context");
    Ctx& c = *static_cast<Ctx*>(ctx);
    Ctx::Tune t;
    const double ms = autotune(c, n, repeats, &t);
    if (best) *best = tuning_of(t);
    if (best_device_ms) *best_device_ms = ms;
  });
}

int qpeps_ctx_device_name(void* ctx, char* out, size_t len) {
  if (!ctx || !out || !len) return QPEPS_ERR_INVALID;
  cudaDeviceProp prop;
  if (cudaGetDeviceProperties(&prop, static_cast<Ctx*>(ctx)->device) != cudaSuccess) return QPEPS_ERR_CUDA;
  std::snprintf(out, len, "%s", prop.name);
  return QPEPS_OK;
}

int qpeps_explicit_frontier(void* ctx, uint32_t n, uint32_t order, uint64_t support_limit,
                            qpeps_explicit_result* out, char* err, size_t err_len) {
  return guarded(err, err_len, [&] {
    if (!ctx || !out) fail(QPEPS_ERR_INVALID, "null context or result");
    Ctx& c = *static_cast<Ctx*>(ctx);
    ExplicitRun r;
    explicit_frontier(c, n, order, support_limit, r);
    std::memset(out, 0, sizeof *out);
    out->n = r.n;
    out->order = r.order;
    out->complete = r.complete ? 1 : 0;
    out->merge = r.merge;
    out->count = to_abi(r.complete ? r.count : 0);
    out->elapsed_s = r.elapsed;
    out->peak_states = r.peak_states;
    out->peak_open_bonds = r.peak_open_bonds;
    out->tensor_entries_examined = to_abi(r.examined);
    out->tensor_entries_accepted = to_abi(r.accepted);
    out->contracted_sites = r.contracted_sites;
    out->peak_rss_bytes = c.peak_pool_bytes;
    out->gpu_launches = r.launches;
    out->device_ms = r.device_ms;
  });
}

int qpeps_certify_c(const uint32_t* legs, const uint64_t* values, uint32_t len, char* err, size_t err_len) {
  return guarded(err, err_len, [&] {
    std::vector<CEntryH> c;
    for (uint32_t i = 0; i < len; ++i) c.push_back(CEntryH{legs[i], values[i]});
    certify_c(c);
  });
}

void qpeps_serve_config_default(qpeps_serve_config* cfg) {
  std::memset(cfg, 0, sizeof *cfg);
  cfg->struct_size = sizeof(qpeps_serve_config);
  cfg->max_slots = kServeMaxSlots;
  cfg->use_cache = 1;
}

int qpeps_serve_open(int device, const qpeps_serve_config* cfg, void** server_out, char* err, size_t err_len) {
  return guarded(err, err_len, [&] {
    if (!server_out) fail(QPEPS_ERR_INVALID, "null server output");
    Server* sv = new Server();
    try {
      qpeps_serve_config_default(&sv->cfg);
      if (cfg) {
        if (cfg->struct_size != sizeof(qpeps_serve_config)) fail(QPEPS_ERR_INVALID, "qpeps_serve_config.struct_size mismatch");
        sv->cfg = *cfg;
      }
      if (sv->cfg.max_slots == 0 || sv->cfg.max_slots > kServeMaxSlots) sv->cfg.max_slots = kServeMaxSlots;
      sv->device = device;
      if (sv->cfg.large_workers == 0) sv->cfg.large_workers = 2;
      if (sv->cfg.large_workers > 8) fail(QPEPS_ERR_INVALID, "large_workers must be at most 8");
      sv->batch = ctx_create(device);
      for (uint32_t w = 0; w < sv->cfg.large_workers; ++w) sv->large.push_back(ctx_create(device));
      size_t fr = 0, tot = 0;
      cuda_check(cudaMemGetInfo(&fr, &tot), "cudaMemGetInfo");
      if (!sv->cfg.batch_budget_bytes) sv->cfg.batch_budget_bytes = (uint64_t)(fr * 0.25);
      if (!sv->cfg.large_budget_bytes) sv->cfg.large_budget_bytes = (uint64_t)(fr * 0.60);
      // Requests estimated above 16 M frontier states run alone on the large
      // context: a shared step costs as much as its largest member's row, so
      // keeping big requests out of the batch keeps its steps (and the small
      // requests' latency) short.
      if (!sv->cfg.large_threshold_states)
        sv->cfg.large_threshold_states = std::min<uint64_t>(
            16ull << 20, (uint64_t)((double)sv->cfg.batch_budget_bytes / (2.4 * 16.0) / 4.0));
      sv->t_batch = std::thread(serve_thread_main, std::ref(*sv), false, (size_t)0);
      for (size_t w = 0; w < sv->large.size(); ++w)
        sv->t_large.emplace_back(serve_thread_main, std::ref(*sv), true, w);
    } catch (...) {
      {
        std::lock_guard<std::mutex> lk(sv->mu);
        sv->stop = true;
      }
      sv->cv.notify_all();
      if (sv->t_batch.joinable()) sv->t_batch.join();
      for (std::thread& t : sv->t_large)
        if (t.joinable()) t.join();
      if (sv->batch) ctx_free(sv->batch);
      for (Ctx* c : sv->large) ctx_free(c);
      delete sv;
      throw;
    }
    *server_out = sv;
  });
}

int qpeps_serve_submit(void* server, uint32_t n, const uint32_t* prefix, uint32_t k, uint64_t tag, char* err,
                       size_t err_len) {
  return guarded(err, err_len, [&] {
    Server* sv = static_cast<Server*>(server);
    if (!sv) fail(QPEPS_ERR_INVALID, "null server");
    if (n < 1 || n > 19) fail(QPEPS_ERR_RANGE, "serving supports 1 <= N <= 19");
    if (k > n || (k && !prefix)) fail(QPEPS_ERR_RANGE, "prefix longer than the board");
    ServeRequest r;
    r.tag = tag;
    r.n = n;
    r.prefix.assign(prefix, prefix + k);
    for (uint32_t c : r.prefix)
      if (c >= n) fail(QPEPS_ERR_RANGE, "prefix column out of range");
    r.t_submit = ServeClock::now();
    r.cache_key = serve_cache_key(n, r.prefix);
    r.est_states = serve_estimate(n, k);
    std::unique_lock<std::mutex> lk(sv->mu);
    if (!sv->fatal.empty()) fail(QPEPS_ERR_CUDA, "server stopped: " + sv->fatal);
    sv->stats.submitted += 1;
    if (sv->cfg.use_cache) {
      auto it = sv->cache.find(r.cache_key);
      if (it != sv->cache.end()) {
        const u128 count = it->second;
        sv->stats.cache_hits += 1;
        lk.unlock();
        serve_complete(*sv, tag, n, k, count, QPEPS_OK, 2, r.t_submit, r.t_submit);
        return;
      }
      auto in = sv->inflight.find(r.cache_key);
      if (in != sv->inflight.end()) {
        in->second.push_back(ServeWaiter{tag, n, k, r.t_submit});
        sv->stats.coalesced += 1;
        return;
      }
      sv->inflight[r.cache_key];
    }
    if (r.est_states > (double)sv->cfg.large_threshold_states)
      sv->q_large.push_back(std::move(r));
    else
      sv->q_small.push_back(std::move(r));
    lk.unlock();
    sv->cv.notify_all();
  });
}

int qpeps_serve_poll(void* server, qpeps_serve_completion* out, uint32_t cap, uint32_t* got, uint32_t wait_ms) {
  Server* sv = static_cast<Server*>(server);
  if (!sv || !got) return QPEPS_ERR_INVALID;
  std::unique_lock<std::mutex> lk(sv->mu);
  if (sv->done.empty() && wait_ms)
    sv->cv_done.wait_for(lk, std::chrono::milliseconds(wait_ms), [&] { return !sv->done.empty() || !sv->fatal.empty(); });
  const uint32_t m = (uint32_t)std::min<size_t>(cap, sv->done.size());
  for (uint32_t i = 0; i < m; ++i) out[i] = sv->done[i];
  sv->done.erase(sv->done.begin(), sv->done.begin() + m);
  *got = m;
  return sv->fatal.empty() ? QPEPS_OK : QPEPS_ERR_CUDA;
}

int qpeps_serve_error(void* server, char* err, size_t err_len) {
  Server* sv = static_cast<Server*>(server);
  if (!sv) return QPEPS_ERR_INVALID;
  std::lock_guard<std::mutex> lk(sv->mu);
  set_err(err, err_len, sv->fatal);
  return sv->fatal.empty() ? QPEPS_OK : sv->fatal_code;
}

int qpeps_serve_stats_get(void* server, qpeps_serve_stats* out) {
  Server* sv = static_cast<Server*>(server);
  if (!sv || !out) return QPEPS_ERR_INVALID;
  std::lock_guard<std::mutex> lk(sv->mu);
  *out = sv->stats;
  return QPEPS_OK;
}

void qpeps_serve_close(void* server) {
  Server* sv = static_cast<Server*>(server);
  if (!sv) return;
  {
    std::lock_guard<std::mutex> lk(sv->mu);
    sv->stop = true;
  }
  sv->cv.notify_all();
  if (sv->t_batch.joinable()) sv->t_batch.join();
  for (std::thread& t : sv->t_large)
    if (t.joinable()) t.join();
  cudaSetDevice(sv->device);
  if (sv->batch) {
    buf_release(*sv->batch, sv->slot_buf);
    ctx_free(sv->batch);
  }
  for (Ctx* c : sv->large) ctx_free(c);
  delete sv;
}

}  // extern "C"
