// Internal interface between the host engine and the CUDA kernels.
#pragma once

#include <cstddef>
#include <cstdint>

#include <cuda_runtime.h>

namespace qpeps {

// Explicit local tensor C in the form the site kernel reads from constant
// memory: for each 4-bit input signature (column_in | row_in<<1 |
// diag_dr_in<<2 | diag_dl_in<<3, src/lib.rs:152-157) the matching entries'
// outputs (column_out | row_out<<1 | diag_dr_out<<2 | diag_dl_out<<3) and
// their values reduced modulo each residue prime.
struct CTableDev {
  uint32_t count[16];
  uint32_t out[16][4];
  uint32_t value_mod[16][4][4];
};

// Device view of one boundary buffer (structure of arrays).
struct FrontierView {
  void* keys;          // u64[cap] or u128[cap]
  uint32_t* res;       // u32[R][cap]
  uint64_t cap;        // entries per residue plane
};

// Per-step device scalars (one cache line each to avoid false sharing).
struct StepScalars {
  unsigned long long terms;          // successor terms generated
  unsigned long long out_count;      // entries written by compaction
  unsigned long long weight_sum[4];  // sum of residues of written entries
  unsigned long long final_sum[4];   // sum of residues of entries with all columns set
  unsigned long long final_states;   // entries with all columns set
  unsigned int error;                // ErrorBits
  unsigned int next_terms_ok;        // 1: the merge counted next_terms (fixed-layout row merges)
  unsigned long long sitewise_examined;  // row count: C entries the reference's per-parent sitewise
                                         // row kernel matches over the input (sitewise_entries())
  unsigned long long plan_units;         // class-grouped partitions: units of the step's plan (graph replay)
  unsigned long long next_terms;         // successor terms of the written boundary at the next row
  unsigned long long t_scatter, t_merge, t_end; // queued steps: start of each kernel, end of the second
                                                // (global timer, ns; 0: the next step's start)
  unsigned long long row_terms;          // queued site steps that end a row: successor terms of its boundary
};

// Sizes of a queued step: read on the device from the scalars the step before
// left, so that the host queues a chain of steps without waiting for each. A
// step that does not fit (or follows one that failed) raises a flag, and its
// kernels and those after it return at once; its input boundary stands.
struct StepSource {
  const StepScalars* prev = nullptr;  // nullptr: the host passes the sizes
  double mean = 0;                    // planned candidates per partition
  uint32_t parts_cap = 0;             // partitions the regions hold
  uint32_t spread = 1;                // partitions of a small step, one for each merge CTA the device holds
  uint64_t limit = ~0ull;             // entries a boundary may have: the chain ends behind a larger one

  // Partitions of a step. A small step takes more of them than its candidates
  // fill: with 60 partitions for 100 K candidates the cursor atomics queue up
  // 1,600 deep on each cursor, and most merge CTAs idle. At least 64 candidates
  // each.
  __host__ __device__ uint64_t partitions(uint64_t terms) const {
    const uint64_t full = (uint64_t)((double)terms / mean) + 1, wide = terms / 64 + 1;
    const uint64_t small = wide < spread ? wide : spread;
    return full > small ? full : small;
  }
};

// Launch a kernel of a chain so that it may start while the kernel before it
// in the stream finishes (it waits for that kernel's results itself).
template <typename... Params, typename... Args>
inline cudaError_t launch_overlapped(void (*kernel)(Params...), unsigned grid, unsigned block, size_t smem,
                                     cudaStream_t stream, bool overlapped, Args... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = overlapped ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

// The same for a queued step on the global table: the slots follow from the
// terms the step before counted, and the compaction leaves the table empty.
struct TableSource {
  const StepScalars* prev = nullptr;  // nullptr: the host passes the sizes
  uint64_t slots_cap = 0;             // slots the table holds (a power of two)
  bool last = false;                  // the chain's last step: its compaction stamps its end

  // A small step's time is its longest probe sequence, a trip to L2 each: at
  // loads up to 1/2, 30 K terms took 18 us, at up to 1/8 7 us. Larger steps
  // are bound by reading the table back.
  __host__ __device__ uint64_t slots(uint64_t terms) const {
    const uint64_t want = terms <= 65536 ? 8 * terms : terms <= 262144 ? 4 * terms : 2 * terms;
    uint64_t s = 1024;
    while (s < want) s <<= 1;
    return s;
  }
};

struct LaunchCfg {
  int key_bits;  // 64 or 128
  int residues;  // 1..4
  int threads;   // block size of the expand kernel
  int sms;       // SM count of the device
};

// All launchers enqueue on `stream` and return cudaGetLastError().
cudaError_t upload_c_table(const CTableDev& table, cudaStream_t stream);

// Sum over entries of popcount(free columns): the row step's successor count.
cudaError_t launch_row_count(const LaunchCfg& cfg, const FrontierView& in, uint64_t n_in, unsigned n,
                             StepScalars* scalars, cudaStream_t stream);

// Fused compiled-row expansion + global-table insertion.
cudaError_t launch_row_expand_insert(const LaunchCfg& cfg, const FrontierView& in, uint64_t n_in, unsigned n,
                                     void* table, uint64_t table_slots, StepScalars* scalars, cudaStream_t stream);

// Number of explicit-C terms produced at site `site` (mid-row key layout).
cudaError_t launch_site_count(const LaunchCfg& cfg, const FrontierView& in, uint64_t n_in, unsigned n, unsigned site,
                              StepScalars* scalars, cudaStream_t stream);

// Explicit-C site update (one launch per site) + global-table insertion.
cudaError_t launch_site_expand_insert(const LaunchCfg& cfg, const FrontierView& in, uint64_t n_in, unsigned n,
                                      unsigned site, void* table, uint64_t table_slots, StepScalars* scalars,
                                      cudaStream_t stream, const TableSource& queued = TableSource{});

// Table -> boundary buffer; accumulates weight sums and final (v1) sums. A
// queued step's compaction also empties the table and counts the next site's
// terms (`next_site` in [0, n); at 0 the successor terms and sitewise entries
// of the row that follows, too).
cudaError_t launch_compact(const LaunchCfg& cfg, void* table, uint64_t table_slots, const FrontierView& out,
                           unsigned n, bool write_out, StepScalars* scalars, cudaStream_t stream,
                           const TableSource& queued = TableSource{}, unsigned next_site = 0);

// Bytes per table slot for a key width / residue count.
size_t slot_bytes(int key_bits, int residues);

// Explicit-C generic site frontier: one site step. The boundary key holds the
// values of the open virtual bonds (bit i = i-th open bond in increasing bond
// id). The bonds that stay open move to their new positions by a few masked
// shifts (the map is monotone), and every C entry allowed at the site becomes
// a transition: a key matching (req_mask, req_value) on the bonds the site
// closes yields the moved key OR `added` (the values of the bonds it opens).
constexpr int kFrontierMaxRuns = 16;
constexpr int kFrontierMaxTrans = 17;
struct FrontierStepDev {
  uint32_t n_runs, n_trans;
  int32_t run_shift[kFrontierMaxRuns];  // > 0 left, < 0 right
  unsigned __int128 run_mask[kFrontierMaxRuns];
  unsigned __int128 req_mask[kFrontierMaxTrans], req_value[kFrontierMaxTrans], added[kFrontierMaxTrans];
};

cudaError_t upload_frontier_step(const FrontierStepDev& step, cudaStream_t stream);

// Every (boundary entry, matching transition) successor into the u128-keyed
// global table; `scalars->terms` receives the number of matches.
cudaError_t launch_frontier_expand_insert(const LaunchCfg& cfg, const FrontierView& in, uint64_t n_in, void* table,
                                          uint64_t table_slots, StepScalars* scalars, cudaStream_t stream);

// Partitioned merge (u64 keys): `parts` hash partitions of `cap` candidate
// slots each.
struct PartitionCfg {
  int residues;
  int sms;
  uint32_t parts;
  uint32_t cap;
  int merge_blocks_per_sm;
  uint32_t cursor_stride = 1;     // u32 slots between partition cursors (1 or 8)
  uint32_t parents_per_lane = 2;  // scatter: parents per lane per iteration (2 or 4)
  uint32_t wide = 0;              // merge CTA shape: 0 = 512 threads, 4096-slot table, 2048 candidates,
                                  // two CTAs per SM; 1 = 1024 threads, 8192 slots, 4096 candidates,
                                  // one CTA per SM (R <= 2 only: the table is 8 KiB x (8 + 8R) bytes);
                                  // 2 = 256 threads, 2048 slots, 1024 candidates, four CTAs per SM (R <= 2)
  uint32_t scatter_kind = 1;      // scatter: 0 = shuffle search for each successor's parent,
                                  // 1 = per-warp shared-memory candidate window,
                                  // 2 = two-level (coarse buckets, then partitions; runs staged and
                                  //     ordered in shared memory), where two_level_plan() accepts the step
  uint32_t merge_kind = 1;        // merge: 0 = ballot/scan compaction over the whole table,
                                  // 1 = claim list + first-claimant stores (three phases)
  uint32_t fold = 0;              // merge_kind 1, R = 2, one 64-bit accumulator plane:
                                  // 1 = CRT-folded residues, 2 = the planes hold an exact weight's
                                  // low and high words (both exact only when N! < p0 * p1, N <= 20)
  uint32_t key_bits = 64;         // 128: wide-key scatter and merge (32-byte candidates, `cap` = 1024)
  uint32_t count_next = 1;        // fixed-layout row merges: count the next row's successor terms
  uint32_t scatter_block = 256;   // one-level scatters: threads per CTA (128, 256 or 512; 256 for R > 2)
  uint32_t merge_regs = 0;        // merge_kind 1, fixed layout: first claimants write their entries from
                                  // registers (no slot list in shared memory)
  uint32_t tl_nb = 0;             // two-level scatter: coarse buckets (0 = one-level scatter)
  uint32_t tl_p2 = 0;             // two-level scatter: partitions per bucket (parts = tl_nb * tl_p2)
  uint64_t tl_bcap = 0;           // two-level scatter: candidate slots per bucket
  StepSource queued;              // one-level scatters and claim-list merges: sizes come from the device
                                  // (`parts` and n_in bound the grids); the merge clears the cursors it reads
};

size_t candidate_bytes(int residues);
// Partitioned merge with 128-bit keys: candidate slots per partition (1024),
// and its scatter and merge (window scatter; claim-list merge over residue
// planes with a 2048-slot table of 128-bit keys).
uint32_t wide_key_partition_capacity();
cudaError_t launch_wide_partition_scatter(const PartitionCfg& pc, const FrontierView& in, uint64_t n_in, unsigned n,
                                          void* regions, uint32_t* cursors, StepScalars* scalars, cudaStream_t stream);
// With n > 0 (row keys) the merge counts the written boundary's successor
// terms at the next row; with n = 0 and `next_step` (explicit-C bond keys, a
// device copy of the next site step) it counts the boundary's matches there.
// Either count lands in scalars->next_terms with next_terms_ok set.
cudaError_t launch_wide_partition_merge(const PartitionCfg& pc, const void* regions, const uint32_t* cursors,
                                        const FrontierView& out, unsigned n, bool write_out, StepScalars* scalars,
                                        cudaStream_t stream, const FrontierStepDev* next_step = nullptr);
// Access-pattern probe (qpeps_probe_append): `total` pseudo-random 16-byte
// records into `parts` partitions of `cap` slots (cap a power of two) by mode
// 0 append (cursor atomic + store), 1 store only, 2 atomic only, 3 stream.
cudaError_t launch_append_probe(uint32_t mode, uint64_t total, uint32_t parts, uint32_t cap, void* regions,
                                uint32_t* cursors, uint32_t cursor_stride, int sms, uint64_t seed,
                                unsigned long long* sink, cudaStream_t stream);
// Explicit-C frontier step through the same 128-bit partitions: the number of
// (boundary entry, matching transition) pairs into `scalars->terms`, and
// every such pair as one candidate (merged by launch_wide_partition_merge
// with n = 0). Keys must not set all 128 bits (at most 127 open bonds).
cudaError_t launch_frontier_count(const FrontierView& in, uint64_t n_in, const FrontierStepDev& step, int sms,
                                  StepScalars* scalars, cudaStream_t stream);
// (`step`: its copy on the device, at most kFrontierMaxRuns runs and
// kFrontierMaxTrans transitions.)
cudaError_t launch_frontier_partition_scatter(const PartitionCfg& pc, const FrontierView& in, uint64_t n_in,
                                              const FrontierStepDev* step, void* regions, uint32_t* cursors,
                                              StepScalars* scalars, cudaStream_t stream);
// Candidate slots per partition for a merge shape (PartitionCfg::wide).
uint32_t partition_capacity(uint32_t wide = 0);
// Whether the wide merge shape is available for a residue count.
bool wide_merge_supported(int residues);

// Two-level scatter plan for a step of `terms` successors and at least
// `parts` partitions: sets tl_nb, tl_p2, tl_bcap and parts (= tl_nb * tl_p2,
// rounded up from `parts`). False where it does not apply (more than 16-byte
// candidates, or more partitions than its bins address).
bool two_level_plan(uint64_t terms, uint32_t parts, int residues, PartitionCfg* pc);
// Its scratch follows the partition cursors (parts x 4 x cursor_stride bytes,
// rounded up to 256) in the same allocation: bucket cursors, then bucket slots.
size_t two_level_cursor_bytes(const PartitionCfg& pc);
size_t two_level_extra_bytes(const PartitionCfg& pc);

cudaError_t launch_partition_scatter(const PartitionCfg& pc, const FrontierView& in, uint64_t n_in, unsigned n,
                                     void* regions, uint32_t* cursors, StepScalars* scalars, cudaStream_t stream);

// Class-grouped partitions (scatter_kind 3, 16-byte candidates). A
// candidate's class is its columns and the t outermost diagonal pairs; classes
// hash into 2^lg buckets (four sibling classes, equal but for pair 0, in
// consecutive buckets), and a plan maps each bucket to a run of "units"
// (merge partitions of `cap` slots) from a sampled histogram.
struct UnitClassPlan {
  unsigned n;   // board size
  unsigned t;   // window pairs (0: columns only); t <= n / 2
  unsigned lg;  // log2 of the bucket count (>= 3 when t >= 1)
};
struct UnitPlanArgs {
  uint32_t lg;      // log2 of the bucket count
  uint32_t sample;  // one parent block of 512 in `sample` is counted
  uint64_t target;  // planned candidates per unit
};
struct UnitPlanTotals {
  unsigned long long small_units;  // units of packed small buckets (unit ids [0, small_units))
  unsigned long long units;        // all units (the merge's partition count)
  unsigned long long small_e;      // estimated candidates of the packed buckets
  unsigned long long pad;
};
struct UnitPlanDev {
  const uint2* table = nullptr;         // per bucket {first unit, units}
  UnitPlanTotals* totals = nullptr;     // device
};
bool unit_scatter_supported(int residues);
// Device scratch of a plan with 2^lg buckets (histogram, table, scan partials, totals).
size_t unit_plan_scratch_bytes(uint32_t lg);
// Sampled histogram of the step's successors and the bucket -> units table;
// the unit count lands in out->totals (device) for the host to read.
cudaError_t launch_unit_plan(const FrontierView& in, uint64_t n_in, const UnitClassPlan& c, const UnitPlanArgs& a,
                             void* scratch, int sms, cudaStream_t stream, UnitPlanDev* out,
                             StepScalars* scalars = nullptr);
cudaError_t launch_unit_scatter(const PartitionCfg& pc, const FrontierView& in, uint64_t n_in,
                                const UnitClassPlan& c, const uint2* table, void* regions, uint32_t* cursors,
                                StepScalars* scalars, cudaStream_t stream);

cudaError_t launch_partition_merge(const PartitionCfg& pc, const void* regions, const uint32_t* cursors,
                                   const FrontierView& out, unsigned n, bool write_out, StepScalars* scalars,
                                   cudaStream_t stream);



// Rows [row, n) of a few seed states in one CTA, the boundary in shared memory
// (qpeps_resident_kernels.cu): u64 keys, exact 64-bit weights. out[i] takes row
// row + i's scalars (out_count, next_terms, weight_sum[0], final_sum[0],
// final_states; the start and end stamps of the whole in out[0].t_scatter and
// the last row's t_merge); `out` may be pinned host memory. A boundary that
// outgrows the CTA stops it with kErrCapacity in out[0].error.
constexpr uint32_t kResidentSeeds = 24;
struct ResidentArgs {
  uint32_t n, row, count;
  uint64_t key[kResidentSeeds];
  uint64_t weight[kResidentSeeds];
  StepScalars* out;
};
uint32_t resident_capacity();
cudaError_t launch_resident_rows(const ResidentArgs& a, cudaStream_t stream);

// Column-grouped row step (qpeps_group_kernels.cu): exact weights, the
// boundary grouped by column set.
constexpr unsigned kGroupMaxN = 18;  // widest board whose 2 N - 2 live diagonal bits fit 32 but for two

struct GroupDir {   // per column set, in colex rank order
  uint32_t base;    // unit of its first bucket
  uint32_t bits;    // log2 of its buckets
  uint32_t total;   // entries
  uint32_t pad;
};

// One row's scalars (device; zero before the row's plan runs).
struct GroupRow {
  unsigned long long out_count;   // merged entries
  unsigned long long alloc;       // output entries handed out in blocks (counted past the buffer's end too)
  unsigned long long next_terms;  // their successor terms at the next row
  unsigned long long weight_sum, weight_max;
  unsigned long long t_plan, t_pull, t_end;  // global timer, ns
  uint32_t units, next_unit, pieces, ctas_done;
  uint32_t error;
  float merge_rate;  // merged entries per term
};

struct GroupSide {    // a boundary
  uint32_t* keys;     // [cap]
  uint32_t* lo;       // [cap] weights
  uint64_t cap;       // < 2^32
  GroupDir* gdir;     // [C(n, m)]
  uint4* udir;        // [unit_cap] {first entry, entries of quarters 0 | 1 << 16, 2 | 3 << 16,
                      //  further piece or 0}
  uint32_t unit_cap;
};

struct GroupStepArgs {
  GroupSide in, out;
  const GroupRow* prev;  // the input boundary's scalars
  GroupRow* row;
  uint2* units;          // [unit_cap] {columns | bits << 24, bucket}
  const uint32_t* binomials;  // [(kGroupMaxN + 2)^2]
  uint32_t n, m;         // board size, columns set after the row
  uint32_t rm;           // top u bits implied by the bucket
  uint32_t max_bits;
  uint32_t write_out;
  uint32_t block;        // output entries a CTA takes at a time, at least a table's
  float target;          // expected outputs of a unit, at most
  float share;           // and at most this share of the row's
};

float group_unit_target();
float group_unit_share(int sms);
// Output block of a boundary of about `states` entries, and the entries its
// buffer needs with the blocks' unused ends.
uint32_t group_block(double states, int sms);
uint64_t group_capacity(double states, int sms);
cudaError_t launch_group_plan(const GroupStepArgs& a, uint32_t groups, cudaStream_t stream);
cudaError_t launch_group_pull(const GroupStepArgs& a, int sms, cudaStream_t stream);
// One bucket of the seed boundary, its entries in place: the directories.
struct GroupSeedUnit {
  uint32_t first, unit;
  uint32_t quarters01, quarters23;  // entries by quarter, 16 bits each
  uint32_t rank, bits, total;       // the group's entry, with its first bucket (total > 0)
};
cudaError_t launch_group_seed(const GroupSeedUnit* list, uint32_t count, const GroupSide& side, cudaStream_t stream);

// Serving (slotted keys, exact 64-bit weights in two planes): scatter and merge
// of a boundary shared by requests of different board sizes. slot_mask[s] is
// the board mask of the request in slot s; finished boards are summed into
// slot_final[s * 4] and leave the boundary. One pair of kernels: the window
// scatter and the exact claim-list merge in its small shape; of `pc` only the
// partitions, their cursors' stride and the queued sizes count.
cudaError_t launch_serve_scatter(const PartitionCfg& pc, const FrontierView& in, uint64_t n_in,
                                 const uint64_t* slot_mask, void* regions, uint32_t* cursors, StepScalars* sc,
                                 cudaStream_t stream);
cudaError_t launch_serve_merge(const PartitionCfg& pc, const void* regions, const uint32_t* cursors,
                               const FrontierView& out, const uint64_t* slot_mask, unsigned long long* slot_final,
                               StepScalars* sc, cudaStream_t stream);

// Slice-tail kernel control block (device memory). Row statistics per tail
// row q (row0 + q): [0] input states, [1] output states, [2] successor terms,
// [3 + r] output weight residue r.
constexpr int kTailMaxRows = 32;
constexpr int kTailRowFields = 7;
struct TailControl {
  unsigned long long next_item;
  unsigned long long overflow_count;
  unsigned long long overflow_cap;
  uint64_t* overflow_items;
  unsigned long long final_sum[4];
  unsigned long long row_acc[kTailMaxRows][kTailRowFields];
  unsigned int error;
  unsigned int pad[3];
};

// Contract rows [row0, n) of every boundary entry independently, one warp per
// entry, in shared memory. Entries whose frontier exceeds tail_capacity()
// states are listed in ctl->overflow_items.
uint32_t tail_capacity();
cudaError_t launch_gather_entries(int residues, const FrontierView& in, const uint64_t* idx, uint64_t m,
                                  uint64_t* out_keys, uint32_t* out_res, int sms, cudaStream_t stream);
cudaError_t launch_slice_tail(int residues, const FrontierView& in, uint64_t n_items, unsigned n, unsigned row0,
                              TailControl* ctl, int sms, cudaStream_t stream);

}  // namespace qpeps
