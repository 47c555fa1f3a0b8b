// Column-grouped row step (exact weights, u64 boards up to N = 18).
//
// The boundary is held grouped by its column set C: the N - row children
// groups of a parent group are known before a single key is read, so the row
// step runs the other way round from the partitioned merge. One CTA owns a
// piece of an output group (a "unit"), reads the parents of its C-groups
// C \ {c}, keeps those whose diagonals are free at c, and merges the
// successors in a shared-memory table. Nothing is scattered and no candidate
// is ever written to memory: the step reads 4-byte keys (each parent once per
// free column, from L2 or in coalesced runs from HBM), the weights of the
// parents that match, and writes the merged entries once.
//
// Inside a group the column set is implicit and only the 2N - 2 live diagonal
// bits are stored (32 bits up to N = 17; at N = 18 the two top bits are
// implied by the bucket, see below). A group is cut into 2^b buckets by the
// top b bits of the up-moving diagonal u, and each bucket into quarters by the
// next two. A row step moves u up by one, so the outputs of bucket beta come
// from the parents whose top bits are x beta (x in {0, 1}, beta with the new
// queen's bit cleared): whole buckets, halves or quarters of the parents' groups, in
// contiguous runs, never a filtered scan of a whole group (a parent group cut
// more coarsely than the output is read with the missing bits as a filter).
//
// What bounds it: instruction issue (N = 16's largest row, 119 M candidates:
// about 400 warp instructions per 32 candidates at 2.5 a cycle and SM, half of
// them the insertions; DRAM at 13 %). GB300, device ms of a board, partitioned
// rows against these: N = 15 2.43 / 1.96, N = 16 15.6 / 8.3, N = 17 117 / 53.4,
// N = 18 (nine batches) 821 / 481. The partitioned rows' time is their scatter,
// a random 16-byte append a candidate at 42 to 48 G/s, and a merge on top of it.
#include <cuda_runtime.h>

#include <algorithm>

#include "qpeps_device.cuh"
#include "qpeps_internal.h"

namespace qpeps {

namespace {

constexpr u32 kFull = 0xffffffffu;
constexpr int kBinDim = kGroupMaxN + 2;

template <int I>
struct Items {
  static constexpr int value = I;
};
struct TrueTag {
  static constexpr bool value = true;
};
struct FalseTag {
  static constexpr bool value = false;
};

__device__ __forceinline__ u32 lt_mask() {
  u32 m;
  asm("mov.u32 %0, %lanemask_lt;" : "=r"(m));
  return m;
}

// Binomials into shared memory: s_bin[n * kBinDim + k].
__device__ __forceinline__ void fill_binomials(u32* s_bin, const u32* __restrict__ bin) {
  for (int i = threadIdx.x; i < kBinDim * kBinDim; i += blockDim.x) s_bin[i] = bin[i];
}

// Expected merged outputs of a unit per pair (parent, column) it reads: the
// row's exact match rate times the last row's merge rate (both change slowly
// from row to row).
__device__ __forceinline__ float out_rate(const GroupRow* __restrict__ prev, unsigned n, unsigned m) {
  const float pairs = (float)prev->out_count * (float)(n - m + 1);
  const float match = pairs > 0.f ? (float)prev->next_terms / pairs : 0.f;
  return match * prev->merge_rate;
}

// ---- plan: buckets per output group ----------------------------------------
//
// One thread per output group: sums its parents' sizes, cuts it into 2^b
// buckets of about `target` expected outputs and takes a run of units for
// them. Groups without parents get none.
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) group_plan_kernel(GroupStepArgs a) {
  __shared__ u32 s_bin[kBinDim * kBinDim];
  __shared__ u32 s_warp[BLOCK / 32];
  __shared__ u32 s_base;
  const GroupRow* prev = a.prev;
  GroupRow* row = a.row;
  if (prev->error) {
    if (blockIdx.x == 0 && threadIdx.x == 0) row->error = kErrSkipped;
    return;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) row->t_plan = global_ns();
  fill_binomials(s_bin, a.binomials);
  __syncthreads();
  const unsigned n = a.n, m = a.m;
  const float rate = out_rate(prev, n, m);
  const u32 groups = s_bin[n * kBinDim + m];
  const u32 g = blockIdx.x * BLOCK + threadIdx.x;
  u32 units = 0, b = a.rm, cols = 0;
  if (g < groups) {
    // Colex unranking: the i-th element (1-based, from the top) is the largest
    // c with C(c, i) <= remaining rank.
    u32 r = g;
    int c = (int)n - 1;
    for (int i = (int)m; i >= 1; --i) {
      while (s_bin[c * kBinDim + i] > r) --c;
      r -= s_bin[c * kBinDim + i];
      cols |= 1u << c;
      --c;
    }
    // rank(C \ {c_j}) = sum_{i<j} C(c_i, i) + sum_{i>j} C(c_i, i - 1)
    u32 below = 0, above = 0;
    for (u32 left = cols, i = 1; left; left &= left - 1, ++i) above += s_bin[(__ffs(left) - 1) * kBinDim + i - 1];
    u64 pairs = 0;
    u32 deepest = 0;
    for (u32 left = cols, i = 1; left; left &= left - 1, ++i) {
      const u32 ci = __ffs(left) - 1;
      above -= s_bin[ci * kBinDim + i - 1];
      const GroupDir d = a.in.gdir[below + above];
      below += s_bin[ci * kBinDim + i];
      if (d.total) {
        pairs += d.total;
        deepest = max(deepest, d.bits);
      }
    }
    if (pairs) {
      const float est = (float)pairs * rate;
      // A bucket reads at most two buckets a side of a parent cut two bits
      // more finely, which bounds the segment list.
      if (deepest > 2 && deepest - 2 > b) b = deepest - 2;
      // A row with few outputs is cut finely enough for eight units a CTA.
      const float share = (float)prev->next_terms * prev->merge_rate * a.share;
      const float target = fminf(a.target, fmaxf(share, 64.f));
      while (b < a.max_bits && est > target * (float)(1u << b)) ++b;
      units = 1u << b;
    }
  }
  // Units in group order: block scan, one atomic a block.
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  u32 incl = units;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const u32 t = __shfl_up_sync(kFull, incl, d);
    if (lane >= d) incl += t;
  }
  if (lane == 31) s_warp[wid] = incl;
  __syncthreads();
  if (threadIdx.x == 0) {
    u32 t = 0;
    for (int w = 0; w < BLOCK / 32; ++w) {
      const u32 x = s_warp[w];
      s_warp[w] = t;
      t += x;
    }
    s_base = t ? atomicAdd(&row->units, t) : 0u;
  }
  __syncthreads();
  const u32 base = s_base + s_warp[wid] + incl - units;
  const bool fits = base + units <= a.out.unit_cap;
  if (units && !fits) atomicOr(&row->error, kErrOverflow);
  if (g < groups) a.out.gdir[g] = GroupDir{base, b, 0u, 0u};
  if (fits)
    for (u32 q = 0; q < units; ++q) {
      a.units[base + q] = make_uint2(cols | (b << 24), q);
      a.out.udir[base + q] = make_uint4(0u, 0u, 0u, 0u);
    }
}

// ---- pull: one unit per CTA at a time ---------------------------------------

// (Both limits can be set lower when this file is compiled: no board of up to 18
// columns passes them, and what happens beyond them has to be run somewhere.)
#ifndef QPEPS_GROUP_MAX_SEG
#define QPEPS_GROUP_MAX_SEG 128
#endif
#ifndef QPEPS_GROUP_WEIGHT_BITS
#define QPEPS_GROUP_WEIGHT_BITS 32
#endif
constexpr int kMaxSeg = QPEPS_GROUP_MAX_SEG;
constexpr int kWeightBits = QPEPS_GROUP_WEIGHT_BITS;
static_assert(kMaxSeg <= 128 && kWeightBits <= 32, "a run's segment takes 8 bits, a weight one word");
constexpr int kRuns = 144;  // runs of a unit besides one per segment
constexpr u32 kBatch = 128; // matches a warp inserts at a time

// What the producer warp hands to the others for one unit.
struct PullUnit {
  u32 test_mask[kMaxSeg], test_value[kMaxSeg], added[kMaxSeg];  // per segment; `added`: bits of the table key
  uint2 run[kRuns + kMaxSeg];       // {first entry, entries | segment << 24}
  u32 valid, cols, b, beta, unit, rank;
  u32 nseg, nrun, nlong, pairs;     // runs [0, min(nrun, kRuns)), then nlong from kRuns
};

// Named barriers: kConsumers among the W scanning warps; full(p) and empty(p)
// hand producer p's slot over and back.
__device__ __forceinline__ void bar_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int threads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
constexpr int kBarConsumers = 1;
__device__ __forceinline__ int bar_full(int p) { return 2 + 2 * p; }
__device__ __forceinline__ int bar_empty(int p) { return 3 + 2 * p; }

template <int W, int P, int H>
struct PullSmem {
  u32 key[H + 32];                  // the last 32: standing keys for idle lanes
  u32 lo[H + 32];
  uint2 queue[W][2 * kBatch];       // per warp: matches {table key, parent entry}
  PullUnit unit[P];
  unsigned long long red[3][W];
  unsigned long long apos[2], aend; // this CTA's output block
  u32 claims[2][2];                 // by pass parity: entries of quarters 0 | 1 << 16, 2 | 3 << 16
  u32 over;
  static constexpr u32 kList = H / 16 * 9;  // most entries of half a table
  uint16_t list[2][kList];          // claimed slots: quarters 0 and 2 from the front, 1 and 3 from the back
};

// The table holds a successor before its shift: the parent's diagonals without
// the two that leave the board (or the stored bits), with the new queen's. The
// two freed places hold the signals that enter: u' bit 1 (a queen in column 0)
// at the top of u, d' bit n - 2 (a queen in the last column) at the bottom of
// d. One and-or a match instead of both shifts; shift_key does them once per
// merged entry.
struct KeyShape {
  u32 nu;              // u bits stored: 1 .. nu at 0 .. nu-1; d bits 0 .. n-2 above them
  u32 up_mask, dn_mask;
  u32 keep;            // bits a successor keeps
  u32 d_top;           // place of d bit n-2
  __device__ __forceinline__ KeyShape(unsigned n, unsigned rm) {
    nu = n - 1 - rm;
    up_mask = (1u << nu) - 1u;
    dn_mask = (u32)((((1ull << (n - 1)) - 1ull)) << nu);
    keep = (up_mask >> 1) | (dn_mask & ~(1u << nu));
    d_top = nu + n - 2;
  }
  // Bits column c must have clear in the parent.
  __device__ __forceinline__ u32 test(u32 c, u32 n) const {
    return (c >= 1 && c <= nu ? 1u << (c - 1) : 0u) | (c + 2 <= n ? 1u << (nu + c) : 0u);
  }
  // Bits a queen in column c adds to the table key.
  __device__ __forceinline__ u32 added(u32 c, u32 n) const {
    return (c == 0 ? 1u << (nu - 1) : c < nu ? 1u << (c - 1) : 0u) |
           (c == n - 1 ? 1u << nu : c >= 1 ? 1u << (nu + c) : 0u);
  }
  __device__ __forceinline__ u32 shift_key(u32 t) const {
    return ((t << 1) & up_mask) | ((t >> (nu - 1)) & 1u) | ((t >> 1) & (dn_mask >> 1) & dn_mask) |
           (((t >> nu) & 1u) << d_top);
  }
};

// One warp: the runs of parents that hold a unit's matches, into `u`.
// Lane = column c.
__device__ __forceinline__ bool group_unit_runs(const GroupStepArgs& a, const KeyShape& ks, u32 units,
                                                u32 unit, uint2 ud, PullUnit& u) {
  const u32 lane = threadIdx.x & 31, lt = lt_mask();
  const u32 n = a.n;
  if (lane == 0) {
    u.valid = unit < units;
    u.unit = unit;
    u.nseg = u.nrun = u.nlong = u.pairs = 0;
  }
  if (unit >= units) return false;
  const u32 cols = ud.x & 0xffffffu, b = ud.x >> 24, beta = ud.y;
  const u32 c = lane;
  const bool in_c = c < n && ((cols >> c) & 1u);
  const u32 j = __popc(cols & lt);
  u32 ia = in_c ? a.binomials[c * kBinDim + j + 1] : 0u;
  u32 ib = in_c ? a.binomials[c * kBinDim + j] : 0u;
  const u32 xa = ia;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const u32 ta = __shfl_up_sync(kFull, ia, d), tb = __shfl_up_sync(kFull, ib, d);
    if (lane >= (u32)d) {
      ia += ta;
      ib += tb;
    }
  }
  const u32 all_a = __shfl_sync(kFull, ia, 31), all_b = __shfl_sync(kFull, ib, 31);
  if (lane == 0) {
    u.cols = cols;
    u.b = b;
    u.beta = beta;
    u.rank = all_a;
  }
  __syncwarp();
  const u32 ci = n - 1 - c;  // c's place among the prefix bits (from the top)
  // Bit i of the (b + 1)-bit prefix is u[n - 1 - i]: x, then beta.
  if (!in_c || !(ci == 0 || ci > b || ((beta >> (b - ci)) & 1u))) return true;
  const GroupDir gd = a.in.gdir[(ia - xa) + (all_b - ib)];
  if (!gd.total) return true;
  const u32 bp = gd.bits;
  const u32 add = ks.added(c, n), mask = ks.test(c, n);
#pragma unroll
  for (u32 x = 0; x < 2; ++x) {
    if (ci == 0 && x) break;
    u32 pi = (x << b) | beta;
    if (ci >= 1 && ci <= b) pi &= ~(1u << (b - ci));
    // A bucket stores its quarters in order (the next two bits), so a parent
    // cut one bit more coarsely still gives an exact run.
    u32 fmask = mask, fval = 0, q0, q1, s0 = 0, s1 = 4;  // quarters [s0, s1) of buckets [q0, q1)
    if (bp > b) {
      q0 = pi << (bp - b - 1);
      q1 = q0 + (1u << (bp - b - 1));
    } else if (bp == b) {
      q0 = pi >> 1;
      q1 = q0 + 1;
      s0 = (pi & 1u) * 2u;
      s1 = s0 + 2u;
    } else {
      // The w prefix bits a coarser parent does not resolve are tested.
      const u32 w = b - 1 - bp, top = pi >> w, low = (1u << w) - 1u;
      q0 = top >> 2;
      q1 = q0 + 1;
      s0 = top & 3u;
      s1 = s0 + 1u;
      fmask |= low << (n - 2 - b);
      fval = (pi & low) << (n - 2 - b);
    }
    for (u32 q = q0; q < q1; ++q) {
      uint4 e = a.in.udir[gd.base + q];
      for (;;) {
        const u32 e1 = e.y & 0xffffu, e2 = e1 + (e.y >> 16), e3 = e2 + (e.z & 0xffffu), e4 = e3 + (e.z >> 16);
        const u32 lo = s0 == 0 ? 0u : s0 == 1 ? e1 : s0 == 2 ? e2 : e3;
        const u32 hi = s1 == 1 ? e1 : s1 == 2 ? e2 : s1 == 3 ? e3 : e4;
        if (hi != lo) {
          const u32 off = e.x + lo, len = hi - lo;
          const u32 at = atomicAdd(&u.nseg, 1u);
          if (at < (u32)kMaxSeg) {
            u.test_mask[at] = fmask;
            u.test_value[at] = fval;
            u.added[at] = add;
            atomicAdd(&u.pairs, len);
            // Runs of 128 entries, doubled until the segment has at most 16.
            u32 sh = 7;
            while (len > (16u << sh)) ++sh;
            const u32 cnt = (len + (1u << sh) - 1u) >> sh;
            const u32 first = atomicAdd(&u.nrun, cnt);
            if (first + cnt <= (u32)kRuns) {
              for (u32 k = 0; k < cnt; ++k)
                u.run[first + k] = make_uint2(off + (k << sh), min(1u << sh, len - (k << sh)) | (at << 24));
            } else {
              for (u32 k = first; k < (u32)kRuns; ++k) u.run[k] = make_uint2(0u, 0u);
              u.run[kRuns + atomicAdd(&u.nlong, 1u)] = make_uint2(off, len | (at << 24));  // the whole segment
            }
          }
        }
        if (!e.w) break;
        e = a.in.udir[e.w];
      }
    }
  }
  return true;
}

// W warps scan and insert ("consumers"); P more build the runs of the coming
// units, each in a slot of its own: a unit's runs take four dependent trips to
// L2 (its number, its columns, its parents' directories, their buckets), about
// 3 us, of which the first two are made for the unit after (N = 18 497 -> 489 ms)
// and which P units in the making hide.
template <int W, int P, int H, int CTAS>
__global__ void __launch_bounds__((W + P) * 32, CTAS) group_pull_kernel(GroupStepArgs a) {
  constexpr int BLOCK = (W + P) * 32;
  constexpr int CONS = W * 32;
  constexpr u32 kEmpty = kFull;
  constexpr u32 kStanding = kFull - 1u;  // no key: at most 26 of 32 diagonals are ever taken
  using Smem = PullSmem<W, P, H>;
  constexpr u32 kList = Smem::kList;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Smem& s = *reinterpret_cast<Smem*>(smem_raw);
  const GroupRow* prev = a.prev;
  GroupRow* row = a.row;
  // (One answer for the whole CTA: another CTA may be raising a flag.)
  if (__syncthreads_or(*reinterpret_cast<volatile const u32*>(&row->error) != 0u)) return;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const unsigned n = a.n, m = a.m, rm = a.rm;
  // Sums must stay within a word: an output key has at most four parents a
  // column (the diagonal bits that leave the board). (The rows of 17 and 18
  // columns do.)
  if (prev->weight_max * (4ull * m) >> kWeightBits) {
    if (blockIdx.x == 0 && tid == 0) atomicOr(&row->error, kErrNeedWide);
    return;
  }
  if (blockIdx.x == 0 && tid == 0) row->t_pull = global_ns();
  const u32 units = min(row->units, a.out.unit_cap);
  const KeyShape ks(n, rm);
  for (int i = tid; i < H + 32; i += BLOCK) {
    s.key[i] = i < H ? kEmpty : kStanding;
    s.lo[i] = 0u;
  }
  if (tid == 0) {
    s.claims[0][0] = s.claims[0][1] = s.claims[1][0] = s.claims[1][1] = s.over = 0;
    s.apos[0] = s.apos[1] = s.aend = 0;
  }
  __syncthreads();
  if (wid >= W) {
    // Producer: build, hand over, wait for the slot; ends with an invalid unit.
    // The unit after is taken, and its columns read, meanwhile.
    const int p = wid - W;
    auto take = [&]() { return lane == 0 ? atomicAdd(&row->next_unit, 1u) : 0u; };
    u32 unit = __shfl_sync(kFull, take(), 0);
    uint2 ud = unit < units ? a.units[unit] : make_uint2(0u, 0u);
    for (;;) {
      u32 next = take();
      const bool more = group_unit_runs(a, ks, units, unit, ud, s.unit[p]);
      __syncwarp();
      __threadfence_block();
      bar_arrive(bar_full(p), CONS + 32);
      if (!more) return;
      unit = __shfl_sync(kFull, next, 0);
      ud = unit < units ? a.units[unit] : make_uint2(0u, 0u);
      bar_sync(bar_empty(p), CONS + 32);
    }
  }
  const u32 lt = lt_mask();
  const float rate = out_rate(prev, n, m);
  const u32 board = (1u << n) - 1u;
  unsigned long long wsum = 0, nterms = 0, wmax = 0, total = 0;
  u32 abuf = 0;
  u32 live = (1u << P) - 1u;  // producers that still hand over units
  int slot_at = 0;
  // The stride on its way: first entry, entries left of its run, segment; run
  // r of `runs`, every W-th of which is this warp's.
  u32 src = 0, left = 0, sg = 0, r = 0, runs = 0, nrun = 0;
  u32 kn[4];
  // The next unit's slot, once it is full; -1 when no producer is left. `held`:
  // a slot not yet handed back; its producer cannot fill it, so when it is the
  // next in turn the answer is -2 (ask again after handing it back).
  auto next_slot = [&](int held) -> int {
    while (live) {
      const int p = slot_at;
      if (p == held) return -2;
      slot_at = slot_at + 1 == P ? 0 : slot_at + 1;
      if (!((live >> p) & 1u)) continue;
      bar_sync(bar_full(p), CONS + 32);
      if (s.unit[p].valid) return p;
      live &= ~(1u << p);
    }
    return -1;
  };
  auto load_run = [&](const PullUnit& u) {
    const uint2 rn = u.run[r < nrun ? r : r - nrun + kRuns];
    src = rn.x;
    left = rn.y & 0xffffffu;
    sg = rn.y >> 24;
  };
  auto fetch = [&]() {
    const u32* p = a.in.keys + (u64)src + lane;
    if (left >= 128u) {
#pragma unroll
      for (int i = 0; i < 4; ++i) kn[i] = p[i * 32];
    } else {
      const int rem = (int)left - lane;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (rem > i * 32) kn[i] = p[i * 32];
    }
  };
  auto begin = [&](int p) {
    const PullUnit& u = s.unit[p];
    nrun = min(u.nrun, (u32)kRuns);
    runs = nrun + u.nlong;
    r = wid;
    if (r < runs) {
      load_run(u);
      fetch();
    }
  };
  int slot_u = next_slot(-1);
  if (slot_u >= 0) begin(slot_u);
  while (slot_u >= 0) {
    const PullUnit& u = s.unit[slot_u];
    const u32 b = u.b;
    // The columns taken by the unit's successors, and by their implied bits.
    const u32 fixed = u.cols | (rm ? (u.beta >> (b - rm)) << (n - rm) : 0u);
    if (tid == 0 && u.nseg > (u32)kMaxSeg) atomicOr(&row->error, kErrBounds);
    // A unit expected to pass the table takes several passes over its
    // parents, one range of hashes each.
    const float est = (float)u.pairs * rate;
    u32 width = 0;  // hash range of a pass; 0 = all
    if (est > 0.65f * H) width = (u32)(4294967295.0f / (est / (0.5f * H))) + 1u;
    u32 from = 0;
    uint4 head = make_uint4(0u, 0u, 0u, 0u);
    u32 chain = 0, written = 0;
    int slot_n = -2;                    // the next unit's slot (-2: not known yet)
    bool begun = false;                 // its first keys are on their way
    const u32 quarter_at = n - 4 - b;   // u' bits n-1-b and n-2-b, before the shift
    for (;;) {
      // Scan this warp's runs for matches; insert them 128 at a time.
      u32 qn = 0;
      uint2* const q = s.queue[wid];
      // Queue entries [first, first + count), 32 * items of them if `full`. Lanes
      // beyond the last one insert the key that stands in a slot beyond the
      // table, so that nothing below is predicated.
      auto insert = [&](auto items, auto full, u32 first, u32 count) {
        constexpr int I = decltype(items)::value;
        u32 k[I], slot[I], lo[I];
        u32 todo = (1u << I) - 1u, fresh = 0;
#pragma unroll
        for (int i = 0; i < I; ++i) {
          const u32 at = i * 32 + lane;
          uint2 e;
          if constexpr (decltype(full)::value)
            e = q[first + at];
          else
            e = q[first + min(at, count - 1u)];
          lo[i] = a.in.lo[e.y];
          k[i] = e.x;
          slot[i] = __umulhi(e.x * 0x9E3779B1u, (u32)H);
          if constexpr (!decltype(full)::value)
            if (at >= count) {
              k[i] = kStanding;
              slot[i] = (u32)H + lane;
            }
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < I; ++i) {
          const u32 old = atomicCAS(&s.key[slot[i]], kEmpty, k[i]);
          if (old == kEmpty) fresh |= 1u << i;
          if (old == kEmpty || old == k[i]) todo ^= 1u << i;
        }
        for (u32 probes = 0; todo; ++probes) {
          if (probes == 256u) {
            s.over = 1u;
            break;
          }
          // The lowest one left takes its next slot, a step of the key's own away.
          // (One a turn: 8 % of the board's time less than all four's tests.)
          const u32 one = todo & (0u - todo);
          u32 at = slot[0], key = k[0];
#pragma unroll
          for (int i = 1; i < I; ++i)
            if (one == 1u << i) {
              at = slot[i];
              key = k[i];
            }
          at += ((key * 0x9E3779B1u) >> 4 & 63u) | 1u;
          at = at >= (u32)H ? at - (u32)H : at;
          const u32 old = atomicCAS(&s.key[at], kEmpty, key);
#pragma unroll
          for (int i = 0; i < I; ++i)
            if (one == 1u << i) slot[i] = at;
          if (old == kEmpty) fresh |= one;
          if (old == kEmpty || old == key) todo ^= one;
        }
        __syncwarp();
        // List the claimed slots by quarter: one scan of four byte counts (at
        // most 128 each), two atomics a warp.
        u32 mine = 0;
#pragma unroll
        for (int i = 0; i < I; ++i) mine += ((fresh >> i) & 1u) << (((k[i] >> quarter_at) & 3u) * 8u);
        u32 incl = mine;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const u32 v = __shfl_up_sync(kFull, incl, d);
          if (lane >= d) incl += v;
        }
        const u32 all = __shfl_sync(kFull, incl, 31);
        u32 at = 0;
        if (lane < 2) {
          const u32 both = all >> (lane * 16);
          const u32 c0 = both & 0xffu, c1 = (both >> 8) & 0xffu;
          at = atomicAdd(&s.claims[abuf][lane], c0 | (c1 << 16));
          if ((at & 0xffffu) + (at >> 16) + c0 + c1 > kList) s.over = 1u;
        }
        const u32 at0 = __shfl_sync(kFull, at, 0), at1 = __shfl_sync(kFull, at, 1);
        u32 excl = incl - mine;
#pragma unroll
        for (int i = 0; i < I; ++i) {
          atomicAdd(&s.lo[slot[i]], lo[i]);
          if ((fresh >> i) & 1u) {
            const u32 qt = (k[i] >> quarter_at) & 3u, sh = qt * 8u;
            const u32 base = qt & 2u ? at1 : at0;
            const u32 p = (qt & 1u ? base >> 16 : base & 0xffffu) + ((excl >> sh) & 0xffu);
            excl += 1u << sh;
            if (p < kList) s.list[qt >> 1][qt & 1u ? kList - 1u - p : p] = (uint16_t)slot[i];
          }
        }
      };
      while (r < runs) {
        u32 kc[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) kc[i] = kn[i];
        const u32 tmask = u.test_mask[sg], tval = u.test_value[sg], add = u.added[sg];
        const u32 entry = src + lane;
        const int rem = (int)left - lane;
        if (left > 128u) {
          src += 128u;
          left -= 128u;
          fetch();
        } else {
          r += W;
          if (r < runs) {
            load_run(u);
            fetch();
          }
        }
        bool hit[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          hit[i] = (kc[i] & tmask) == tval && rem > i * 32;
          kc[i] = (kc[i] & ks.keep) | add;
        }
        if (width) {
#pragma unroll
          for (int i = 0; i < 4; ++i) hit[i] = hit[i] && (kc[i] * 0xC2B2AE35u) - from < width;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const u32 bal = __ballot_sync(kFull, hit[i]);
          if (hit[i]) q[qn + __popc(bal & lt)] = make_uint2(kc[i], entry + i * 32);
          qn += __popc(bal);
        }
        if (qn >= kBatch) {
          __syncwarp();
          qn -= kBatch;
          insert(Items<4>{}, TrueTag{}, qn, kBatch);
        }
      }
      __syncwarp();
      // (A warp's last part batch is 40 matches on average: half as wide, N = 17
      // takes 53.4 ms instead of 54.0. Narrower still, in turns: 54.6 and 55.9.)
      if (qn > 64u)
        insert(Items<4>{}, FalseTag{}, 0, qn);
      else if (qn)
        insert(Items<2>{}, FalseTag{}, 0, qn);
      bar_sync(kBarConsumers, CONS);
      const bool over = s.over != 0;
      const u32 c01 = s.claims[abuf][0], c23 = s.claims[abuf][1];
      const u32 e1 = c01 & 0xffffu, e2 = e1 + (c01 >> 16), e3 = e2 + (c23 & 0xffffu), cnt = e3 + (c23 >> 16);
      unsigned long long base = s.apos[abuf];
      const bool refill = base + cnt > s.aend;
      if (over || refill) {
        bar_sync(kBarConsumers, CONS);
        if (over) {
          // Too many keys for the table: clear it and take half the range.
          for (u32 i = tid; i < (u32)H; i += CONS) {
            s.key[i] = kEmpty;
            s.lo[i] = 0u;
          }
          if (tid == 0) s.over = s.claims[abuf][0] = s.claims[abuf][1] = 0;
          width = width ? width / 2 : 0x80000000u;
          bar_sync(kBarConsumers, CONS);
          if (width > 1024u) {
            begin(slot_u);
            continue;
          }
          if (tid == 0) atomicOr(&row->error, kErrBounds);  // not reached: 1024 hashes fit the table
          break;
        }
        // A new output block (the rest of the last one stays unused).
        if (tid == 0) {
          base = atomicAdd(&row->alloc, (unsigned long long)a.block);
          s.apos[abuf] = base;
          s.aend = base + a.block;
        }
        bar_sync(kBarConsumers, CONS);
        base = s.apos[abuf];
      }
      const bool last = !width || from + width < from || from + width == 0;
      if (last) {
        // The next unit's first keys travel while this one is written.
        slot_n = next_slot(slot_u);
        if (slot_n >= 0) begin(slot_n);
        begun = slot_n >= 0;
      }
      const bool fits = base + cnt <= a.out.cap;
      const bool wr = a.write_out && fits;
      // Compaction in list order, quarter by quarter; the table is left empty.
      u32* const okey = a.out.keys + base;
      u32* const olo = a.out.lo + base;
      u32 terms = 0;
      for (u32 i = tid; i < cnt; i += CONS) {
        const u32 h = i >= e2;
        const u32 j = h ? i - e2 : i, front = h ? e3 - e2 : e1;
        const u32 slot = s.list[h][j < front ? j : kList - 1u - (j - front)];
        const u32 key = ks.shift_key(s.key[slot]);
        const u32 lo = s.lo[slot];
        s.key[slot] = kEmpty;
        s.lo[slot] = 0u;
        wsum += lo;
        wmax = max((u32)wmax, lo);
        terms += __popc(board & ~(fixed | ((key & ks.up_mask) << 1) | (key >> ks.nu)));
        if (wr) {
          okey[i] = key;
          olo[i] = lo;
        }
      }
      nterms += terms;
      if (tid == 0) {
        if (cnt && a.write_out) {
          const uint4 piece = make_uint4((u32)base, c01, c23, 0u);
          if (!fits) {
            atomicOr(&row->error, kErrOverflow);
          } else if (!written) {
            head = piece;
          } else {
            const u32 at = units + atomicAdd(&row->pieces, 1u);
            if (at < a.out.unit_cap) {
              a.out.udir[at] = make_uint4(piece.x, piece.y, piece.z, chain);
              chain = at;
            } else {
              atomicOr(&row->error, kErrOverflow);
            }
          }
        }
        written += cnt;
        if (last && a.write_out && written) {
          a.out.udir[u.unit] = make_uint4(head.x, head.y, head.z, chain);
          atomicAdd(&a.out.gdir[u.rank].total, written);
        }
        s.apos[abuf ^ 1] = base + cnt;
        s.claims[abuf ^ 1][0] = s.claims[abuf ^ 1][1] = 0;  // (this pass's are still being read)
        total += cnt;
      }
      abuf ^= 1;
      bar_sync(kBarConsumers, CONS);
      if (last) break;
      from += width;
      if (from + width < from) width = 0u - from;  // the last range
      begin(slot_u);
    }
    bar_arrive(bar_empty(slot_u), CONS + 32);
    if (slot_n == -2) slot_n = next_slot(-1);
    if (slot_n >= 0 && !begun) begin(slot_n);
    slot_u = slot_n;
  }
  // Row sums.
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    wsum += __shfl_xor_sync(kFull, wsum, d);
    nterms += __shfl_xor_sync(kFull, nterms, d);
    const unsigned long long o = __shfl_xor_sync(kFull, wmax, d);
    wmax = o > wmax ? o : wmax;
  }
  if (lane == 0) {
    s.red[0][wid] = wsum;
    s.red[1][wid] = nterms;
    s.red[2][wid] = wmax;
  }
  bar_sync(kBarConsumers, CONS);
  if (tid == 0) {
    wsum = nterms = wmax = 0;
    for (int w = 0; w < W; ++w) {
      wsum += s.red[0][w];
      nterms += s.red[1][w];
      wmax = s.red[2][w] > wmax ? s.red[2][w] : wmax;
    }
    if (total) atomicAdd(&row->out_count, total);
    if (wsum) atomicAdd(&row->weight_sum, wsum);
    if (nterms) atomicAdd(&row->next_terms, nterms);
    if (wmax) atomicMax(&row->weight_max, wmax);
    atomicMax(&row->t_end, global_ns());
    // The last CTA out knows the row's merge rate for the next plan.
    __threadfence();
    if (atomicAdd(&row->ctas_done, 1u) + 1u == gridDim.x) {
      __threadfence();
      const unsigned long long out = *reinterpret_cast<volatile unsigned long long*>(&row->out_count);
      row->merge_rate = prev->next_terms ? (float)out / (float)prev->next_terms : 1.f;
    }
  }
}

__global__ void group_seed_kernel(const GroupSeedUnit* __restrict__ list, u32 count, GroupSide side) {
  const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const GroupSeedUnit e = list[i];
  if (e.unit < side.unit_cap) side.udir[e.unit] = make_uint4(e.first, e.quarters01, e.quarters23, 0u);
  if (e.total) side.gdir[e.rank] = GroupDir{e.unit, e.bits, e.total, 0u};
}

constexpr int kPlanBlock = 256;
// Two CTAs an SM with tables as large as fit beside the queues, since a unit
// costs about 2 us besides its candidates. N = 16 / 17, device ms, warps +
// producers x slots at two CTAs: 12 + 2 x 7744 8.4 / 54.5; 10 + 2 x 8192
// 8.7 / 56.1; 9 + 2 x 8416 8.8 / 57.1; 13 + 2 x 7520 9.1 / 57.7 and 14 + 2 x 7296
// 9.4 / 59.6 (too few registers); 10 + 3 x 7872 9.0 / 56.9; 12 + 1 x 7872
// 10.7 / 68.5. Three CTAs with 5376 slots were 20 % slower, one with 16384 30 %.
constexpr int kPullWarps = 12;
constexpr int kPullProducers = 2;
constexpr int kPullTable = 7744;
constexpr int kPullCtas = 2;  // per SM

}  // namespace

// Buckets of a group are uneven (the largest hundredth hold 3 to 4 times the
// mean), and one beyond 0.65 of the table is scanned twice or more. N = 16 / 17,
// ms, at 0.22: 8.7 / 56.4, at 0.25: 8.45 / 55.2, at 0.28: 8.44 / 54.5.
float group_unit_target() { return 0.28f * kPullTable; }

// A row with few outputs is cut finely enough for eight units a CTA: its largest
// bucket is one CTA's work (the last row of N = 15 was 128 buckets and 143 us;
// board 2.07 -> 1.97 ms).
float group_unit_share(int sms) { return 1.f / (8.f * (float)(sms * kPullCtas)); }

uint32_t group_block(double states, int sms) {
  const double share = states / ((double)sms * kPullCtas * 16.0);
  return (uint32_t)std::min(65536.0, std::max((double)kPullTable, share));
}

uint64_t group_capacity(double states, int sms) {
  const double block = group_block(states, sms);
  // A block's unused end is below half a table on average.
  return (uint64_t)(states * (1.0 + 0.5 * kPullTable / block * 0.5) + block * sms * kPullCtas) + 4096;
}

cudaError_t launch_group_plan(const GroupStepArgs& a, uint32_t groups, cudaStream_t stream) {
  group_plan_kernel<kPlanBlock><<<(groups + kPlanBlock - 1) / kPlanBlock, kPlanBlock, 0, stream>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_group_pull(const GroupStepArgs& a, int sms, cudaStream_t stream) {
  using Smem = PullSmem<kPullWarps, kPullProducers, kPullTable>;
  static_assert(kPullCtas * (sizeof(Smem) + 1024) <= 228 * 1024, "resident CTAs' shared memory");
  auto* k = group_pull_kernel<kPullWarps, kPullProducers, kPullTable, kPullCtas>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Smem));
  if (e != cudaSuccess) return e;
  k<<<sms * kPullCtas, (kPullWarps + kPullProducers) * 32, sizeof(Smem), stream>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_group_seed(const GroupSeedUnit* list, uint32_t count, const GroupSide& side, cudaStream_t stream) {
  group_seed_kernel<<<(count + 255) / 256, 256, 0, stream>>>(list, count, side);
  return cudaGetLastError();
}

}  // namespace qpeps
