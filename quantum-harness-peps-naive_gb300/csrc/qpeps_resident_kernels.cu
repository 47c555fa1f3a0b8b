// Small contractions in one CTA.
//
// A partly placed board of a few hundred states has rows of some hundred
// successors: as two kernels a row, launches and trips to L2 take 7 us for
// work of well under one. Here one CTA keeps the boundary in shared memory
// from the first row to the last: every thread expands its states into a
// shared-memory table (a 64-bit compare-and-swap claims a key's slot, the
// weight is added), and the table is read back into the state list. What is
// left is two block barriers and a handful of shared-memory trips a row, about
// 1.5 us.
#include <cuda_runtime.h>

#include "qpeps_device.cuh"
#include "qpeps_internal.h"

namespace qpeps {

namespace {

constexpr u32 kAll = 0xffffffffu;
constexpr int kResidentBlock = 512;
constexpr u32 kResidentStates = 4096;
constexpr u32 kResidentSlots = 8192;
constexpr u64 kNoKey = ~0ull;  // no u64 row key is all ones

struct ResidentSmem {
  u64 key[kResidentStates];
  u64 weight[kResidentStates];
  u64 slot_key[kResidentSlots];
  unsigned long long slot_weight[kResidentSlots];
  unsigned long long sum[2][4];  // by row parity: weights, final weights, final states, next row's terms
  u32 states[2];                 // by row parity: merged states
};

__global__ void __launch_bounds__(kResidentBlock) resident_rows_kernel(const __grid_constant__ ResidentArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  ResidentSmem& s = *reinterpret_cast<ResidentSmem*>(smem_raw);
  const u32 tid = threadIdx.x, lane = tid & 31;
  const u32 n = a.n;
  const u64 board = (1ull << n) - 1;
  if (tid == 0) a.out[0].t_scatter = global_ns();
  u32 states = a.count;
  u64 terms = 0;
  for (u32 i = 0; i < a.count; ++i) {
    const State st = unpack<u64>(a.key[i], n, board);
    terms += __popcll(~(st.cols | st.dr | st.dl) & board);
    if (tid == 0) {
      s.key[i] = a.key[i];
      s.weight[i] = a.weight[i];
    }
  }
  // Only as much of the table as a row's terms need at a load of 1/4 (at most
  // 3/4 when it is full) is used and read back; all of it is kept empty.
  auto slots_for = [](u64 t) {
    u32 h = 256;
    while (h < kResidentSlots && h < 4 * t) h <<= 1;
    return h;
  };
  u32 clean = 0;  // slots [0, clean) are empty
  for (u32 row = a.row; row < n; ++row) {
    StepScalars* const out = a.out + (row - a.row);
    const u32 par = row & 1u;
    if (terms > kResidentSlots * 3 / 4) {
      if (tid == 0) a.out[0].error = kErrCapacity;
      return;
    }
    const u32 slots = slots_for(terms);
    const u32 shift = 64 - (31 - __clz(slots));
    for (u32 i = clean + tid; i < slots; i += kResidentBlock) {
      s.slot_key[i] = kNoKey;
      s.slot_weight[i] = 0ull;
    }
    clean = max(clean, slots);
    if (tid < 4) s.sum[par][tid] = 0ull;
    if (tid == 0) s.states[par] = 0;
    __syncthreads();
    for (u32 i = tid; i < states; i += kResidentBlock) {
      const State st = unpack<u64>(s.key[i], n, board);
      const unsigned long long w = s.weight[i];
      u64 fr = ~(st.cols | st.dr | st.dl) & board;
      while (fr) {
        const u64 b = fr & (0ull - fr);
        fr ^= b;
        const u64 k = row_successor<u64>(st, b, n, board);
        u32 at = (u32)(fib_hash_b(k) >> shift);
        for (;;) {  // ends: the table has more slots than terms
          const u64 old = atomicCAS(reinterpret_cast<unsigned long long*>(&s.slot_key[at]), kNoKey, k);
          if (old == kNoKey || old == k) break;
          at = (at + 1) & (slots - 1);
        }
        atomicAdd(&s.slot_weight[at], w);
      }
    }
    __syncthreads();
    unsigned long long v[4] = {0, 0, 0, 0};
    bool over = false;
    for (u32 i0 = 0; i0 < slots; i0 += kResidentBlock) {
      const u32 i = i0 + tid;
      const u64 k = i < slots ? s.slot_key[i] : kNoKey;
      const bool used = k != kNoKey;
      const u32 b = __ballot_sync(kAll, used);
      u32 at = 0;
      if (lane == 0 && b) at = atomicAdd(&s.states[par], __popc(b));
      at = __shfl_sync(kAll, at, 0) + __popc(b & ((1u << lane) - 1u));
      if (used) {
        const unsigned long long w = s.slot_weight[i];
        const State st = unpack<u64>(k, n, board);
        v[0] += w;
        if (st.cols == board) {
          v[1] += w;
          v[2] += 1;
        }
        v[3] += __popcll(~(st.cols | st.dr | st.dl) & board);
        over |= at >= kResidentStates;
        if (at < kResidentStates) {
          s.key[at] = k;
          s.weight[at] = w;
        }
        s.slot_key[i] = kNoKey;
        s.slot_weight[i] = 0ull;
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) v[q] += __shfl_xor_sync(kAll, v[q], d);
      if (lane == 0 && v[q]) atomicAdd(&s.sum[par][q], v[q]);
    }
    const bool stop = __syncthreads_or(over);
    states = s.states[par];
    const u64 next = s.sum[par][3];
    if (tid == 0) {
      out->terms = terms;
      out->out_count = states;
      out->weight_sum[0] = s.sum[par][0];
      out->final_sum[0] = s.sum[par][1];
      out->final_states = s.sum[par][2];
      out->next_terms = next;
      if (stop) a.out[0].error = kErrCapacity;
    }
    if (stop) return;
    terms = next;
  }
  if (tid == 0) a.out[n - 1 - a.row].t_merge = global_ns();
}

}  // namespace

uint32_t resident_capacity() { return kResidentStates; }

cudaError_t launch_resident_rows(const ResidentArgs& a, cudaStream_t stream) {
  if (a.count == 0 || a.count > kResidentSeeds || a.row >= a.n || a.n > kU64MaxN) return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(resident_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)sizeof(ResidentSmem));
  if (e != cudaSuccess) return e;
  resident_rows_kernel<<<1, kResidentBlock, sizeof(ResidentSmem), stream>>>(a);
  return cudaGetLastError();
}

}  // namespace qpeps
