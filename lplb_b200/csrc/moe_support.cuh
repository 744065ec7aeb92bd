// Dispatch planning, token dispatch over NVLink peer memory, and the final weighted
// reduction of the benchmark MoE layer (sm_100a).  The reference has no MoE layer; these
// kernels consume the planner's redirected indices for the end-to-end measurement.
#pragma once

#include <cuda_bf16.h>

#include "common.cuh"
#include "moe_gemm.cuh"

namespace lplb {
namespace moe {

constexpr int kSupportThreads = 256;
constexpr int kCombineMaxTopk = 64;
// The layer's status block: words 0-7 its own (word 0 = first error), 8-15 the counting
// kernel's, 16-31 the record of the bounds-checking build (same layout as the planner's block).
constexpr int kMoeStatusWords = 32;
constexpr int kMoeBoundsBase = 16;

__device__ __forceinline__ unsigned long long ldv_u64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.volatile.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void stv_u64(unsigned long long* p, unsigned long long v) {
  asm volatile("st.volatile.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

struct RouteArgs {
  const void* idx;                           // [n_pairs] physical expert ids, -1 = skip
  int* ordinal;                              // [n_pairs] out: position of the pair among this rank's pairs for its expert
  int* totals;                               // [P] zero before the launch, left at zero
  unsigned* ticket;                          // zero before the launch, left at zero
  int* count_status;                         // planner status block: out-of-range ids
  unsigned long long* cnt_words[kMaxRanks];  // per rank: uint64 [2][n_ranks][P]
  int* plan;                                 // see plan_words() in moe_api.h
  int* status;
  long long n_pairs;
  int idx_is64, n_ranks, my_rank, n_local, capacity;
  int fused;  // the launch uses the fused dispatch: advance the cumulative arrival targets
  uint32_t epoch;
  unsigned long long timeout_ns;
};

__device__ __forceinline__ long long pair_expert(const void* idx, int is64, long long i) {
  return is64 ? ((const long long*)idx)[i] : (long long)((const int*)idx)[i];
}

// Exclusive prefix over n elements by one warp: put(i, sum of get(j) for j < i); returns the total.
template <typename Get, typename Put>
__device__ __forceinline__ int warp_exclusive_prefix(int n, int lane, Get get, Put put) {
  int carry = 0;
  for (int i0 = 0; i0 < n; i0 += 32) {
    const int i = i0 + lane;
    const int v = i < n ? get(i) : 0;
    int inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += up;
    }
    if (i < n) put(i, carry + inc - v);
    carry += __shfl_sync(0xffffffffu, inc, 31);
  }
  return carry;
}

// Counting and planning in one launch.  Every CTA ranks its own pairs with shared-memory
// atomics, reserves a range per expert with one returning atomicAdd on the rank's totals, and
// stores each pair's ordinal; the CTA that finishes last all-gathers the totals (packed
// (epoch, value) words, as in the planner's exchange) and derives for this launch
//   rows[le], row_start[le]      rows each local expert receives and where they start
//   dst_row_start[p]             first row, on the target rank, of this rank's pairs for expert p
//   all_counts[src][p], send_base[p], order_base[p], arrive_target[le]
// With the ordinal of every pair at hand, whatever runs next can work on the pairs in any order
// and on any number of CTAs.  What bounds it is the chain of dependent memory round trips, so
// there is no column scan over the CTAs' counts (the ranges come from atomics) and every prefix
// is a warp scan.  Launch of its own for each half, column scan and serial prefixes: 25 us for
// 512 pairs on 48 experts.
__global__ void __launch_bounds__(kSupportThreads) route_kernel(const RouteArgs a) {
  extern __shared__ int sm[];
  allow_successor();
  wait_predecessors();
  const int P = a.n_ranks * a.n_local, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int* hist = sm;  // [P] this CTA's counts, then its first ordinal per expert
  __shared__ int s_last, s_missing;
  constexpr int kHold = 4;  // pairs per thread whose expert and ordinal stay in registers
  const long long begin = slice_begin(a.n_pairs, blockIdx.x, gridDim.x, 32);
  const long long end = slice_begin(a.n_pairs, blockIdx.x + 1, gridDim.x, 32);
  int e_hold[kHold], k_hold[kHold];
#pragma unroll
  for (int j = 0; j < kHold; ++j) {
    const long long i = begin + tid + (long long)j * kSupportThreads;
    const long long e = i < end ? pair_expert(a.idx, a.idx_is64, i) : -1;
    e_hold[j] = e >= 0 && e < P ? (int)e : (e == -1 ? -1 : -2);
  }
  for (int i = tid; i < P; i += kSupportThreads) hist[i] = 0;
  if (tid == 0) s_missing = 0;
  __syncthreads();
  int bad = 0;
#pragma unroll
  for (int j = 0; j < kHold; ++j) {
    k_hold[j] = e_hold[j] >= 0 ? atomicAdd(&hist[e_hold[j]], 1) : 0;
    bad += e_hold[j] == -2;
  }
  for (long long i = begin + tid + (long long)kHold * kSupportThreads; i < end; i += kSupportThreads) {
    const long long e = pair_expert(a.idx, a.idx_is64, i);
    if (e >= 0 && e < P) a.ordinal[i] = atomicAdd(&hist[e], 1);
    else bad += e != -1;
  }
  if (bad) {
    atomicAdd(&a.count_status[kStBadIdx], bad);
    raise_status(a.count_status, kErrBadIndex, kPhCount, bad);
  }
  __syncthreads();
  for (int i = tid; i < P; i += kSupportThreads) {
    const int c = hist[i];
    hist[i] = c ? atomicAdd(&a.totals[i], c) : 0;
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) s_last = atomicAdd(a.ticket, 1u) == gridDim.x - 1;  // the reservations above precede it
#pragma unroll
  for (int j = 0; j < kHold; ++j)
    if (e_hold[j] >= 0) a.ordinal[begin + tid + (long long)j * kSupportThreads] = hist[e_hold[j]] + k_hold[j];
  for (long long i = begin + tid + (long long)kHold * kSupportThreads; i < end; i += kSupportThreads) {
    const long long e = pair_expert(a.idx, a.idx_is64, i);
    if (e >= 0 && e < P) a.ordinal[i] += hist[e];
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();

  // ---- the plan -----------------------------------------------------------------------------
  int* rows = a.plan;
  int* row_start = rows + a.n_local;
  int* dst_row_start = row_start + a.n_local;
  int* all_counts = dst_row_start + P;
  int* tail = all_counts + a.n_ranks * P;
  int* local = sm;              // [P] this rank's totals (the reservations are no longer needed)
  int* n_all = sm + P;          // [P] rows of expert p on its own rank
  int* start_all = sm + 2 * P;  // [P] row start of expert p on its own rank
  int* before = sm + 3 * P;     // [P] rows of expert p from ranks in front of this one
  for (int i = tid; i < P; i += kSupportThreads) {
    local[i] = __ldcg(&a.totals[i]);
    a.totals[i] = 0;
  }
  if (tid == 0) *a.ticket = 0;
  const int parity = a.epoch & 1;
  if (a.n_ranks > 1) {
    const unsigned long long tag = (unsigned long long)a.epoch << 32;
    for (int i = tid; i < P; i += kSupportThreads)  // each thread pushes the entries it just loaded
      for (int r = 0; r < a.n_ranks; ++r)
        stv_u64(a.cnt_words[r] + ((size_t)parity * a.n_ranks + a.my_rank) * P + i, tag | (uint32_t)local[i]);
    const unsigned long long* base = a.cnt_words[a.my_rank] + (size_t)parity * a.n_ranks * P;
    const uint64_t t0 = global_timer_ns();
    for (int p = tid; p < P; p += kSupportThreads) {
      int n = 0, b = 0;
      for (int src = 0; src < a.n_ranks; ++src) {
        const unsigned long long* word = &base[(size_t)src * P + p];
        unsigned long long w = ldv_u64(word);
        uint32_t spins = 0;
        while ((uint32_t)(w >> 32) != a.epoch) {
          if ((++spins & 63u) == 0) {
            if (global_timer_ns() - t0 > a.timeout_ns) {
              s_missing = 1;
              break;
            }
            __nanosleep(100);
          }
          w = ldv_u64(word);
        }
        const int c = (uint32_t)(w >> 32) == a.epoch ? (int)(uint32_t)w : 0;
        all_counts[src * P + p] = c;
        if (src < a.my_rank) b += c;
        n += c;
      }
      n_all[p] = n;
      before[p] = b;
    }
  } else {
    for (int i = tid; i < P; i += kSupportThreads) {
      all_counts[i] = n_all[i] = local[i];
      before[i] = 0;
    }
  }
  __syncthreads();
  if (tid == 0 && s_missing) atomicCAS(a.status, 0, kMoeFlagTimeout);
  int* order_base = tail + 8;
  int* send_base = order_base + P;
  int* arrive_target = send_base + P;
  int* arrive_cum = arrive_target + a.n_local;
  for (int task = warp; task < a.n_ranks + 2; task += kSupportThreads / 32) {
    if (task < a.n_ranks) {  // row starts on rank `task`
      const int first = task * a.n_local;
      const int total = warp_exclusive_prefix(
          a.n_local, lane, [&](int i) { return n_all[first + i]; }, [&](int i, int v) { start_all[first + i] = v; });
      if (task == a.my_rank && lane == 0) {
        tail[0] = total;
        tail[1] = total > a.capacity;
        if (total > a.capacity) atomicCAS(a.status, 0, kMoeOverflow);
      }
    } else if (task == a.n_ranks) {
      // Send order of this rank's pairs: local expert index first, then target rank starting
      // with this rank and rotating, so that at any moment the senders aim at different
      // receivers while every rank's expert 0 completes first, then expert 1, ...
      auto at = [&](int i) { return ((a.my_rank + i % a.n_ranks) % a.n_ranks) * a.n_local + i / a.n_ranks; };
      const int total = warp_exclusive_prefix(
          P, lane, [&](int i) { return local[at(i)]; }, [&](int i, int v) { order_base[at(i)] = v; });
      if (lane == 0) tail[2] = total;
    } else {  // return slots: physical expert order
      warp_exclusive_prefix(P, lane, [&](int i) { return local[i]; }, [&](int i, int v) { send_base[i] = v; });
    }
  }
  __syncthreads();
  for (int p = tid; p < P; p += kSupportThreads) dst_row_start[p] = start_all[p] + before[p];
  for (int le = tid; le < a.n_local; le += kSupportThreads) {
    // rows past the receive buffer's capacity are dropped by the senders; clamp to match
    const int st = start_all[a.my_rank * a.n_local + le];
    const int n = n_all[a.my_rank * a.n_local + le];
    const int kept = max(0, min(n, a.capacity - st));
    rows[le] = kept;
    row_start[le] = min(st, a.capacity);
    // the fused dispatch counts landed rows cumulatively over launches
    const int cum = arrive_cum[le] + (a.fused ? kept : 0);
    arrive_cum[le] = cum;
    arrive_target[le] = cum;
  }
}

struct ScheduleArgs {
  const void* idx;           // [n_pairs] physical expert ids
  const int* ordinal;        // [n_pairs] from route_kernel
  const int* dst_row_start;  // [P]
  const int* order_base;     // [P]
  const int* send_base;      // [P]
  int* pair_slot;            // [n_pairs] out
  int* send_pair;            // [n_send] out
  int* send_target;          // [n_send] out
  int* status;
  long long n_pairs;
  int idx_is64, n_local, n_ranks, capacity;
};

// Fused dispatch: for the k-th pair this rank sends to physical expert e: target row
// dst_row_start[e] + k, return slot send_base[e] + k, send position order_base[e] + k.
__global__ void __launch_bounds__(kSupportThreads) schedule_kernel(const ScheduleArgs a) {
  allow_successor();
  wait_predecessors();
  const int P = a.n_ranks * a.n_local;
  const long long stride = (long long)gridDim.x * kSupportThreads;
  for (long long i = (long long)blockIdx.x * kSupportThreads + threadIdx.x; i < a.n_pairs; i += stride) {
    const long long e = pair_expert(a.idx, a.idx_is64, i);
    int slot = -1;
    if (e >= 0 && e < P) {
      const int k = a.ordinal[i];
      const int row = a.dst_row_start[e] + k;
      const int pos = a.order_base[e] + k;
      if (!LPLB_CHECKED(pos, a.n_pairs, a.status + kMoeBoundsBase, kPhRedirect)) continue;
      a.send_pair[pos] = (((int)e % a.n_local) << 20) | (int)i;  // local expert index rides along
      if (row < a.capacity) {
        slot = a.send_base[e] + k;
        a.send_target[pos] = (((int)e / a.n_local) << 24) | row;
      } else {
        a.send_target[pos] = -1;
      }
    }
    a.pair_slot[i] = slot;
  }
}

struct DispatchArgs {
  __nv_bfloat16* recv_x[kMaxRanks];  // per rank: [capacity, hidden]
  int* recv_meta[kMaxRanks];         // per rank: [capacity]
  uint32_t* flags[kMaxRanks];        // per rank: uint32 [2][n_ranks]
  const __nv_bfloat16* x;            // [tokens, hidden] local hidden states
  const void* idx;                   // [tokens * topk] physical expert ids, -1 = skip
  const int* ordinal;                // [tokens * topk] from route_kernel
  const int* dst_row_start;          // [P]
  const int* send_base;              // [P]
  int* pair_slot;                    // [tokens * topk] out: return slot of every pair, -1 = dropped
  int* status;
  unsigned* ticket;
  int n_tokens;
  int idx_is64, topk, hidden, n_local, n_ranks, my_rank, capacity;
  uint32_t epoch;
};

constexpr int kDispatchVec = 4;  // 16-byte vectors per lane and work item: an item is 2 KB of one token

// Push dispatch.  A work item is one token's hidden state, 2 KB of it: a warp loads that piece
// once and stores it to the rows of all the token's pairs, straight into the target ranks'
// receive buffers (16-byte stores, over NVLink for peers); the last CTA to finish raises this
// rank's "dispatch done" flag on every peer.  Bound by the bytes written, topk rows per token;
// splitting rows into pieces keeps every SM busy from 64 tokens on, and loading a piece once
// for all its pairs halves the traffic through L2.  One CTA per slice of 256 pairs and a row per
// warp and pair took 179 us for 64 tokens x top-8 x 7168 (two CTAs at work) and 495 us for 8192.
//
// Return path: the k-th pair this rank sends to physical expert e gets return slot
// send_base[e] + k, where send_base is the exclusive prefix of this rank's own counts.  The
// slot travels with the row (meta), and the expert's rank writes the result row to that slot
// of this rank's return buffer.  Consecutive rows of an expert therefore come back to
// consecutive slots: the stores that cross NVLink walk through memory sequentially instead of
// hitting a random page per row.
__global__ void __launch_bounds__(kSupportThreads) dispatch_kernel(const DispatchArgs a) {
  allow_successor();
  wait_predecessors();
  const int P = a.n_ranks * a.n_local;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int vec_per_row = a.hidden / 8;  // 16-byte vectors per row
  const int pieces = (vec_per_row + 32 * kDispatchVec - 1) / (32 * kDispatchVec);
  const int n_items = a.n_tokens * pieces, n_warps = gridDim.x * (kSupportThreads / 32);
  for (int item = blockIdx.x * (kSupportThreads / 32) + warp; item < n_items; item += n_warps) {
    const int tok = item / pieces, v0 = (item - tok * pieces) * 32 * kDispatchVec + lane;
    const uint4* src = reinterpret_cast<const uint4*>(a.x + (size_t)tok * a.hidden);
    uint4 q[kDispatchVec];
#pragma unroll
    for (int u = 0; u < kDispatchVec; ++u)
      if (v0 + 32 * u < vec_per_row) q[u] = __ldg(&src[v0 + 32 * u]);
    for (int k0 = 0; k0 < a.topk; k0 += 32) {
      const int nk = min(32, a.topk - k0);
      int t = -1;
      if (lane < nk) {
        const long long i = (long long)tok * a.topk + k0 + lane;
        const long long e = pair_expert(a.idx, a.idx_is64, i);
        int slot = -1;
        if (e >= 0 && e < P) {
          const int k = a.ordinal[i];
          const int row = a.dst_row_start[e] + k;
          if (row >= 0 && row < a.capacity) {
            const int dr = (int)e / a.n_local;
            slot = a.send_base[e] + k;
            if (LPLB_CHECKED(dr, a.n_ranks, a.status + kMoeBoundsBase, kPhRedirect) &&
                LPLB_CHECKED(slot, (long long)a.n_tokens * a.topk, a.status + kMoeBoundsBase, kPhRedirect)) {
              t = (dr << 24) | row;
              if (v0 < 32) a.recv_meta[dr][row] = (a.my_rank << 20) | slot;
            } else {
              slot = -1;
            }
          }
        }
        if (v0 < 32) a.pair_slot[i] = slot;  // the piece that starts the row keeps the books
      }
      for (int k = 0; k < nk; ++k) {
        const int tg = __shfl_sync(0xffffffffu, t, k);
        if (tg < 0) continue;
        uint4* dst = reinterpret_cast<uint4*>(a.recv_x[tg >> 24] + (size_t)(tg & 0xFFFFFF) * a.hidden);
#pragma unroll
        for (int u = 0; u < kDispatchVec; ++u)
          if (v0 + 32 * u < vec_per_row) dst[v0 + 32 * u] = q[u];
      }
    }
  }
  if (a.n_ranks == 1) return;  // nobody waits for the flags: the next kernel follows on the stream
  __threadfence_system();
  __syncthreads();
  if (threadIdx.x == 0) {
    if (atomicAdd(a.ticket, 1u) == gridDim.x - 1) {
      *a.ticket = 0;
      __threadfence_system();
      for (int r = 0; r < a.n_ranks; ++r) st_release_sys(a.flags[r] + a.my_rank, a.epoch);
    }
  }
}

struct CombineArgs {
  const __nv_bfloat16* comb;  // [tokens * topk, hidden] rows written by the experts' ranks
  const float* weights;       // [tokens, topk]
  const int* pair_slot;       // [tokens * topk] row of `comb` that holds each pair's result, -1 = none
  __nv_bfloat16* out;         // [tokens, hidden]
  const uint32_t* wait_flags; // this rank's "combine done" flags [n_ranks]
  int* status;
  int n_tokens, topk, hidden, n_ranks;
  uint32_t epoch;
  unsigned long long timeout_ns;
};

// out[t] = sum_k weights[t, k] * comb[pair_slot[t * topk + k]], fp32 accumulation, after every rank has
// signalled that its expert outputs for this launch are in place.
__global__ void __launch_bounds__(kSupportThreads) combine_kernel(const CombineArgs a) {
  wait_predecessors();
  __shared__ int ok;
  if (threadIdx.x == 0) {
    ok = 1;
    const uint64_t t0 = global_timer_ns();
    for (int r = 0; r < a.n_ranks && ok; ++r) {
      while ((int32_t)(ld_acquire_sys(a.wait_flags + r) - a.epoch) < 0) {
        if (global_timer_ns() - t0 > a.timeout_ns) {
          ok = 0;
          atomicCAS(a.status, 0, kMoeFlagTimeout);
          break;
        }
        __nanosleep(200);
      }
    }
  }
  __syncthreads();
  if (!ok) return;
  const int vec_per_row = a.hidden / 8;
  // Per token: the slots and weights of its pairs go through shared memory once, then every
  // thread has the rows of up to eight pairs in flight before it starts to accumulate.
  __shared__ int s_slot[kCombineMaxTopk];
  __shared__ float s_w[kCombineMaxTopk];
  for (int t = blockIdx.x; t < a.n_tokens; t += gridDim.x) {
    __syncthreads();
    for (int k = threadIdx.x; k < a.topk; k += kSupportThreads) {
      const long long pair = (long long)t * a.topk + k;
      s_slot[k] = a.pair_slot[pair];
      s_w[k] = a.weights[pair];
    }
    __syncthreads();
    for (int v = threadIdx.x; v < vec_per_row; v += kSupportThreads) {
      float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      for (int k0 = 0; k0 < a.topk; k0 += 8) {
        uint4 raw[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int slot = k0 + j < a.topk ? s_slot[k0 + j] : -1;
          raw[j] = make_uint4(0, 0, 0, 0);
          if (slot >= 0 && LPLB_CHECKED(slot, (long long)a.n_tokens * a.topk, a.status + kMoeBoundsBase, kPhRedirect))
            raw[j] = __ldcg(reinterpret_cast<const uint4*>(a.comb + (size_t)slot * a.hidden) + v);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float w = (k0 + j < a.topk && s_slot[k0 + j] >= 0) ? s_w[k0 + j] : 0.f;  // dropped pair: no term
          const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw[j]);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float2 f = __bfloat1622float2(h[q]);
            acc[2 * q] += w * f.x;
            acc[2 * q + 1] += w * f.y;
          }
        }
      }
      uint4 o;
      o.x = pack_bf16(acc[0], acc[1]);
      o.y = pack_bf16(acc[2], acc[3]);
      o.z = pack_bf16(acc[4], acc[5]);
      o.w = pack_bf16(acc[6], acc[7]);
      reinterpret_cast<uint4*>(a.out + (size_t)t * a.hidden)[v] = o;
    }
  }
}

}  // namespace moe
}  // namespace lplb
