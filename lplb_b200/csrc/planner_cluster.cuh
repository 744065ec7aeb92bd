// Planner step of one thread-block cluster (sm_100a): the step of fused_run_kernel for batches that
// the 16 SMs of a cluster can count.
//
//   CTA 0 ("solver"):     waits for the workers' counts, exchanges them with the peers, solves the LPs and
//                         sends every worker the quotas of the replicated experts.
//   CTAs 1.. ("workers"): count a slice of the indices, send the counts, rewrite at once what selects an expert
//                         without a replica, and the rest when the quotas are there.
//
// What bounds a step is its chain of latencies, and in the grid-wide kernel seven of them are trips through
// L2 (launch number, returning atomics, arrival, the solver's look at it, totals, quotas, and a wait
// of every worker for the slowest).  Here a message is one trip from shared memory to shared memory (st.async),
// counted in by the receiver's mbarrier: the workers' counts go to a row each in the solver's memory, which adds them
// up and finds every worker's first ordinal by the way, and the quotas come back with it.  Only
// replicated experts need either, so most indices are rewritten while the LP is solved.  The
// hardware schedules a cluster as a whole, so the launch need not be cooperative and can start early.
#pragma once

#include "planner_kernels.cuh"
#include "tcgen05.cuh"

namespace lplb {

constexpr int kClusterMaxCtas = 16;       // the largest cluster that sm_100a schedules
constexpr uint32_t kNoReplica = 0xFFFF;   // physical ids in 16 bits: there are at most two per expert
constexpr int kClusterMaxExperts = 1024;  // a row of counts per worker in the solver's shared memory
// Indices per worker before a step takes a larger cluster.  2 / 4 / 8 / 16 CTAs, one after the other and from a graph, us: 256
// indices 15.1 each, 18.5 / 17.7 / 17.6 / 18.9; 1,024 15.8 each, 20.8 / 18.7 / 18.7 / 18.5; 2,048 16.7 / 16.2 / 16.2 / 15.9, 20.9 each; 4,096 15.8 /
// 14.9 / 14.5 / 14.2, 19.6 / 19.1 / 18.4 / 17.8.
constexpr long long kClusterShare = 256;
// Indices of a result in host memory: a worker writes its slice in two passes, each with holes where the other writes, so every
// line crosses PCIe in pieces, from 15 SMs.  Ids and result in pinned memory, one call and the wait for it, grid / cluster, us:
// 8 ranks 256 experts 8,192 indices 29.5 / 26.6, 14,336 27.9 / 27.0, 16,384 30.0 / 31.3, 32,768 35.2 / 44.4, 131,072 64.9 / 114;
// 512 experts 16,384 32.0 / 31.5; 16 ranks 12,288 31.6 / 31.2, 16,384 34.9 / 36.1; 32 ranks 15,200 44.3 / 43.4.  Ids alone may be there
// whatever their number (32,768 27.3 / 26.2, 131,072 41.8 / 41.2).
constexpr long long kClusterHostResult = 15360;
constexpr int kClusterAhead = 2;          // indices of one thread on their way at once

// Threads of a CTA.  With 512 the solver CTA keeps the first kBlock, and the registers of the others, which exit; the solvers
// of several warps are slower that way (16 ranks 8.0 -> 8.9 us, 32 ranks 11.0 -> 12.3, from the same source without spills).
__host__ __device__ constexpr int cluster_threads(int gp) { return gp == -1 ? 512 : 256; }
// Indices of one worker at most (8 bytes of shared memory each).
__host__ __device__ constexpr int cluster_max_slice(int gp) { return gp == -1 ? 10240 : gp == -2 ? 2560 : 1024; }
// Indices of one worker up to which the cluster is the faster one: where a step and a lookup of its result, one after the other, replayed
// from a graph behind a copy of the ids, and as single calls that are waited for, together stop gaining.  With groups of 8 ranks this
// depends on how many experts have a replica, whose tokens a worker handles twice.  Grid / cluster of 16, us, the three in
// this order, at the last size that gains and the first that loses:
//   1 of 32 (512 experts)   131,072: 20.5/18.5 22.6/22.6 29.9/29.3   -
//   1 of 16 (256 experts)   114,688: 19.5/18.5 22.6/23.5 28.9/28.6   131,072: 18.5/18.5 20.5/22.6 27.9/29.1
//   1 of 8 (256 experts)     81,920: 19.8/17.8 22.0/22.6 28.9/28.4    98,304: 19.2/18.5 20.8/22.6 28.6/28.7
//   1 of 4 (256 experts)     65,536: 20.6/19.2 22.6/23.3 29.9/29.7    81,920: 19.4/19.2 21.5/23.9 29.9/31.5
//   1 of 2 (256 experts)     16,384: 20.1/17.8 20.8/21.4 31.9/30.6    32,768: 18.5/18.4 19.5/21.5 28.6/29.7
//   all (48 experts)         32,768: 17.8/15.8 19.2/19.9 27.6/27.1    65,536: 17.1/16.5 19.4/21.2 26.7/27.4
//   16 ranks                 38,400: 22.6/20.6 23.7/23.7 32.0/31.4   32 ranks 15,360: 28.0/24.0 29.1/28.0 34.4/33.7
// Above those two the kernel alone loses (16 ranks 65,536 indices 13.9 / 17.2, 32 ranks 32,768 15.8 / 17.4), though a step and a lookup
// of 32 ranks gains one after the other (32,768: 24.6 / 22.6, from a graph 28.2 / 28.6).
__host__ __device__ constexpr int cluster_paying_slice(int gp, int e, int n_rep) {
  int slice = cluster_max_slice(gp);
  if (gp == -1)
    for (int share = 32 * n_rep; share > e && slice > 2048; share /= 2) slice -= 2048;
  return slice;
}

__host__ __device__ inline int cluster_row(int e) { return (e + 3) & ~3; }  // a row of counts, in words: whole messages
__host__ __device__ inline int cluster_slice(long long n, int n_workers, int threads) {  // indices of a worker, in whole rounds of its threads
  const long long round = (long long)n_workers * threads;
  return (int)((n + round - 1) / round) * threads;
}
// Experts with a replica, at most.
__host__ __device__ inline int cluster_replicated(const Topo& tp) { return tp.n_group * tp.g * tp.c * tp.d; }
__host__ __device__ inline size_t cluster_worker_smem(const Topo& tp, long long n, int n_workers, int threads) {
  return sizeof(int) * (3 * (size_t)cluster_row(tp.e) + 4 * (size_t)cluster_replicated(tp)) +
         sizeof(uint2) * (size_t)cluster_slice(n, n_workers, threads);
}
// In the solver's shared memory, in words: where the replicated experts' totals are, and the bundle sums behind them.
__host__ __device__ inline size_t cluster_total_at(const Topo& tp, int n_workers) {
  return (size_t)cluster_row(tp.e) * (n_workers + 3) + (((size_t)cluster_replicated(tp) * (n_workers + 2) + 1) & ~(size_t)1);
}
__host__ __device__ inline size_t cluster_solver_words(const Topo& tp, int n_workers) {
  return cluster_total_at(tp, n_workers) + 2 * (size_t)cluster_replicated(tp);
}

__device__ __forceinline__ void st_async_v4(uint32_t addr, uint32_t bar, int4 v) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr),
               "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// even_pick with the division by `total` turned into a multiplication by `inverse` = (2^32 - 1) / total.
__device__ __forceinline__ bool even_pick(unsigned k, unsigned quota, unsigned total, unsigned inverse) {
  if (quota >= total) return true;
  if (quota == 0) return false;
  if (total > 65536u) return even_pick(k, quota, total);
  const unsigned x = k * quota;  // below 2^32
  unsigned rem = x - __umulhi(x, inverse) * total;  // the quotient is at most two short
  if (rem >= total) rem -= total;
  if (rem >= total) rem -= total;
  return rem + quota >= total;
}

// Waits for the first phase of `bar`; false when `budget_ns` ran out.
__device__ __forceinline__ bool wait_messages(uint32_t bar, uint64_t budget_ns) {
  const uint32_t nap_ns = (uint32_t)(budget_ns < sm100::kSuspendNs ? budget_ns : sm100::kSuspendNs);
  if (sm100::mbar_try_wait_cluster(bar, 0, nap_ns)) return true;
  const uint64_t t0 = global_timer_ns();
  do {
    if (sm100::mbar_try_wait_cluster(bar, 0, nap_ns)) return true;
  } while (global_timer_ns() - t0 <= budget_ns);
  return false;
}

// A CTA whose wait has run out may not leave before the messages that it stopped waiting for are there: they are stores to its
// shared memory.  All have been issued when it gets here (the cluster barrier), so this has nothing to do with the caller's
// budget, which may be as short as the caller likes.
constexpr uint64_t kLandingNs = 1000000000;
__device__ __forceinline__ void await_landing(uint32_t bar) { wait_messages(bar, kLandingNs); }

// Threads wait each for themselves, so one may give up on what another still sees arrive: whichever does so first reports it,
// once per CTA.
__device__ __forceinline__ void report_late(bool late, int* reported, int* status, int code, int phase, int detail) {
  if (late && atomicExch(reported, 1) == 0) {
    atomicAdd(&status[kStTimeouts], 1);
    raise_status(status, code, phase, detail);
  }
}

// Numbers the experts with a replica in ascending order: has(j, i) and put(j, i, number) of the calling thread's j-th
// expert i = j T + thread.  Called by the first T threads of a CTA, all that have not exited; `counts` is
// kNumberWords of shared memory.
constexpr int kNumberWords = kClusterMaxExperts / 32;
template <int T, typename Has, typename Put>
__device__ __forceinline__ void number_replicated(int e, int* counts, Has has, Put put) {
  static_assert(kNumberWords == 32, "one count per lane");
  constexpr int kRounds = (kClusterMaxExperts + T - 1) / T;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned mine[kRounds];
#pragma unroll
  for (int j = 0; j < kRounds; ++j) {
    const int i = j * T + threadIdx.x;
    mine[j] = __ballot_sync(0xffffffffu, i < e && has(j, i));
    if (lane == 0 && j * T + 32 * warp < kClusterMaxExperts) counts[j * (T / 32) + warp] = __popc(mine[j]);
  }
  __syncthreads();
  int before = counts[lane];
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int up = __shfl_up_sync(0xffffffffu, before, o);
    if (lane >= o) before += up;
  }
  before -= counts[lane];
#pragma unroll
  for (int j = 0; j < kRounds; ++j) {
    const int first = __shfl_sync(0xffffffffu, before, (j * (T / 32) + warp) & 31);
    if ((mine[j] >> lane) & 1u) put(j, j * T + threadIdx.x, first + __popc(mine[j] & ((1u << lane) - 1u)));
  }
}

// What bounds this CTA besides the solve is code that runs once per launch and comes from L2 line by line (other
// kernels run in between), so the way from the counts to the solve and from the shares to the workers is kept short:
// the solving warps hold their tables and the saved iterate in registers before the counts are there, and the other
// warps prepare what goes out with the quotas meanwhile.
template <int GP, int D>
__device__ __forceinline__ void cluster_solver(const Topo& tp, const Exchange& ex, IpmParams prm, Workspace* ws,
                                               float* __restrict__ probs, Counter avail, int* status, int n_workers,
                                               unsigned long long timeout_ns, unsigned long long* __restrict__ trace, int* smem,
                                               uint64_t* bar, int* counts, int* reported) {
  const int e = tp.e, row = cluster_row(e), n_rep = cluster_replicated(tp), warp = threadIdx.x >> 5;
  const bool tracing = trace != nullptr && threadIdx.x == 0;
  int* rows = smem;                                    // [n_workers][row]
  int* vec = rows + (size_t)n_workers * row;           // [e] totals, of all ranks if there are several
  float* share = reinterpret_cast<float*>(vec + row);  // [n_group * g * d], at most e
  int* slots = reinterpret_cast<int*>(share) + row;    // [e] where an expert's count goes in `bundle`
  int* rep_expert = slots + row;                       // [n_rep]
  int* rep_edge = rep_expert + n_rep;                  // [n_rep]
  int* first_ordinal = rep_edge + n_rep;               // [n_workers][n_rep] of a worker's tokens for the expert
  int2* rep_total = reinterpret_cast<int2*>(smem + cluster_total_at(tp, n_workers));  // [n_rep] rank-local tokens, (2^32 - 1) / that
  int* bundle = smem + cluster_solver_words(tp, n_workers);
  __shared__ ExchangeShared xs;
  __shared__ uint32_t s_epoch;
  const int n_bundle = tp.n_group * tp.g * (tp.d + 1);
  if (tracing) trace[0] = global_timer_ns();
  // this thread's experts: where their counts go, and which are replicated
  constexpr int kMine = kClusterMaxExperts / kBlock;
  int slot_of[kMine], replica[kMine], edge[kMine];
#pragma unroll
  for (int j = 0; j < kMine; ++j) {
    const int i = j * kBlock + threadIdx.x;
    slot_of[j] = i < e ? tp.log2slot[i] : 0;
    replica[j] = i < e ? tp.log2phy[2 * i + 1] : -1;
    edge[j] = i < e ? tp.log2edge[i] : -1;
  }
  // Warps from `first_sender` on do not solve: they prepare and send the results.  Where most solve, all do it afterwards.
  using Step = TileStep<GP>;
  const int solving = Step::solving(tp), first_sender = solving <= kWarps / 2 ? solving : 0;
  const bool rehearsal = ex.n_ranks <= 1 && Step::rehearses(tp), rehearses = rehearsal && warp == Step::kRehearsing;
  const int n_threads = rehearsal ? kBlock - 32 : kBlock;  // those that do not rehearse
  const TileLane mine = load_step_lane<GP, D, true>(tp, prm, rehearses, status);
  // The rows start at zero: what is summed when the wait for them runs out is a part of the counts and nothing else.  (The tables
  // are on their way meanwhile.)
  for (int i = threadIdx.x; i < n_workers * row / 4; i += kBlock) reinterpret_cast<int4*>(rows)[i] = int4{0, 0, 0, 0};
  const uint32_t my_bar = sm100::smem_u32(bar);
  if (threadIdx.x == 0) {
    *reported = 0;
    sm100::mbar_init(my_bar, 1);
    sm100::mbar_expect_tx(my_bar, (uint32_t)(n_workers * row) * sizeof(int));
    sm100::fence_barrier_init();
    s_epoch = ld_acquire_gpu(&ws->epoch) + 1;
    status[kStLpIters] = status[kStGapPpb] = 0;
  }
  __syncwarp();
  cluster_arrive();
  for (int i = threadIdx.x; i < n_bundle; i += kBlock) bundle[i] = 0;
  for (int i = threadIdx.x; i < n_rep; i += kBlock) rep_expert[i] = rep_edge[i] = -1;
  exchange_prepare(ex, &xs);
  number_replicated<kBlock>(
      e, counts, [&](int j, int) { return replica[j] >= 0; },
      [&](int j, int i, int k) {
        if (k >= n_rep) return;
        rep_expert[k] = i;
        rep_edge[k] = edge[j];
      });
#pragma unroll
  for (int j = 0; j < kMine; ++j)
    if (j * kBlock + (int)threadIdx.x < e) slots[j * kBlock + threadIdx.x] = slot_of[j];
  __shared__ int made_up[GP == -1 ? 8 * (D + 1) : 1];
  if (GP == -1) make_up_loads(made_up, 8 * (D + 1));
  __syncthreads();
  const uint32_t epoch = s_epoch;
  __syncwarp();
  cluster_wait();
  bool late = false;
  if (!rehearses) {
    late = !wait_messages(my_bar, timeout_ns);
    if (tracing) trace[2] = global_timer_ns();
    report_late(late, reported, status, kErrGridTimeout, kPhCount, 0);
#pragma unroll 1
    for (int i = threadIdx.x; i < e; i += n_threads) {
      const int slot = slots[i];
      int total = 0;
#pragma unroll 1
      for (int w0 = 0; w0 < n_workers; w0 += 8) {
        int c[8];
#pragma unroll
        for (int w = 0; w < 8; ++w) c[w] = w0 + w < n_workers ? rows[(w0 + w) * row + i] : 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) total += c[w];
      }
      vec[i] = total;
      if (ex.n_ranks <= 1 && total && LPLB_CHECKED(slot, n_bundle, status, kPhSolve)) atomicAdd(&bundle[slot], total);
    }
    sync_threads(n_threads);
    if (ex.n_ranks > 1) {
      exchange_step(ex, &xs, epoch, tp, vec, prm, status, trace);
#pragma unroll 1
      for (int i = threadIdx.x; i < e; i += kBlock)
        if (vec[i] && LPLB_CHECKED(slots[i], n_bundle, status, kPhSolve)) atomicAdd(&bundle[slots[i]], vec[i]);
      __syncthreads();
    }
    if (tracing) trace[3] = global_timer_ns();
  }
  if (rehearses || warp < solving)
    solve_step_tiles<GP, D, true>(bundle, made_up, rehearses, tp, prm, mine, probs, share, avail, status, [&] {
      if (!rehearses && first_sender > 0) asm volatile("bar.arrive 3, %0;" ::"r"(n_threads) : "memory");
    });
  const int n_senders = n_threads - first_sender * 32, sender = (int)threadIdx.x - first_sender * 32;
  auto prepare = [&] {
    if (sender == 0) {  // bookkeeping, and what the next launch of the grid-wide kernel finds
      ws->arrive[(epoch & 1) ^ 1] = 0;
      ws->epoch = epoch;
      atomicAdd(&status[kStCalls], 1);
    }
    int *other = ws_total(ws, (epoch & 1) ^ 1, e), *glob = ws_global(ws, e);
#pragma unroll 1
    for (int i = sender; i < e; i += n_senders) {
      other[i] = 0;
      glob[i] = vec[i];  // a copy for the host
    }
#pragma unroll 1
    for (int k = sender; k < n_rep; k += n_senders) {
      const int expert = rep_expert[k];
      int total = 0;
#pragma unroll 1
      for (int w = 0; w < n_workers; ++w) {
        first_ordinal[w * n_rep + k] = total;
        if (expert >= 0) total += rows[w * row + expert];
      }
      rep_total[k] = make_int2(total, (int)(0xFFFFFFFFu / (unsigned)max(total, 1)));
    }
  };
  auto send = [&] {
    const uint32_t res = sm100::smem_u32(smem + 3 * (size_t)row);  // where a worker keeps its results
    int w = sender / n_rep, k = sender - w * n_rep;
    const int step_w = n_senders / n_rep, step_k = n_senders - step_w * n_rep;
#pragma unroll 1
    while (w < n_workers) {
      const int2 total = rep_total[k];
      const int4 msg = make_int4(quota_of(total.x, rep_edge[k], share), total.x, first_ordinal[w * n_rep + k], total.y);
      st_async_v4(sm100::map_to_rank(res + 16 * k, w + 1), sm100::map_to_rank(my_bar, w + 1), msg);
      k += step_k;
      w += step_w;
      if (k >= n_rep) {
        k -= n_rep;
        ++w;
      }
    }
  };
  if (warp >= first_sender && !rehearses) {
    prepare();
    asm volatile("bar.sync 3, %0;" ::"r"(n_threads) : "memory");
    send();
  }
  if (trace != nullptr && sender == 0) trace[4] = global_timer_ns();
  __syncwarp();
  cluster_arrive();
  cluster_wait();  // the workers have what was sent; nobody's shared memory goes before that
  if (late) await_landing(my_bar);
}

// What the workers need, in one place: the first of their instructions wait for it.
template <typename IdxT>
struct ClusterHead {
  const IdxT* idx;
  IdxT* out;
  const int2* log2phy;
  long long n;
  int slice;  // indices of a worker
  int e, n_rep;
};

// A worker's code comes from L2 line by line too, so its loads are issued before anything else.
template <int T, typename IdxT>
__device__ __forceinline__ void cluster_worker(const ClusterHead<IdxT>& head, Workspace* ws, int* status, int q, int n_workers,
                                               unsigned long long timeout_ns, unsigned long long* __restrict__ trace, int* smem,
                                               uint64_t* bar, int* counts, int* reported) {
  const long long begin = min((long long)q * head.slice, head.n);
  const int m = (int)min((long long)head.slice, head.n - begin), e = head.e, row = cluster_row(e), n_rep = head.n_rep;
  const IdxT* __restrict__ idx = head.idx + begin;
  IdxT* __restrict__ out = head.out + begin;
  uint32_t* phys = reinterpret_cast<uint32_t*>(smem);    // [row] original, and in the upper half the replica or kNoReplica
  int* hist = smem + row;                                // [row]
  int* number = hist + row;                              // [row] of the experts with a replica
  int4* res = reinterpret_cast<int4*>(number + row);     // [n_rep] quota, rank-local total, this worker's first ordinal, (2^32 - 1) / total
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint2* later = reinterpret_cast<uint2*>(res + n_rep) + warp * (head.slice / (T / 32));  // what waits for a quota, a list per warp
  const bool tracing = trace != nullptr && threadIdx.x == 0 && q == 0;
  IdxT ahead[kClusterAhead];
  auto load = [&](int first) {
#pragma unroll
    for (int j = 0; j < kClusterAhead; ++j) ahead[j] = first + j * T < m ? __ldcv(idx + first + j * T) : (IdxT)-1;
  };
  load(threadIdx.x);
  constexpr int kRounds = (kClusterMaxExperts + T - 1) / T;
  int2 table[kRounds];
#pragma unroll
  for (int j = 0; j < kRounds; ++j)
    if (j * T + (int)threadIdx.x < e) table[j] = head.log2phy[j * T + threadIdx.x];
  const uint32_t bar_result = sm100::smem_u32(bar);
  if (threadIdx.x == 0) {
    *reported = 0;
    sm100::mbar_init(bar_result, 1);
    sm100::mbar_expect_tx(bar_result, (uint32_t)n_rep * 16);
    sm100::fence_barrier_init();
  }
  __syncwarp();
  cluster_arrive();
#pragma unroll
  for (int j = 0; j < kRounds; ++j) {
    const int i = j * T + threadIdx.x;
    if (i < row) hist[i] = 0;
    if (i < e) phys[i] = (uint32_t)(table[j].x & 0xFFFF) | (uint32_t)table[j].y << 16;
  }
  __syncthreads();
  int bad = 0;
  int n_later = 0;
  for (int i0 = threadIdx.x; i0 - lane < m; i0 += kClusterAhead * T) {
    // one kind of access after the other, so that each is under way for all indices at once
    int v[kClusterAhead], k[kClusterAhead];
    uint32_t ph[kClusterAhead];
#pragma unroll
    for (int j = 0; j < kClusterAhead; ++j) {
      const bool valid = ahead[j] >= 0 && ahead[j] < e;
      bad += !valid && ahead[j] != -1;
      v[j] = valid ? (int)ahead[j] : -1;
    }
    load(i0 + kClusterAhead * T);
#pragma unroll
    for (int j = 0; j < kClusterAhead; ++j) {
      ph[j] = kNoReplica << 16;
      if (v[j] >= 0) {
        ph[j] = phys[v[j]];
        k[j] = atomicAdd(&hist[v[j]], 1);
      }
    }
#pragma unroll
    for (int j = 0; j < kClusterAhead; ++j) {
      const int i = i0 + j * T;
      const bool waits = ph[j] >> 16 != kNoReplica;
      const unsigned all = __ballot_sync(0xffffffffu, waits);
      if (waits) {  // place within the slice; expert, ordinal within the slice
        later[n_later + __popc(all & ((1u << lane) - 1u))] = make_uint2((uint32_t)i, (uint32_t)v[j] << 20 | (uint32_t)k[j]);
      } else if (i < m) {
        out[i] = (IdxT)(v[j] >= 0 ? (int)(ph[j] & 0xFFFFu) : -1);
      }
      n_later += __popc(all);
    }
  }
  static_assert(cluster_max_slice(-1) < 1 << 20 && kClusterMaxExperts <= 1 << 12, "packing of `later`");
  __syncwarp();
  cluster_wait();  // the solver's barrier is ready
  __syncthreads();
  {
    const uint32_t solver_bar = sm100::map_to_rank(bar_result, 0);  // the same place in its shared memory
    const uint32_t to = sm100::map_to_rank(sm100::smem_u32(smem + (size_t)q * row), 0);
    for (int i = threadIdx.x; i < row / 4; i += T) st_async_v4(to + 16 * i, solver_bar, reinterpret_cast<const int4*>(hist)[i]);
  }
  if (tracing) trace[1] = global_timer_ns();
  if (bad) {
    atomicAdd(&status[kStBadIdx], bad);
    raise_status(status, kErrBadIndex, kPhCount, bad);
  }
  number_replicated<T>(
      e, counts, [&](int, int i) { return phys[i] >> 16 != kNoReplica; }, [&](int, int i, int k) { number[i] = min(k, n_rep - 1); });
  __syncthreads();
  // Two rounds through the same code: the first, on one entry, writes nothing and only fetches it.
  bool late = false;
#pragma unroll 1
  for (int round = 0; round < 2; ++round) {
    const int stop = round == 0 ? min(n_later, 1) : n_later;
    if (round == 1) {
      late = !wait_messages(bar_result, timeout_ns);
      __syncwarp();
      cluster_arrive();
    }
#pragma unroll 1
    for (int at = lane; at < stop; at += 32) {
      const uint2 it = later[at];
      const int v = (int)(it.y >> 20);
      const unsigned k = it.y & 0xFFFFFu;
      const uint32_t ph = phys[v];
      const int4 r = res[number[v]];
      // without shares half of a replicated expert's tokens stay
      const bool stay = late ? k & 1u : even_pick((unsigned)r.z + k, (unsigned)r.x, (unsigned)r.y, (unsigned)r.w);
      if (round == 1) out[it.x] = (IdxT)(int)(stay ? ph & 0xFFFFu : ph >> 16);
    }
  }
  report_late(late, reported, status, kErrLpTimeout, kPhRedirect, q);
  if (trace != nullptr) {  // tracing only: find the worker that leaves last
    __syncthreads();
    if (tracing) trace[5] = global_timer_ns();
    if (threadIdx.x == 0) {
      __threadfence();
      if (atomicAdd(&ws->exit_cnt, 1u) == (unsigned)n_workers - 1) {
        ws->exit_cnt = 0;
        trace[6] = global_timer_ns();
      }
    }
  }
  __syncwarp();
  cluster_wait();
  if (late) await_landing(bar_result);
}

// It starts early, but does not let its successor do so: a MoE pass behind it, whose kernels then all started and waited while it
// ran, took 4.6 us longer (64 tokens x 2048: behind the grid-wide step 148, here 147, with early successors 153).
//
// Grid = one cluster: a solver CTA and gridDim.x - 1 worker CTAs.  Shapes of the tile solver for up to 32 ranks (GP = -1, -2, -4;
// with 64 a step is the solve: 52.7 us grid-wide against 53.3 here when it was measured, with the solver as it was when a call of it
// took 51 us; 46 now).
template <int GP, int D, typename IdxT>
__global__ void __launch_bounds__(cluster_threads(GP), 1) cluster_run_kernel(const ClusterHead<IdxT> head, unsigned long long timeout_ns,
                                                                               unsigned long long* __restrict__ trace, int* status,
                                                                               Workspace* ws, Topo tp, Exchange ex, IpmParams prm,
                                                                               float* __restrict__ probs, Counter avail) {
  extern __shared__ __align__(16) int smem[];
  __shared__ __align__(8) uint64_t bar;       // the solver's: counts; a worker's: results
  __shared__ int counts[kNumberWords];
  __shared__ int reported;  // that a wait of this CTA ran out
  wait_predecessors();
  constexpr int T = cluster_threads(GP);
  const int n_workers = (int)gridDim.x - 1;
  if (blockIdx.x == 0) {
    if constexpr (T > kBlock) {
      // 128 registers a thread at launch: the solving warps take 216, those that leave keep 40 (256 x (216 + 40) = 512 x 128)
      static_assert(T == 512 && kBlock == 256, "register split");
      if (threadIdx.x >= kBlock) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
        return;
      }
      asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
    }
    cluster_solver<GP, D>(tp, ex, prm, ws, probs, avail, status, n_workers, timeout_ns, trace, smem, &bar, counts, &reported);
  } else {
    cluster_worker<T, IdxT>(head, ws, status, (int)blockIdx.x - 1, n_workers, timeout_ns, trace, smem, &bar, counts, &reported);
  }
}

}  // namespace lplb
