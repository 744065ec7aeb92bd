// Expert placement from the load history and every table derived from it, in one launch (sm_100a).
//
// The same decisions as the host balancer (lplb_b200/eplb.py, lplb_b200/mapping.py), item by item:
// expert groups to nodes, experts to the ranks of a node, both heaviest first into the lightest
// pack with room (reference lplb/eplb.py:6-46, :80-148), then the tables (reference
// lplb/planner.py:115-182).  Loads are float64 on both sides.  A rank's load grows item by item, in
// the same order on both; a group's load is added in another order than on the host, which gives
// the same sum as long as no partial sum can pass 2^53.  Where one could, the kernel writes no table
// and reports it, and the host places the experts.  So the results are identical.
//
// One CTA.  What bounds it is the greedy packing, a chain of dependent rounds: a warp holds the
// packs (one per lane up to 32), ranks them by load, and hands out an item to each at once as
// far as the order of the items allows it.  The orders come from counting, for every
// expert, the experts in front of it.  256 experts on 8 ranks: 21 us (one item after the
// other 27 to 32), 35 us for the whole call until the host has its word (39 us with a wait for the stream and a kernel of
// its own that cleared the saved iterates); on the host, some twenty tensor operations per expert, 8.9 ms.
#include "place_api.h"

#include <stdint.h>

namespace lplb {

namespace {

constexpr int kPlaceThreads = 1024;
constexpr unsigned kAll = 0xffffffffu;

struct Shared {
  double* w;      // [E] loads in node-major order
  double* gw;     // [n_group] group loads
  double* load;   // [packs] of one packing, per node
  int* fill;      // [packs]
  int* order;     // [E] items of a packing, heaviest first
  int* nlog2log;  // [E]
  int* own;       // [E] expert in every rank's own slots
};

size_t shared_bytes(const PlaceArgs& a) {
  const size_t e = a.n_logical, packs = a.ep_size > a.n_group ? a.ep_size : a.n_group;
  return 8 * (e + a.n_group + packs) + 4 * (packs + 3 * e);
}

__device__ __forceinline__ double load_of(const PlaceArgs& a, int e) {
  return a.is64 ? (double)((const long long*)a.history)[e] : (double)((const int*)a.history)[e];
}

// Unsigned order of the result = order of the doubles.
__device__ __forceinline__ unsigned long long ordered(double x) {
  const long long b = __double_as_longlong(x);
  return (unsigned long long)b ^ ((unsigned long long)(b >> 63) | 0x8000000000000000ull);
}

// order[k] = the item with k items in front of it: heavier ones, and equal ones of lower index.
// Rows of `n` items each, `rows` of them, by all threads of the CTA; several neighbouring threads
// share an item where there are threads to spare (256 items: one 64-step pass instead of 256 steps).
__device__ void sort_rows(const double* w, int* order, int rows, int n) {
  int parts = 1;
  while (parts < 32 && parts * 2 * rows * n <= kPlaceThreads) parts *= 2;
  const int part = threadIdx.x & (parts - 1);
  for (int base_slot = 0; base_slot < rows * n * parts; base_slot += kPlaceThreads) {
    const int i = (base_slot + (int)threadIdx.x) / parts;
    const bool item = i < rows * n;
    const int base = item ? i / n * n : 0, me = item ? i - base : 0;
    const double mine = w[base + me];
    int front = 0;
    for (int j = part; j < n; j += parts) {
      const double other = w[base + j];
      front += other > mine || (other == mine && j < me);
    }
    for (int o = parts / 2; o > 0; o >>= 1) front += __shfl_xor_sync(kAll, front, o);
    if (item && part == 0) order[base + front] = me;
  }
}

// One warp: items order[0], order[1], ... each into the lightest of `packs` packs of `cap` items that
// has room, the lowest-numbered one among equals.  put(item, pack, position in the pack).
template <typename Put>
__device__ void pack_items(const double* w, const int* order, int n, int packs, int cap, double* load, int* fill,
                           Put put) {
  const int lane = threadIdx.x & 31;
  if (packs == 1) {
    for (int k = lane; k < n; k += 32) put(order[k], 0, k);
    return;
  }
  if (packs <= 32) {
    // A pack per lane, in registers.  A round hands out one item to each of the lightest packs at once: the
    // j-th next item goes to the j-th lightest pack, as one after the other it would, as long as that
    // pack is lighter than every pack is after its item of this round.  So many items of the round
    // count, at least the first.  (Loads drawn like gate logits: 34 rounds for 256 items on 8 packs; a
    // Zipf history 99.)
    unsigned long long* keys = reinterpret_cast<unsigned long long*>(load);
    double mine = 0.0;
    int held = 0;
    for (int step = 0; step < n;) {
      const bool room = lane < packs && held < cap;
      const unsigned long long key = room ? ordered(mine) : ~0ull;
      if (lane < packs) {
        keys[lane] = key;
        fill[lane] = cap - held;
      }
      __syncwarp();
      int rank = 0;  // packs with room in front of this one
#pragma unroll 4
      for (int q = 0; q < packs; ++q) {
        const unsigned long long other = keys[q];
        rank += other < key || (other == key && q < lane);
      }
      const int takers = min(__popc(__ballot_sync(kAll, room)), n - step);
      const bool takes = room && rank < takers;
      const int item = order[step + (takes ? rank : 0)];
      const double weight = w[item], grown = mine + weight;
      if (__ballot_sync(kAll, takes && rank == 0 && weight == 0.0) && w[order[n - 1]] == 0.0) {
        // nothing but empty items left: they fill up the packs, the lightest first
        int at = step;
        for (int q = 0; q < packs; ++q) {
          const unsigned long long other = keys[q];
          if (other < key || (other == key && q < lane)) at += fill[q];
        }
        if (room)
          for (int k = held; k < cap && at < n; ++k, ++at) put(order[at], lane, k);
        return;
      }
      const unsigned long long after = takes ? ordered(grown) : ~0ull;
      const unsigned hi = (unsigned)(after >> 32), least_hi = __reduce_min_sync(kAll, hi);
      const unsigned least_lo = __reduce_min_sync(kAll, hi == least_hi ? (unsigned)after : ~0u);
      const bool counts = takes && (rank == 0 || key < ((unsigned long long)least_hi << 32 | least_lo));
      step += __popc(__ballot_sync(kAll, counts));
      if (counts) {
        put(item, lane, held);
        mine = grown;
        ++held;
      }
    }
    return;
  }
  for (int p = lane; p < packs; p += 32) {
    load[p] = 0.0;
    fill[p] = 0;
  }
  __syncwarp();
  for (int step = 0; step < n; ++step) {
    unsigned long long best = ~0ull;
    int best_pack = 0x7fffffff;
    for (int p = lane; p < packs; p += 32) {
      if (fill[p] >= cap) continue;
      const unsigned long long key = ordered(load[p]);
      if (best_pack == 0x7fffffff || key < best) {
        best = key;
        best_pack = p;
      }
    }
    const bool room = best_pack != 0x7fffffff;
    const unsigned hi = (unsigned)(best >> 32), lo = (unsigned)best;
    const unsigned least_hi = __reduce_min_sync(kAll, hi);
    const unsigned least_lo = __reduce_min_sync(kAll, hi == least_hi ? lo : ~0u);
    const int pack = (int)__reduce_min_sync(
        kAll, room && hi == least_hi && lo == least_lo ? (unsigned)best_pack : 0x7fffffffu);
    if (lane == 0) {
      const int item = order[step];
      put(item, pack, fill[pack]);
      load[pack] += w[item];
      ++fill[pack];
    }
    __syncwarp();
  }
}

// gw[g] = the load of group g, a warp per group.  Returns whether a partial sum, in some order of
// adding, could pass 2^53 (in a group of the calling warp).
__device__ bool group_loads(const PlaceArgs& a, double* gw, int groups, int per_group) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  bool large = false;
  for (int g = warp; g < groups; g += kPlaceThreads / 32) {
    double sum = 0.0, size = 0.0;
    for (int i = lane; i < per_group; i += 32) {
      const double x = load_of(a, g * per_group + i);
      sum += x;
      size += fabs(x);
    }
    for (int o = 16; o > 0; o >>= 1) {
      sum += __shfl_xor_sync(kAll, sum, o);
      size += __shfl_xor_sync(kAll, size, o);
    }
    if (lane == 0) gw[g] = sum;
    large |= size >= 9007199254740992.0;  // 2^53
  }
  return large;
}

// The last thing the kernel does, called by all threads: whoever sees `outcome` in the host's word sees all that the
// CTA has written, on any stream that gets work after that.
__device__ __forceinline__ void report(const PlaceArgs& a, int outcome) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence_system();
    *reinterpret_cast<volatile int*>(a.report) = outcome;
  }
}

__global__ void __launch_bounds__(kPlaceThreads) place_kernel(const PlaceArgs a) {
  extern __shared__ double sm[];
  __shared__ int uncovered;
  const int tid = threadIdx.x, warp = tid >> 5, n_warps = kPlaceThreads / 32;
  const int E = a.n_logical, ranks = a.ep_size, ll = E / ranks, rep = a.combined * a.dup, pl = ll + rep;
  const int max_packs = ranks > a.n_group ? ranks : a.n_group;
  Shared s;
  s.w = sm;
  s.gw = s.w + E;
  s.load = s.gw + a.n_group;
  s.fill = reinterpret_cast<int*>(s.load + max_packs);
  s.order = s.fill + max_packs;
  s.nlog2log = s.order + E;
  s.own = s.nlog2log + E;

  if (tid == 0) uncovered = 0;
  for (int i = tid; i < a.n_anchor; i += kPlaceThreads) a.anchor_valid[i] = 0;
  if (a.history == nullptr) {  // natural order
    for (int e = tid; e < E; e += kPlaceThreads) s.own[e] = e;
  } else {
    // whole groups to nodes; without groups that divide over the nodes, one group on one node
    const bool hier = a.n_group % a.n_nodes == 0;
    const int groups = hier ? a.n_group : 1, nodes = hier ? a.n_nodes : 1;
    const int per_group = E / groups, groups_per_node = groups / nodes, per_node = E / nodes;
    int* place_of_group = s.own;  // position of the group in node-major order
    if (groups_per_node == 1) {
      for (int g = tid; g < groups; g += kPlaceThreads) place_of_group[g] = g;
    } else {
      const bool inexact = group_loads(a, s.gw, groups, per_group);
      if (__syncthreads_or(inexact)) {
        report(a, kPlaceInexact);
        return;
      }
      sort_rows(s.gw, s.order, 1, groups);
      __syncthreads();
      if (warp == 0)
        pack_items(s.gw, s.order, groups, nodes, groups_per_node, s.load, s.fill,
                   [&](int g, int node, int pos) { place_of_group[g] = node * groups_per_node + pos; });
    }
    __syncthreads();
    for (int e = tid; e < E; e += kPlaceThreads) {
      const int to = place_of_group[e / per_group] * per_group + e % per_group;
      s.nlog2log[to] = e;
      s.w[to] = load_of(a, e);
    }
    __syncthreads();
    const int packs = ranks / nodes;
    if (ll == 1) {
      for (int e = tid; e < E; e += kPlaceThreads) s.own[e] = s.nlog2log[e];
    } else {
      sort_rows(s.w, s.order, nodes, per_node);
      __syncthreads();
      // A pack fills heaviest first, so every rank's own slots are in the order of the history.  The
      // packing warp stores positions; looking the experts up there would put a load on its chain
      // (41 instead of 35 us).
      for (int node = warp; node < nodes; node += n_warps) {
        const int base = node * per_node;
        pack_items(s.w + base, s.order + base, per_node, packs, ll, s.load + node * packs, s.fill + node * packs,
                   [&](int item, int pack, int pos) { s.own[base + pack * ll + pos] = base + item; });
      }
      __syncthreads();
      for (int i = tid; i < E; i += kPlaceThreads) s.own[i] = s.nlog2log[s.own[i]];
    }
  }
  int* slot_of = reinterpret_cast<int*>(s.w);  // the packing is through with the loads
  for (int i = tid; i < E; i += kPlaceThreads)
    if ((unsigned)s.own[i] < (unsigned)E) slot_of[s.own[i]] = i;
  __syncthreads();

  for (int i = tid; i < ranks * pl; i += kPlaceThreads) {
    const int rank = i / pl, slot = i - rank * pl;
    int e;
    if (slot < ll) {
      e = s.own[rank * ll + slot];
      if ((unsigned)e >= (unsigned)E || slot_of[e] != rank * ll + slot) {  // every expert in exactly one own slot
        uncovered = 1;
        continue;
      }
      const int first = slot < rep ? slot % a.dup : a.dup;  // bundle of the slot; dup = not replicated
      int replica = -1;
      if (slot < rep) {
        const int grp = rank / a.g;
        replica = (grp * a.g + a.o2r[(rank - grp * a.g) * a.dup + first]) * pl + ll + slot;
      }
      const int edge = slot < rep ? rank * a.dup + first : -1;
      a.log2phy[2 * e] = a.table_log2phy[2 * e] = i;
      a.log2phy[2 * e + 1] = a.table_log2phy[2 * e + 1] = replica;
      a.logcnt[e] = replica >= 0 ? 2 : 1;
      a.log2edge[e] = a.table_log2edge[e] = edge;
      a.table_log2slot[e] = rank * (a.dup + 1) + first;
    } else {
      const int grp = rank / a.g, at = slot - ll;
      const int src = grp * a.g + a.r2o[(rank - grp * a.g) * a.dup + at % a.dup];
      e = s.own[src * ll + at];
    }
    a.phy2log[i] = a.table_phy2log[i] = e;
  }
  __syncthreads();
  report(a, uncovered ? kPlaceUncovered : kPlaceOk);
}

}  // namespace

cudaError_t launch_place(const PlaceArgs& a, cudaStream_t stream) {
  const size_t bytes = shared_bytes(a);
  const cudaError_t err = cudaFuncSetAttribute(place_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (err != cudaSuccess) return err;
  place_kernel<<<1, kPlaceThreads, bytes, stream>>>(a);
  return cudaGetLastError();
}

size_t place_shared_bytes(const PlaceArgs& a) { return shared_bytes(a); }

}  // namespace lplb
