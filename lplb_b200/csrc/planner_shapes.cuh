// What planner_launch.cu hands to the instantiations of the solving kernels, one per (group size, replicas per
// rank) shape.  Their definitions are in planner_shapes_impl.cuh, which the planner_tiles*.cu, planner_warp*.cu
// and planner_block.cu files instantiate, a few shapes each, so that they compile side by side.  (One file with
// nvcc's --split-compile compiles as fast, but not to the same code every time: of two outcomes for
// moe_launch.cu, by chance, one runs the grouped GEMMs 2 to 3 % slower, 404 and 232 us against 411 and 240.)
#pragma once

#include "planner_api.h"
#include "planner_cluster.cuh"

namespace lplb {

inline int padded_dup(int d) { return d <= 4 ? d : 8; }
inline size_t fused_smem(int e) { return sizeof(int) * 5 * (size_t)e; }
inline size_t bundle_smem(const Topo& tp) { return sizeof(int) * (size_t)tp.n_group * tp.g * (tp.d + 1); }
// bundle sums followed by the solver's scratch area, if it has one
template <int GP>
size_t solver_smem(const Topo& tp, int teams = kWarps) {
  if constexpr (GP > 0) return bundle_smem(tp);
  else return bundle_bytes_aligned(tp.n_group * tp.g, tp.d) +
              (GP == 0 ? block_solver_smem_bytes(tp.g, padded_dup(tp.d)) : tile_solver_smem_bytes(tp.g, tp.d, GP == -1 ? teams : 1));
}

template <int GP>
size_t cluster_smem(const Topo& tp, long long n, int n_cta) {
  const size_t solver = sizeof(int) * cluster_solver_words(tp, n_cta - 1) + solver_smem<GP>(tp);
  const size_t worker = cluster_worker_smem(tp, n, n_cta - 1, cluster_threads(GP));
  return solver > worker ? solver : worker;
}

template <typename K>
cudaError_t allow_smem(K kernel, size_t bytes) {
  if (bytes <= 48 * 1024) return cudaSuccess;
  if (bytes > 227 * 1024) return cudaErrorInvalidValue;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

struct SolveLaunch {
  const int* workload;
  Topo tp;
  IpmParams prm;
  float* probs;
  float* normalised;
  Counter avail;
  int* status;
  cudaStream_t stream;
  template <int GP, int D>
  cudaError_t operator()() const;
};

template <typename IdxT>
struct FusedLaunch {
  const IdxT* idx;
  long long n;
  Topo tp;
  Exchange ex;
  IpmParams prm;
  Workspace* ws;
  float* probs;
  Counter avail;
  int* status;
  IdxT* out;
  int n_cta;
  unsigned long long grid_timeout_ns;
  unsigned long long* trace;
  int cooperative;
  cudaStream_t stream;
  template <int GP, int D>
  cudaError_t operator()();
};

// The step in one cluster (planner_cluster.cuh).  `fits` non-null: only asks whether the device can run it.
template <typename IdxT>
struct ClusterLaunch {
  const IdxT* idx;
  long long n;
  Topo tp;
  Exchange ex;
  IpmParams prm;
  Workspace* ws;
  float* probs;
  Counter avail;
  int* status;
  IdxT* out;
  int n_cta;
  unsigned long long timeout_ns;
  unsigned long long* trace;
  cudaStream_t stream;
  int* fits;
  template <int GP, int D>
  cudaError_t operator()() const;
};

struct OccupancyQuery {
  Topo tp;
  int is64;
  int* result;
  template <int GP, int D>
  cudaError_t operator()() const;
};

}  // namespace lplb
