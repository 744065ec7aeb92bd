// Definitions of the launches that planner_shapes.cuh declares; included by the files that instantiate them.
#pragma once

#include <atomic>

#include "planner_shapes.cuh"

namespace lplb {

template <int GP, int D>
cudaError_t SolveLaunch::operator()() const {
  const size_t smem = solver_smem<GP>(tp);
  cudaError_t err;
  if constexpr (GP == 8) {
    return cudaErrorInvalidValue;  // groups of 8 ranks are packed in the fused kernel only
  } else if constexpr (GP == 0 || GP < -1) {
    auto kernel = [] {
      if constexpr (GP == 0) return solve_block_kernel<D>;
      else return tile_solve_kernel<-GP, D>;
    }();
    if ((err = allow_smem(kernel, smem)) != cudaSuccess) return err;
    if constexpr (GP == 0) kernel<<<tp.n_group, kBlock, smem, stream>>>(workload, tp, prm, probs, normalised, avail, status);
    else return launch_after(kernel, tp.n_group + 1, kBlock, smem, stream, workload, tp, prm, probs, normalised, avail, status, 1);
  } else {
    // As few solving warps per CTA as still fit the groups on one wave of CTAs.
    constexpr int kPerWarp = GP == -1 ? 1 : 32 / GP;
    int dev = 0, sms = 1;
    err = cudaGetDevice(&dev);
    if (err == cudaSuccess) err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (err != cudaSuccess) return err;
    int warps = 1;
    while (warps < kWarps && (tp.n_group + warps * kPerWarp - 1) / (warps * kPerWarp) > sms) warps *= 2;
    const int per_cta = warps * kPerWarp;
    const int grid = (tp.n_group + per_cta - 1) / per_cta;
    if constexpr (GP == -1) {
      const size_t smem = solver_smem<GP>(tp, warps);
      if ((err = allow_smem(tile_solve_kernel<1, D>, smem)) != cudaSuccess) return err;
      // an early launch, one call after the other: one group 12.5 -> 11.2 us, 64 groups 14.4 -> 12.4; several warps per
      // group 16 ranks 19.8 -> 18.0, 32 ranks 28.1 -> 26.1, 64 ranks 53.5 -> 52.1
      return launch_after(tile_solve_kernel<1, D>, grid + 1, kBlock, smem, stream, workload, tp, prm, probs, normalised, avail,
                          status, warps);
    } else {
      if ((err = allow_smem(solve_kernel<GP, D>, smem)) != cudaSuccess) return err;
      solve_kernel<GP, D><<<grid, kBlock, smem, stream>>>(workload, tp, prm, probs, normalised, avail, status, warps);
    }
  }
  return cudaGetLastError();
}

template <typename IdxT>
template <int GP, int D>
cudaError_t FusedLaunch<IdxT>::operator()() {
  auto kernel = fused_run_kernel<GP, D, IdxT>;
  const size_t smem = fused_smem(tp.e) + solver_smem<GP>(tp);
  cudaError_t err = allow_smem(kernel, smem);
  if (err != cudaSuccess) return err;
  void* args[] = {&idx, &n, &tp, &ex, &prm, &ws, &probs, &avail, &status, &out, &grid_timeout_ns, &trace};
  if (cooperative)
    return cudaLaunchCooperativeKernel(reinterpret_cast<void*>(kernel), dim3(n_cta), dim3(kBlock), args, smem,
                                       stream);
  return cudaLaunchKernel(reinterpret_cast<void*>(kernel), dim3(n_cta), dim3(kBlock), args, smem, stream);
}

template <typename IdxT>
template <int GP, int D>
cudaError_t ClusterLaunch<IdxT>::operator()() const {
  if constexpr (GP >= 0 || GP < -4) {
    return cudaErrorInvalidValue;
  } else {
    if (n > (long long)(n_cta - 1) * cluster_max_slice(GP)) return cudaErrorInvalidValue;
    auto kernel = cluster_run_kernel<GP, D, IdxT>;
    cudaLaunchAttribute attr[2]{};
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)n_cta;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // see launch_after
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(n_cta);
    config.blockDim = dim3(cluster_threads(GP));
    config.dynamicSmemBytes = cluster_smem<GP>(tp, n, n_cta);
    config.stream = stream;
    config.attrs = attr;
    config.numAttrs = fits != nullptr ? 1 : 2;
    // What a launch may ask for at most is set once per device: both calls together cost the host a microsecond.
    static std::atomic<uint64_t> ready{0};
    int dev = 0, most = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return err;
    const uint64_t bit = 1ull << (dev & 63);
    if (dev > 63 || !(ready.load(std::memory_order_acquire) & bit)) {
      cudaFuncAttributes has{};
      if ((err = cudaFuncGetAttributes(&has, kernel)) != cudaSuccess) return err;
      if ((err = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) != cudaSuccess) return err;
      err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)has.sharedSizeBytes);
      if (err == cudaSuccess) err = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
      if (err != cudaSuccess) return err;
      ready.fetch_or(bit, std::memory_order_release);
    }
    if (fits != nullptr) return cudaOccupancyMaxActiveClusters(fits, kernel, &config);
    const ClusterHead<IdxT> head{idx, out, reinterpret_cast<const int2*>(tp.log2phy), n,
                                 cluster_slice(n, n_cta - 1, cluster_threads(GP)), tp.e, cluster_replicated(tp)};
    return cudaLaunchKernelEx(&config, kernel, head, timeout_ns, trace, status, ws, tp, ex, prm, probs, avail);
  }
}

template <int GP, int D>
cudaError_t OccupancyQuery::operator()() const {
  const size_t smem = fused_smem(tp.e) + solver_smem<GP>(tp);
  int per_sm = 0, dev = 0, sms = 0;
  cudaError_t err;
  if (is64) {
    if ((err = allow_smem(fused_run_kernel<GP, D, int64_t>, smem)) != cudaSuccess) return err;
    err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fused_run_kernel<GP, D, int64_t>, kBlock, smem);
  } else {
    if ((err = allow_smem(fused_run_kernel<GP, D, int32_t>, smem)) != cudaSuccess) return err;
    err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fused_run_kernel<GP, D, int32_t>, kBlock, smem);
  }
  if (err != cudaSuccess) return err;
  if ((err = cudaGetDevice(&dev)) != cudaSuccess) return err;
  if ((err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return err;
  *result = per_sm * sms;
  return cudaSuccess;
}

}  // namespace lplb

// One shape for all callers.
#define LPLB_INSTANTIATE(GP, D)                                         \
  template cudaError_t lplb::SolveLaunch::operator()<GP, D>() const;    \
  template cudaError_t lplb::FusedLaunch<int32_t>::operator()<GP, D>(); \
  template cudaError_t lplb::FusedLaunch<int64_t>::operator()<GP, D>(); \
  template cudaError_t lplb::ClusterLaunch<int32_t>::operator()<GP, D>() const; \
  template cudaError_t lplb::ClusterLaunch<int64_t>::operator()<GP, D>() const; \
  template cudaError_t lplb::OccupancyQuery::operator()<GP, D>() const;
