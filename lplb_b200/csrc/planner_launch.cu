// Launchers for the planner kernels: shape dispatch to the ahead-of-time instantiations.
#include "planner_api.h"
#include "planner_kernels.cuh"

namespace lplb {

namespace {

Topo make_topo(const TopoDesc& t) {
  Topo o;
  o.r2o = t.r2o;
  o.o2r = t.o2r;
  o.phy2log = t.phy2log;
  o.log2phy = t.log2phy;
  o.log2edge = t.log2edge;
  o.log2slot = t.log2slot;
  o.n_group = t.n_group;
  o.g = t.g;
  o.d = t.d;
  o.ll = t.ll;
  o.c = t.c;
  o.pl = t.ll + t.c * t.d;
  o.e = t.n_group * t.g * t.ll;
  return o;
}

int padded_group(int g) { return g <= 8 ? 8 : (g <= 16 ? 16 : 32); }
int padded_dup(int d) { return d <= 4 ? d : 8; }

// The counting and redirect kernels work for any topology; the solvers (and with them the
// fused kernel) cover groups of up to kMaxGroupSize ranks and kMaxDup replicas.
bool shape_ok(const TopoDesc& t, bool need_solver = true, int solver = kSolverAuto) {
  const bool tables = t.g >= 1 && t.d >= 1 && t.n_group >= 1 && t.ll >= t.c * t.d &&
                      (long long)t.n_group * t.g * t.ll <= kMaxLogicalExperts;
  return tables && (!need_solver || resolve_solver(t.g, t.d, solver) > 0);
}

// Calls fn.template operator()<GP, D>() for the instantiation that covers the topology: GP = -1, -2, -4,
// -8 for the tile solver with that many warps per group, 8, 16, 32 for the warp solver, 0 for the
// thread-block solver (D is then the padded count).  The tile solver takes every group that it
// covers (8 ranks 22.6 -> 10.3 us a call, 16 ranks 40.6 -> 17.0, 32 ranks 64 -> 25, 64 ranks 147 -> 52 against the
// other two), except that the warp solver packs four groups of 8 ranks into a warp: `packed` asks for
// that where one CTA has many of them.  The warp solver's larger groups run on request only.
template <typename Fn>
cudaError_t dispatch_shape(int g, int d, int solver, bool packed, Fn&& fn) {
  const int kind = resolve_solver(g, d, solver);
  if (kind != kSolverWarp && kind != kSolverBlock) return cudaErrorInvalidValue;
  const bool tiles = d <= kTileMaxDup && (kind == kSolverWarp ? g <= 8 && !packed : g <= kTileMaxGroup);
  if (tiles) {
    const int nb = tile_rows(g);
#define LPLB_CASE(NB_, D_) \
  if (nb == NB_ && d == D_) return fn.template operator()<-NB_, D_>();
    LPLB_CASE(1, 1) LPLB_CASE(1, 2) LPLB_CASE(1, 3) LPLB_CASE(1, 4)
    LPLB_CASE(2, 1) LPLB_CASE(2, 2) LPLB_CASE(2, 3) LPLB_CASE(2, 4)
    LPLB_CASE(4, 1) LPLB_CASE(4, 2) LPLB_CASE(4, 3) LPLB_CASE(4, 4)
    LPLB_CASE(8, 1) LPLB_CASE(8, 2) LPLB_CASE(8, 3) LPLB_CASE(8, 4)
#undef LPLB_CASE
    return cudaErrorInvalidValue;
  }
  if (kind == kSolverBlock) {
    const int dp = padded_dup(d);
#define LPLB_CASE(D_) \
  if (dp == D_) return fn.template operator()<0, D_>();
    LPLB_CASE(1) LPLB_CASE(2) LPLB_CASE(3) LPLB_CASE(4) LPLB_CASE(8)
#undef LPLB_CASE
    return cudaErrorInvalidValue;
  }
  const int gp = padded_group(g);
#define LPLB_CASE(GP_, D_) \
  if (gp == GP_ && d == D_) return fn.template operator()<GP_, D_>();
  LPLB_CASE(8, 1) LPLB_CASE(8, 2) LPLB_CASE(8, 3) LPLB_CASE(8, 4)
  LPLB_CASE(16, 1) LPLB_CASE(16, 2) LPLB_CASE(16, 3) LPLB_CASE(16, 4)
  LPLB_CASE(32, 1) LPLB_CASE(32, 2) LPLB_CASE(32, 3) LPLB_CASE(32, 4)
#undef LPLB_CASE
  return cudaErrorInvalidValue;
}

size_t fused_smem(int e) { return sizeof(int) * 5 * (size_t)e; }
size_t bundle_smem(const Topo& tp) { return sizeof(int) * (size_t)tp.n_group * tp.g * (tp.d + 1); }
// bundle sums followed by the solver's scratch area, if it has one
template <int GP>
size_t solver_smem(const Topo& tp, int teams = kWarps) {
  if constexpr (GP > 0) return bundle_smem(tp);
  else return bundle_bytes_aligned(tp.n_group * tp.g, tp.d) +
              (GP == 0 ? block_solver_smem_bytes(tp.g, padded_dup(tp.d)) : tile_solver_smem_bytes(tp.g, tp.d, GP == -1 ? teams : 1));
}
// The fused kernel's one solver CTA gives each of its warps up to two groups of 8 ranks, one after the other;
// beyond, the warp solver packs four groups to a warp.  Step with L2 flushed, warm-started, packed against a group
// per warp, us: two replicas 4 groups 24.7 / 16.4, 8 groups 28.8 / 18.4, 9 groups 34.8 / 22.7, 16 groups 36.9 / 26.7, 24
// groups 36.9 / 36.9, 32 groups 41.0 / 45.0, 64 groups 68.5 / 78.0; one replica 16 groups 28.7 / 26.6, 17 groups 30.8 /
// 30.8, 32 groups 36.9 / 43.0; four replicas 47 / 27, 51 / 31 and 58 / 43 there.  Up to two rounds a step also
// solves with the same code as the stand-alone kernel, bit for bit; beyond, shares agree to rounding (1e-6 of their norm).
bool pack_groups(const Topo& tp) { return tp.n_group > 2 * kWarps; }

template <typename K>
cudaError_t allow_smem(K kernel, size_t bytes) {
  if (bytes <= 48 * 1024) return cudaSuccess;
  if (bytes > 227 * 1024) return cudaErrorInvalidValue;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

IpmParams make_params(const SolveParams& prm, int g, int d) {
  IpmParams p{prm.max_iters, prm.tol, prm.anchor, prm.anchor_valid, prm.guard, prm.snap_mu};
  p.pad_rows = resolve_solver(g, d, prm.solver) == kSolverWarp;
  return p;
}

}  // namespace

int resolve_solver(int g, int d, int requested) {
  const bool warp_ok = g >= 1 && d >= 1 && g <= kMaxWarpGroupSize && d <= kMaxWarpDup;
  const bool block_ok = g >= 1 && d >= 1 && g <= kMaxGroupSize && d <= kMaxDup && g <= kBlkMaxGroup;
  if (requested == kSolverWarp) return warp_ok ? kSolverWarp : -1;
  if (requested == kSolverBlock) return block_ok ? kSolverBlock : -1;
  if (warp_ok && g <= 8) return kSolverWarp;
  return block_ok ? kSolverBlock : -1;
}

int anchor_dup(int g, int d, int requested) { return resolve_solver(g, d, requested) == kSolverBlock ? padded_dup(d) : d; }

size_t planner_workspace_bytes(int n_logical) { return workspace_bytes(n_logical); }

cudaError_t launch_count(const void* idx, int idx_is64, long long n, int n_logical, int n_cta, int* by_cta,
                         void* workspace, int* status, cudaStream_t stream) {
  if (n_logical < 1 || n_logical > kMaxLogicalExperts || n_cta < 1) return cudaErrorInvalidValue;
  const size_t smem = sizeof(int) * (size_t)n_logical;
  auto* ws = static_cast<Workspace*>(workspace);
  if (idx_is64)
    count_kernel<int64_t><<<n_cta, kBlock, smem, stream>>>(static_cast<const int64_t*>(idx), n, n_logical, by_cta, ws,
                                                           status);
  else
    count_kernel<int32_t><<<n_cta, kBlock, smem, stream>>>(static_cast<const int32_t*>(idx), n, n_logical, by_cta, ws,
                                                           status);
  return cudaGetLastError();
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
  cudaError_t operator()() const {
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
        // an early launch: 14.3 -> 11.6 us for 64 groups of 8 ranks, one call after the other, 64 ranks 59 -> 52
        return launch_after(tile_solve_kernel<1, D>, grid + 1, kBlock, smem, stream, workload, tp, prm, probs, normalised, avail,
                            status, warps);
      } else {
        if ((err = allow_smem(solve_kernel<GP, D>, smem)) != cudaSuccess) return err;
        solve_kernel<GP, D><<<grid, kBlock, smem, stream>>>(workload, tp, prm, probs, normalised, avail, status, warps);
      }
    }
    return cudaGetLastError();
  }
};

cudaError_t launch_solve(const int* workload, const TopoDesc& topo, SolveParams prm, float* probs, float* normalised,
                         void* avail, int avail_is64, int* status, cudaStream_t stream) {
  if (!shape_ok(topo, true, prm.solver)) return cudaErrorInvalidValue;
  SolveLaunch l{workload, make_topo(topo), make_params(prm, topo.g, topo.d), probs, normalised, Counter{avail, avail_is64}, status,
                stream};
  return dispatch_shape(topo.g, topo.d, prm.solver, false, l);
}

cudaError_t launch_redirect(const void* idx, int idx_is64, long long n, const float* probs, const int* by_cta,
                            const TopoDesc& topo, int n_cta, void* out, cudaStream_t stream) {
  if (!shape_ok(topo, false) || n_cta < 1) return cudaErrorInvalidValue;
  const Topo tp = make_topo(topo);
  const size_t smem = fused_smem(tp.e);
  cudaError_t err;
  if (idx_is64) {
    if ((err = allow_smem(redirect_kernel<int64_t>, smem)) != cudaSuccess) return err;
    redirect_kernel<int64_t><<<n_cta, kBlock, smem, stream>>>(static_cast<const int64_t*>(idx), n, probs, by_cta, tp,
                                                              static_cast<int64_t*>(out));
  } else {
    if ((err = allow_smem(redirect_kernel<int32_t>, smem)) != cudaSuccess) return err;
    redirect_kernel<int32_t><<<n_cta, kBlock, smem, stream>>>(static_cast<const int32_t*>(idx), n, probs, by_cta, tp,
                                                              static_cast<int32_t*>(out));
  }
  return cudaGetLastError();
}

cudaError_t launch_exchange(const int* in, int n_logical, const ExchangeDesc& exd, void* workspace, int* out,
                            int* status, cudaStream_t stream) {
  if (n_logical < 1 || n_logical > kMaxLogicalExperts || exd.n_ranks < 2 || exd.n_ranks > kMaxRanks)
    return cudaErrorInvalidValue;
  Exchange ex{exd.recv, exd.n_ranks, exd.my_rank, exd.node_size, exd.timeout_ns};
  const size_t smem = sizeof(int) * (size_t)n_logical;
  cudaError_t err = allow_smem(exchange_kernel, smem);
  if (err != cudaSuccess) return err;
  exchange_kernel<<<1, kBlock, smem, stream>>>(in, n_logical, ex, static_cast<Workspace*>(workspace), out, status);
  return cudaGetLastError();
}

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
  cudaError_t operator()() {
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
};

cudaError_t launch_fused(const void* idx, int idx_is64, long long n, const TopoDesc& topo, const ExchangeDesc& exd,
                         SolveParams prm, void* workspace, float* probs, void* avail, int avail_is64, int* status,
                         void* out, int n_cta, unsigned long long grid_timeout_ns, unsigned long long* trace,
                         int cooperative, cudaStream_t stream) {
  if (!shape_ok(topo, true, prm.solver) || n_cta < 2 || exd.n_ranks > kMaxRanks) return cudaErrorInvalidValue;
  Exchange ex{exd.recv, exd.n_ranks, exd.my_rank, exd.node_size, exd.timeout_ns};
  if (idx_is64) {
    FusedLaunch<int64_t> l{static_cast<const int64_t*>(idx), n, make_topo(topo), ex, make_params(prm, topo.g, topo.d),
                           static_cast<Workspace*>(workspace), probs, Counter{avail, avail_is64}, status,
                           static_cast<int64_t*>(out), n_cta, grid_timeout_ns, trace, cooperative, stream};
    return dispatch_shape(topo.g, topo.d, prm.solver, pack_groups(l.tp), l);
  }
  FusedLaunch<int32_t> l{static_cast<const int32_t*>(idx), n, make_topo(topo), ex, make_params(prm, topo.g, topo.d),
                         static_cast<Workspace*>(workspace), probs, Counter{avail, avail_is64}, status,
                         static_cast<int32_t*>(out), n_cta, grid_timeout_ns, trace, cooperative, stream};
  return dispatch_shape(topo.g, topo.d, prm.solver, pack_groups(l.tp), l);
}

struct OccupancyQuery {
  Topo tp;
  int is64;
  int* result;
  template <int GP, int D>
  cudaError_t operator()() const {
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
};

int max_fused_ctas(const TopoDesc& topo, int solver, int idx_is64) {
  int result = 0;
  if (!shape_ok(topo, true, solver)) return 0;
  const Topo tp = make_topo(topo);
  OccupancyQuery q{tp, idx_is64, &result};
  if (dispatch_shape(topo.g, topo.d, solver, pack_groups(tp), q) != cudaSuccess) return 0;
  return result;
}

namespace {
__global__ void debug_reciprocals_kernel(const double* __restrict__ x, int n, double* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  out[i] = rcp3(x[i]);
  out[n + i] = step_ratio(x[i], -1.0);
}
}  // namespace

cudaError_t launch_debug_reciprocals(const double* x, int n, double* out, cudaStream_t stream) {
  if (n < 1) return cudaErrorInvalidValue;
  debug_reciprocals_kernel<<<(n + kBlock - 1) / kBlock, kBlock, 0, stream>>>(x, n, out);
  return cudaGetLastError();
}

}  // namespace lplb
