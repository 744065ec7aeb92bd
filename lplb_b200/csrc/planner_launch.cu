// Launchers for the planner kernels: shape dispatch to the ahead-of-time instantiations.
#include "planner_shapes.cuh"

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
// covers (8 ranks 22.6 -> 10.4 us a call, 16 ranks 40.6 -> 17.9, 32 ranks 64 -> 25, 64 ranks 147 -> 46 against the
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

// The fused kernel's one solver CTA gives each of its warps up to two groups of 8 ranks, one after the other;
// beyond, the warp solver packs four groups to a warp.  Step with L2 flushed, warm-started, packed against a group
// per warp, us: two replicas 4 groups 24.7 / 16.4, 8 groups 28.8 / 18.4, 9 groups 34.8 / 22.7, 16 groups 36.9 / 26.7, 24
// groups 36.9 / 36.9, 32 groups 41.0 / 45.0, 64 groups 68.5 / 78.0; one replica 16 groups 28.7 / 26.6, 17 groups 30.8 /
// 30.8, 32 groups 36.9 / 43.0; four replicas 47 / 27, 51 / 31 and 58 / 43 there.  Up to two rounds a step also
// solves with the same code as the stand-alone kernel, bit for bit; beyond, shares agree to rounding (1e-6 of their norm).
bool pack_groups(const Topo& tp) { return tp.n_group > 2 * kWarps; }

IpmParams make_params(const SolveParams& prm, const TopoDesc& t) {
  IpmParams p{prm.max_iters, prm.tol, prm.anchor, prm.anchor_valid, prm.guard, prm.snap_mu};
  p.pad_rows = resolve_solver(t.g, t.d, prm.solver) == kSolverWarp;
  p.plan = TilePlan{t.tile_rounds, t.tile_near};
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

namespace {
struct CodeQuery {
  const char** name;
  template <int GP, int D>
  cudaError_t operator()() const {
    *name = GP < 0 ? "tile" : (GP > 0 ? "warp" : "block");
    return cudaSuccess;
  }
};
}  // namespace

const char* solver_code(const TopoDesc& topo, int requested, bool fused) {
  const char* name = "none";
  if (shape_ok(topo, true, requested)) dispatch_shape(topo.g, topo.d, requested, fused && pack_groups(make_topo(topo)), CodeQuery{&name});
  return name;
}

void plan_topology(int g, int d, const int* r2o, const int* o2r, unsigned long long* rounds, unsigned long long* near) {
  TilePlan plan;
  if (g <= kTileMaxGroup && d <= kTileMaxDup) plan = plan_tiles(g, d, {r2o, o2r});
  *rounds = plan.rounds;
  *near = plan.near;
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

cudaError_t launch_solve(const int* workload, const TopoDesc& topo, SolveParams prm, float* probs, float* normalised,
                         void* avail, int avail_is64, int* status, cudaStream_t stream) {
  if (!shape_ok(topo, true, prm.solver)) return cudaErrorInvalidValue;
  SolveLaunch l{workload, make_topo(topo), make_params(prm, topo), probs, normalised, Counter{avail, avail_is64}, status,
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

namespace {
// Stand-alone all-reduce of int32[E] counts over the peers (one CTA), for callers that
// feed their own statistics to the solver.  Shares the epoch with the fused kernel, so it
// keeps that kernel's invariant: the totals of the other parity are zero when it ends.
__global__ void __launch_bounds__(kBlock) exchange_kernel(const int* __restrict__ in, int e, Exchange ex,
                                                          Workspace* ws, int* __restrict__ out, int* status) {
  extern __shared__ __align__(16) int smem[];
  __shared__ ExchangeShared xs;
  int* vec = smem;
  const uint32_t epoch = ld_acquire_gpu(&ws->epoch) + 1;
  int* other = ws_total(ws, (epoch & 1) ^ 1, e);
  exchange_prepare(ex, &xs);
  for (int i = threadIdx.x; i < e; i += kBlock) {
    vec[i] = in[i];
    other[i] = 0;
  }
  __syncthreads();
  const unsigned miss = exchange_counts<kBlock>(ex, &xs, epoch, e, vec, status, nullptr);
  if (miss && threadIdx.x == 0) {
    atomicAdd(&status[kStTimeouts], 1);
    raise_status(status, kErrPeerTimeout, kPhExchange, (int)miss);
  }
  for (int i = threadIdx.x; i < e; i += kBlock) out[i] = vec[i];
  __syncthreads();
  if (threadIdx.x == 0) {
    ws->arrive[(epoch & 1) ^ 1] = 0;  // every launch leaves the next one's arrival counter at zero
    st_release_gpu(&ws->epoch, epoch);
  }
}
}  // namespace

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

cudaError_t launch_fused(const void* idx, int idx_is64, long long n, const TopoDesc& topo, const ExchangeDesc& exd,
                         SolveParams prm, void* workspace, float* probs, void* avail, int avail_is64, int* status,
                         void* out, int n_cta, unsigned long long grid_timeout_ns, unsigned long long* trace,
                         int cooperative, cudaStream_t stream) {
  if (!shape_ok(topo, true, prm.solver) || n_cta < 2 || exd.n_ranks > kMaxRanks) return cudaErrorInvalidValue;
  Exchange ex{exd.recv, exd.n_ranks, exd.my_rank, exd.node_size, exd.timeout_ns};
  if (idx_is64) {
    FusedLaunch<int64_t> l{static_cast<const int64_t*>(idx), n, make_topo(topo), ex, make_params(prm, topo),
                           static_cast<Workspace*>(workspace), probs, Counter{avail, avail_is64}, status,
                           static_cast<int64_t*>(out), n_cta, grid_timeout_ns, trace, cooperative, stream};
    return dispatch_shape(topo.g, topo.d, prm.solver, pack_groups(l.tp), l);
  }
  FusedLaunch<int32_t> l{static_cast<const int32_t*>(idx), n, make_topo(topo), ex, make_params(prm, topo),
                         static_cast<Workspace*>(workspace), probs, Counter{avail, avail_is64}, status,
                         static_cast<int32_t*>(out), n_cta, grid_timeout_ns, trace, cooperative, stream};
  return dispatch_shape(topo.g, topo.d, prm.solver, pack_groups(l.tp), l);
}

namespace {
template <typename IdxT>
cudaError_t cluster_step(const void* idx, long long n, const Topo& tp, const Exchange& ex, const IpmParams& prm, int solver, void* workspace,
                         float* probs, Counter avail, int* status, void* out, int n_cta, unsigned long long timeout_ns,
                         unsigned long long* trace, cudaStream_t stream, int* fits) {
  const ClusterLaunch<IdxT> l{static_cast<const IdxT*>(idx), n, tp, ex, prm,
                              static_cast<Workspace*>(workspace), probs, avail, status, static_cast<IdxT*>(out), n_cta,
                              timeout_ns, trace, stream, fits};
  return dispatch_shape(tp.g, tp.d, solver, pack_groups(tp), l);
}
}  // namespace

cudaError_t launch_cluster(const void* idx, int idx_is64, long long n, const TopoDesc& topo, const ExchangeDesc& exd,
                           SolveParams prm, void* workspace, float* probs, void* avail, int avail_is64, int* status,
                           void* out, int n_cta, unsigned long long timeout_ns, unsigned long long* trace, cudaStream_t stream) {
  if (!shape_ok(topo, true, prm.solver) || n_cta < 2 || n_cta > kClusterMaxCtas || exd.n_ranks > kMaxRanks) return cudaErrorInvalidValue;
  const Topo tp = make_topo(topo);
  if (tp.e > kClusterMaxExperts || cluster_replicated(tp) < 1) return cudaErrorInvalidValue;
  const Exchange ex{exd.recv, exd.n_ranks, exd.my_rank, exd.node_size, exd.timeout_ns};
  return (idx_is64 ? cluster_step<int64_t> : cluster_step<int32_t>)(idx, n, tp, ex, make_params(prm, topo), prm.solver, workspace, probs, Counter{avail, avail_is64},
                                                                     status, out, n_cta, timeout_ns, trace, stream, nullptr);
}

int cluster_ctas(long long n, bool host_result) {
  if (host_result && n > kClusterHostResult) return 0;
  int n_cta = 2;
  while (n_cta < kClusterMaxCtas && n > (long long)(n_cta - 1) * kClusterShare) n_cta *= 2;
  return n_cta;
}

long long cluster_limit(const TopoDesc& topo, int solver, int idx_is64, int n_cta) {
  const Topo tp = make_topo(topo);
  if (!shape_ok(topo, true, solver) || tp.e > kClusterMaxExperts || cluster_replicated(tp) < 1) return 0;
  const long long n = (long long)(n_cta - 1) * cluster_paying_slice(-tile_rows(tp.g), tp.e, cluster_replicated(tp));
  int fits = 0;
  const cudaError_t err = (idx_is64 ? cluster_step<int64_t> : cluster_step<int32_t>)(
      nullptr, n, tp, Exchange{}, IpmParams{1, 1.0}, solver, nullptr, nullptr, Counter{}, nullptr, nullptr, n_cta, 0, nullptr, nullptr, &fits);
  if (err != cudaSuccess) cudaGetLastError();  // this shape does not run in a cluster
  return err == cudaSuccess && fits > 0 ? n : 0;
}

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
