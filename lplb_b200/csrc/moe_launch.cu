// Launchers of the benchmark MoE layer kernels and the TMA descriptor builder.
#include "moe_api.h"

#include <cudaTypedefs.h>

#include "moe_support.cuh"

namespace lplb {
namespace moe {

size_t gemm_smem_bytes() { return kGemmSmem; }

namespace {

// The driver entry point is fetched at run time so that the library has no link-time
// dependency on libcuda (it is imported on GPU-less build hosts too).
PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return nullptr;
    fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }
  return fn;
}

bool shape_ok(const LayerShape& sh) {
  return sh.n_ranks >= 1 && sh.n_ranks <= kMaxRanks && sh.my_rank >= 0 && sh.my_rank < sh.n_ranks &&
         sh.n_local >= 1 && sh.n_local <= kMaxLocalExperts && sh.hidden % kBM == 0 && sh.hidden % kBK == 0 &&
         (2 * sh.inter) % kBM == 0 && sh.inter % kBK == 0 && sh.topk >= 1 && sh.topk <= kCombineMaxTopk &&
         (long long)sh.max_tokens * sh.topk < (1 << 20) && sh.capacity > 0 && sh.capacity < (1 << 24);
}

}  // namespace

namespace {
int encode_map(CUtensorMap* out, const void* base, uint32_t rank, const cuuint64_t* dims, const cuuint64_t* strides,
               const cuuint32_t* box) {
  auto fn = encode_fn();
  if (!fn) return -1;
  if ((reinterpret_cast<uintptr_t>(base) & 15) || strides[0] % 16) return -2;
  const cuuint32_t elem_strides[5] = {1, 1, 1, 1, 1};
  const CUresult rc = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void*>(base), dims, strides, box,
                         elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return rc == CUDA_SUCCESS ? 0 : (int)rc;
}
int row_map(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows) {
  const cuuint64_t dims[2] = {cols, rows};
  const cuuint64_t strides[1] = {cols * 2};
  const cuuint32_t box[2] = {(cuuint32_t)kBK, box_rows};
  return encode_map(out, base, 2, dims, strides, box);
}
// The gate/up weight tensor as [256-row block][group of 16][gate, up][16 rows][cols]: a box of four
// groups arrives in shared memory as 16 gate rows, their 16 up rows, the next 16 gate rows, ...
// Its strides do not ascend (128 rows, then 16 rows): the documentation of cuTensorMapEncodeTiled has
// every stride a multiple of the one before.  The encoder takes the map as it is, and set_weights
// reports the code where one should refuse it.  With ascending strides either the layout that callers
// lay their weights out in would change, or a stage would take four boxes instead of one.
int gate_up_map(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols) {
  const cuuint64_t row = cols * 2;
  const cuuint64_t dims[5] = {cols, kGateRows, 2, kGateBlock / kGateRows, rows / (2 * kGateBlock)};
  const cuuint64_t strides[4] = {row, kGateBlock * row, kGateRows * row, 2 * kGateBlock * row};
  const cuuint32_t box[5] = {(cuuint32_t)kBK, kGateRows, 2, kCtaM / (2 * kGateRows), 1};
  return encode_map(out, base, 5, dims, strides, box);
}
}  // namespace

int make_gemm_maps(GemmMaps* out, const void* tokens, uint64_t rows, const void* weights, uint64_t weight_rows,
                   uint64_t cols, bool gate_up) {
  int rc = 0;
  for (int b = 0; b < kRowBoxes && rc == 0; ++b) rc = row_map(&out->rows[b], tokens, rows, cols, kBN / 2 >> b);
  if (rc == 0) rc = gate_up ? gate_up_map(&out->w, weights, weight_rows, cols) : row_map(&out->w, weights, weight_rows, cols, kCtaM);
  return rc;
}

namespace {
struct PlanView {  // see plan_words()
  int *rows, *row_start, *dst_row_start, *tail, *order_base, *send_base, *arrive_target;
};
PlanView plan_view(const LayerShape& sh, const LayerBuffers& b) {
  const int P = sh.n_ranks * sh.n_local;
  PlanView v;
  v.rows = b.plan;
  v.row_start = b.plan + sh.n_local;
  v.dst_row_start = b.plan + 2 * sh.n_local;
  v.tail = v.dst_row_start + P + sh.n_ranks * P;
  v.order_base = v.tail + 8;
  v.send_base = v.order_base + P;
  v.arrive_target = v.send_base + P;
  return v;
}
}  // namespace

cudaError_t launch_route(const LayerShape& sh, const LayerBuffers& b, const void* phys_idx, int idx_is64, int n_tokens,
                         int n_sms, uint32_t epoch, unsigned long long timeout_ns, int fused, cudaStream_t stream) {
  if (!shape_ok(sh) || n_sms < 1 || n_tokens < 0 || n_tokens > sh.max_tokens) return cudaErrorInvalidValue;
  const int P = sh.n_ranks * sh.n_local;
  RouteArgs a{};
  a.idx = phys_idx;
  a.ordinal = b.ordinal;
  a.totals = b.totals;
  a.ticket = b.tickets + 3;
  a.count_status = b.status + 8;
  for (int r = 0; r < sh.n_ranks; ++r) a.cnt_words[r] = b.cnt_words[r];
  a.plan = b.plan;
  a.status = b.status;
  a.n_pairs = (long long)n_tokens * sh.topk;
  a.idx_is64 = idx_is64;
  a.n_ranks = sh.n_ranks;
  a.my_rank = sh.my_rank;
  a.n_local = sh.n_local;
  a.capacity = sh.capacity;
  a.fused = fused;
  a.epoch = epoch;
  a.timeout_ns = timeout_ns;
  // one pair per thread while that fits one CTA per SM, up to four (what a thread keeps in registers) above
  long long grid = (a.n_pairs + kSupportThreads - 1) / kSupportThreads;
  if (grid > n_sms) grid = n_sms;
  const long long least = (a.n_pairs + 4 * kSupportThreads - 1) / (4 * kSupportThreads);
  if (grid < least) grid = least;
  if (grid < 1) grid = 1;
  return launch_after(route_kernel, (unsigned)grid, kSupportThreads, sizeof(int) * 4 * P, stream, a);
}

cudaError_t launch_dispatch(const LayerShape& sh, const LayerBuffers& b, const void* x, const void* phys_idx,
                            int idx_is64, int n_tokens, int n_cta, uint32_t epoch, cudaStream_t stream) {
  if (!shape_ok(sh) || n_cta < 1 || n_tokens < 0 || n_tokens > sh.max_tokens) return cudaErrorInvalidValue;
  const PlanView plan = plan_view(sh, b);
  DispatchArgs a{};
  for (int r = 0; r < sh.n_ranks; ++r) {
    a.recv_x[r] = static_cast<__nv_bfloat16*>(b.recv_x[r]);
    a.recv_meta[r] = b.recv_meta[r];
    a.flags[r] = b.flags[r];
  }
  a.x = static_cast<const __nv_bfloat16*>(x);
  a.idx = phys_idx;
  a.ordinal = b.ordinal;
  a.dst_row_start = plan.dst_row_start;
  a.send_base = plan.send_base;
  a.pair_slot = b.pair_slot;
  a.status = b.status;
  a.ticket = b.tickets + 0;
  a.n_tokens = n_tokens;
  a.idx_is64 = idx_is64;
  a.topk = sh.topk;
  a.hidden = sh.hidden;
  a.n_local = sh.n_local;
  a.n_ranks = sh.n_ranks;
  a.my_rank = sh.my_rank;
  a.capacity = sh.capacity;
  a.epoch = epoch;
  return launch_after(dispatch_kernel, n_cta, kSupportThreads, 0, stream, a);
}

cudaError_t launch_schedule(const LayerShape& sh, const LayerBuffers& b, const void* phys_idx, int idx_is64,
                            int n_tokens, cudaStream_t stream) {
  if (!shape_ok(sh) || n_tokens < 0 || n_tokens > sh.max_tokens) return cudaErrorInvalidValue;
  const PlanView plan = plan_view(sh, b);
  ScheduleArgs a{};
  a.idx = phys_idx;
  a.ordinal = b.ordinal;
  a.dst_row_start = plan.dst_row_start;
  a.order_base = plan.order_base;
  a.send_base = plan.send_base;
  a.pair_slot = b.pair_slot;
  a.send_pair = b.send_pair;
  a.send_target = b.send_target;
  a.status = b.status;
  a.n_pairs = (long long)n_tokens * sh.topk;
  a.idx_is64 = idx_is64;
  a.n_local = sh.n_local;
  a.n_ranks = sh.n_ranks;
  a.capacity = sh.capacity;
  const long long grid = (a.n_pairs + kSupportThreads - 1) / kSupportThreads;
  return launch_after(schedule_kernel, (unsigned)(grid < 1 ? 1 : grid), kSupportThreads, 0, stream, a);
}

namespace {
RowMaps row_maps(const GemmMaps& m) {
  RowMaps r;
  for (int b = 0; b < kRowBoxes; ++b) r.box[b] = m.rows[b];
  return r;
}
}  // namespace

cudaError_t fused_resident_pairs(int* pairs) {
  auto kernel = grouped_gemm_kernel<kSwiGLU, true>;
  const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGemmSmem);
  if (err != cudaSuccess) return err;
  cudaLaunchAttribute cluster{};
  cluster.id = cudaLaunchAttributeClusterDimension;
  cluster.val.clusterDim.x = 2;
  cluster.val.clusterDim.y = cluster.val.clusterDim.z = 1;
  cudaLaunchConfig_t config{};
  config.gridDim = dim3(2);
  config.blockDim = dim3(kFusedThreads);
  config.dynamicSmemBytes = kGemmSmem;
  config.attrs = &cluster;
  config.numAttrs = 1;
  return cudaOccupancyMaxActiveClusters(pairs, kernel, &config);
}

cudaError_t launch_dispatch_gemm(const LayerShape& sh, const LayerBuffers& b, const GemmMaps& maps, const void* x, uint32_t epoch,
                                 unsigned long long timeout_ns, FusedGrid grid, cudaStream_t stream) {
  if (!shape_ok(sh) || grid.tile < 2 || grid.tile % 2 || grid.send < 0 || grid.send % 2) return cudaErrorInvalidValue;
  const PlanView plan = plan_view(sh, b);
  GemmArgs a{};
  a.send_ctas = grid.send;
  a.next_tile = b.tickets + 4;
  a.rows = plan.rows;
  a.row_start = plan.row_start;
  a.n_experts = sh.n_local;
  a.n_ranks = sh.n_ranks;
  a.my_rank = sh.my_rank;
  a.epoch = epoch;
  a.status = b.status;
  a.timeout_ns = timeout_ns;
  a.n_tiles_w = 2 * sh.inter / kBM;
  a.k_blocks = sh.hidden / kBK;
  a.act = static_cast<__nv_bfloat16*>(b.act);
  a.act_ld = sh.inter;
  a.wait_flags = nullptr;
  a.ticket = b.tickets + 1;
  a.x = static_cast<const __nv_bfloat16*>(x);
  a.send_pair = b.send_pair;
  a.send_target = b.send_target;
  a.pair_slot = b.pair_slot;
  a.n_send = plan.tail + 2;
  a.arrive_target = plan.arrive_target;
  for (int r = 0; r < sh.n_ranks; ++r) {
    a.recv_x[r] = static_cast<__nv_bfloat16*>(b.recv_x[r]);
    a.recv_meta[r] = b.recv_meta[r];
    a.arrived[r] = b.arrived[r];
  }
  a.topk = sh.topk;
  a.hidden = sh.hidden;
  a.debug = b.debug;
  auto kernel = grouped_gemm_kernel<kSwiGLU, true>;
  cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGemmSmem);
  if (err != cudaSuccess) return err;
  return launch_after(kernel, grid.tile + grid.send, kFusedThreads, kGemmSmem, stream, maps.w, row_maps(maps), a);
}

cudaError_t launch_gemm(const LayerShape& sh, const LayerBuffers& b, const GemmMaps& maps, int which, uint32_t epoch, unsigned long long timeout_ns,
                        int n_cta, cudaStream_t stream) {
  if (!shape_ok(sh) || n_cta < 2 || (which != 0 && which != 1)) return cudaErrorInvalidValue;
  n_cta &= ~1;
  GemmArgs a{};
  a.next_tile = b.tickets + 4;
  a.rows = b.plan;
  a.row_start = b.plan + sh.n_local;
  a.n_experts = sh.n_local;
  a.n_ranks = sh.n_ranks;
  a.my_rank = sh.my_rank;
  a.epoch = epoch;
  a.status = b.status;
  a.timeout_ns = timeout_ns;
  cudaError_t err;
  if (which == 0) {
    a.n_tiles_w = 2 * sh.inter / kBM;
    a.k_blocks = sh.hidden / kBK;
    a.act = static_cast<__nv_bfloat16*>(b.act);
    a.act_ld = sh.inter;
    a.wait_flags = sh.n_ranks > 1 ? b.flags[sh.my_rank] : nullptr;  // dispatch done, one word per source rank
    a.ticket = b.tickets + 1;
    auto kernel = grouped_gemm_kernel<kSwiGLU, false>;
    err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGemmSmem);
    if (err != cudaSuccess) return err;
    return launch_after(kernel, n_cta, kGemmThreads, kGemmSmem, stream, maps.w, row_maps(maps), a);
  } else {
    a.n_tiles_w = sh.hidden / kBM;
    a.k_blocks = sh.inter / kBK;
    a.meta = b.recv_meta[sh.my_rank];
    for (int r = 0; r < sh.n_ranks; ++r) {
      a.comb[r] = static_cast<__nv_bfloat16*>(b.comb[r]);
      a.done_flags[r] = b.flags[r] + sh.n_ranks;  // combine done
    }
    a.out_ld = sh.hidden;
    a.wait_flags = nullptr;
    a.ticket = b.tickets + 2;
    auto kernel = grouped_gemm_kernel<kScatter, false>;
    err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGemmSmem);
    if (err != cudaSuccess) return err;
    return launch_after(kernel, n_cta, kGemmThreads, kGemmSmem, stream, maps.w, row_maps(maps), a);
  }
}

cudaError_t launch_combine(const LayerShape& sh, const LayerBuffers& b, const float* weights, void* out, int n_tokens,
                           uint32_t epoch, unsigned long long timeout_ns, int n_cta, cudaStream_t stream) {
  if (!shape_ok(sh) || n_tokens < 0 || n_tokens > sh.max_tokens || n_cta < 1) return cudaErrorInvalidValue;
  CombineArgs a{};
  a.comb = static_cast<const __nv_bfloat16*>(b.comb[sh.my_rank]);
  a.weights = weights;
  a.pair_slot = b.pair_slot;
  a.out = static_cast<__nv_bfloat16*>(out);
  a.wait_flags = b.flags[sh.my_rank] + sh.n_ranks;
  a.status = b.status;
  a.n_tokens = n_tokens;
  a.topk = sh.topk;
  a.hidden = sh.hidden;
  a.n_ranks = sh.n_ranks;
  a.epoch = epoch;
  a.timeout_ns = timeout_ns;
  return launch_after(combine_kernel, n_cta, kSupportThreads, 0, stream, a);
}

}  // namespace moe
}  // namespace lplb
