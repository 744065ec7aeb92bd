// Host-side launch interface of the benchmark MoE layer kernels (dispatch, grouped GEMMs,
// combine).  Plain C++ so that the CUDA translation unit needs no torch headers.
// The reference contains no MoE layer; these kernels consume the planner's redirected
// indices for the end-to-end measurement.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace lplb {
namespace moe {

constexpr int kApiMaxRanks = 8;

struct LayerShape {
  int hidden;        // H
  int inter;         // I (SwiGLU width); w13 is [experts, 2*I, H], w2 is [experts, H, I]
  int n_local;       // physical experts on this rank
  int n_ranks, my_rank;
  int topk;
  int max_tokens;    // tokens per rank (upper bound)
  int capacity;      // rows of the receive buffer
};

// Pointers into this rank's own and its peers' buffers (peer entries alias the local ones
// when n_ranks == 1).
struct LayerBuffers {
  // peer-visible
  void* recv_x[kApiMaxRanks];          // bf16 [capacity, H]
  int* recv_meta[kApiMaxRanks];        // int32 [capacity]
  void* comb[kApiMaxRanks];            // bf16 [max_tokens * topk, H]
  unsigned long long* cnt_words[kApiMaxRanks];  // uint64 [2][n_ranks][n_ranks * n_local]
  uint32_t* flags[kApiMaxRanks];       // uint32 [2][n_ranks]: dispatch done, combine done
  // local
  void* act;                           // bf16 [capacity, I]
  int* plan;                           // int32 plan block, see plan_words()
  int* ordinal;                        // int32 [max_tokens * topk] position of every pair among its expert's
  int* totals;                         // int32 [n_ranks * n_local], zero between launches
  int* pair_slot;                      // int32 [max_tokens * topk] return slot of every pair
  int* send_pair;                      // int32 [max_tokens * topk] pair index at every send position
  int* send_target;                    // int32 [max_tokens * topk] (rank << 24) | row, or -1
  uint32_t* arrived[kApiMaxRanks];     // per rank: uint32 [n_local] rows that have landed, cumulative
  unsigned long long* debug;           // optional uint64 [n_cta * 4] timing of the fused kernel, may be null
  unsigned* tickets;                   // uint32 [5], zero: dispatch, first GEMM, second GEMM, routing, GEMM tiles
  int* status;                         // int32 [16]
};

// Layout of the plan block (ints), P = n_ranks * n_local:
//   rows[n_local], row_start[n_local], dst_row_start[P], all_counts[n_ranks * P],
//   tail[8] = {total_rows, overflow, n_send, ...},
//   order_base[P]      first send position of this rank's pairs for physical expert p,
//   send_base[P]       first return slot of this rank's pairs for physical expert p,
//   arrive_target[n_local], arrive_cum[n_local]   cumulative rows expected per local expert
//                      (arrive_cum persists across launches, it is never zeroed by a launch).
inline int plan_words(int n_ranks, int n_local) {
  const int p = n_ranks * n_local;
  return 2 * n_local + p + n_ranks * p + 8 + 2 * p + 2 * n_local;
}

size_t gemm_smem_bytes();

// Tensor maps of one grouped GEMM (128-byte swizzle, 64 elements of K per box): weights, received
// rows in boxes of 128, 64, 32 and 16 rows.
struct GemmMaps {
  CUtensorMap w, rows[4];
};
// tokens: bf16 [rows, cols]; weights: bf16 [weight_rows, cols], with `gate_up` in blocks of 128
// gate rows and their 128 up rows.  Returns 0 on success.
int make_gemm_maps(GemmMaps* out, const void* tokens, uint64_t rows, const void* weights, uint64_t weight_rows,
                   uint64_t cols, bool gate_up);

// Step 1: rank the pairs of every physical expert, all-gather the per-expert counts of this
// launch and derive row offsets.
cudaError_t launch_route(const LayerShape& sh, const LayerBuffers& b, const void* phys_idx, int idx_is64, int n_tokens,
                         int n_sms, uint32_t epoch, unsigned long long timeout_ns, int fused, cudaStream_t stream);
// Step 2: copy every (token, k) pair's hidden state into its expert's rows on the target rank.
cudaError_t launch_dispatch(const LayerShape& sh, const LayerBuffers& b, const void* x, const void* phys_idx,
                            int idx_is64, int n_tokens, int n_cta, uint32_t epoch, cudaStream_t stream);
// Step 2a (fused path only): decide the send order and every pair's target row and return slot.
cudaError_t launch_schedule(const LayerShape& sh, const LayerBuffers& b, const void* phys_idx, int idx_is64,
                            int n_tokens, cudaStream_t stream);
// How the fused kernel's CTAs are dealt out: `tile` of them run tiles and `send` only send rows.
struct FusedGrid {
  int tile, send;
};
// The tile CTAs wait for rows that every sender of the launch sends, so all CTAs have to be resident
// at once: no more pairs than the device holds (a GPC with an odd number of SMs leaves one without a
// partner).  send_ctas is rounded up to whole pairs; one pair at least runs tiles.
inline FusedGrid fused_grid(int n_cta, int send_ctas, int resident_pairs) {
  const int pairs = n_cta / 2 < resident_pairs ? n_cta / 2 : resident_pairs;
  int send = (send_ctas + 1) / 2;
  if (send > pairs - 1) send = pairs - 1;
  return FusedGrid{2 * (pairs - send), 2 * send};
}
// CTA pairs of the fused kernel that fit on the current device at once.
cudaError_t fused_resident_pairs(int* pairs);
// Step 2b+3 fused: the first grouped GEMM, which also streams this rank's rows to their targets
// while the tensor cores work on the experts whose rows have landed.  grid.send == 0: four
// extra warps in every CTA send.
cudaError_t launch_dispatch_gemm(const LayerShape& sh, const LayerBuffers& b, const GemmMaps& maps, const void* x, uint32_t epoch,
                                 unsigned long long timeout_ns, FusedGrid grid, cudaStream_t stream);
// Step 3/4: grouped GEMMs.  which = 0: recv_x x w13 -> SwiGLU -> act.  which = 1: act x w2 -> peers' comb.
cudaError_t launch_gemm(const LayerShape& sh, const LayerBuffers& b, const GemmMaps& maps, int which, uint32_t epoch, unsigned long long timeout_ns,
                        int n_cta, cudaStream_t stream);
// Step 5: out[t] = sum_k weight[t, k] * comb[pair_slot[t * topk + k]].
cudaError_t launch_combine(const LayerShape& sh, const LayerBuffers& b, const float* weights, void* out, int n_tokens,
                           uint32_t epoch, unsigned long long timeout_ns, int n_cta, cudaStream_t stream);

}  // namespace moe
}  // namespace lplb
