// Grouped expert GEMM for the benchmark MoE layer on sm_100a: bf16 x bf16 -> fp32 on the
// 5th-generation tensor cores (tcgen05.mma.cta_group::2, accumulators in tensor memory),
// operands staged by TMA into 128-byte-swizzled shared memory, persistent warp-specialised
// CTA pairs.
//
//   C_e[rows_e, N] = A_e[rows_e, K] * B_e[N, K]^T        for every local expert e
//
// A is the row-major receive buffer (all experts' rows back to back, expert e starts at
// row_start[e]); B is the weight tensor [experts * N, K].  Rows per expert are only known
// on the device, so the tile list is derived in-kernel from `rows`.
//
// A pair of CTAs computes a tile of 256 weight rows x up to 256 received rows, weights on the
// tensor core's M side (128 per CTA), received rows on its N side (half of them staged by each
// CTA).  Why this way round: the number of rows an expert receives is arbitrary, and N comes in
// steps of 32 where M does not shrink, so the work for padding is 16 rows per expert on average
// and a decode step's few rows cost few cycles and few bytes.
//
// Which pair computes which tile is decided as they go: a pair that finishes takes the next tile
// of the list.  With many rows the kernel is bound by the board's power limit, and there DRAM
// traffic is what costs most.  The pairs that share a weight tile must therefore read it at the
// same time, before L2 has lost it.  Tiles of different experts differ in size, so dealing the
// list out in turn lets the pairs drift apart: 13.9 GB read from DRAM (8192 tokens x top-8, 48
// experts, 7168 x 2048, first GEMM; 3.8 GB is every operand once).
//
// Roles inside a CTA (192 threads):
//   warp 0      TMA producer: 128 weight rows and half of the tile's received rows per stage
//   warp 1      allocates 512 TMEM columns; in the pair's first CTA issues tcgen05.mma (one lane)
//   warps 2-5   epilogue: tcgen05.ld their 32-lane quarter, transpose through shared memory, store
// Two accumulators (2 x 256 TMEM columns) let the epilogue of tile i overlap the main loop of
// tile i+1.
//
// Epilogues (a TMEM lane is an output feature, a column is a received row; stmatrix.trans turns
// the 8 x 8 fragments round so that a row's features leave as contiguous 16-byte stores):
//   kSwiGLU   the weight tensor holds 128 gate rows, then the 128 matching up rows, and so on;
//             the tensor map deals them out so that every warp's 32 lanes are 16 gate rows and
//             their 16 up rows.  Writes silu(gate)*up as bf16 into act[row, feature].
//   kScatter  converts to bf16 and stores each row to the buffer of the GPU the token came
//             from (peer memory over NVLink), at the return slot meta[row] & 0xFFFFF: this is the
//             combine step of the MoE layer fused into the last GEMM.
//
// The reference has no MoE layer; this kernel exists for the end-to-end benchmark.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>

#include "common.cuh"
#include "tcgen05.cuh"

namespace lplb {
namespace moe {

constexpr int kBM = 256, kBN = 256, kBK = 64, kUmmaK = 16;
constexpr int kCtaM = kBM / 2;       // weight rows per CTA of a pair
constexpr int kStepN = 32;           // received rows per tile are rounded up to this
constexpr int kRowBoxes = 4;         // received rows come in TMA boxes of 128, 64, 32 and 16 rows
constexpr int kGateRows = 16;        // gate (and up) rows of one epilogue warp
constexpr int kGateBlock = 128;      // gate rows in front of their up rows in the weight tensor
constexpr int kGemmThreads = 192;
constexpr int kTmemCols = 512;
constexpr uint32_t kStageBytesW = kCtaM * kBK * 2;
// The ring of operand stages.  A stage holds the weights and as many received rows as the launch's
// largest tile stages per CTA, so the ring is as deep as it can be: 6 stages with tiles of 256
// rows, 11 when no expert received more than 32 (64 tokens, both GEMMs: 643 us, with 6 stages 685).
constexpr uint32_t kRingBytes = 200 * 1024;
constexpr int kMaxStages = 11;
// Tile numbers on their way to the roles.  The producer announces tile i + 1 when it begins tile
// i; then all k blocks but the last kMaxStages have been computed, so with two or more k blocks
// per tile the accumulators of tile i - 7 are complete, the epilogue is through with tile i - 9,
// and no role still has to read a number older than that of tile i - 8.
constexpr int kTileSlots = 16;
static_assert(kMaxStages <= 12, "a slot could be overwritten before the epilogue has read it");
constexpr uint32_t kTurnBytes = kStepN * kCtaM * 2;  // 32 received rows x 128 features, two of these
constexpr uint32_t kBarBytes = 512;
constexpr size_t kGemmSmem = 1024 + kRingBytes + kBarBytes + 2 * kTurnBytes;
constexpr int kMaxLocalExperts = 128;
constexpr int kMaxRanks = 8;

enum Epilogue : int { kSwiGLU = 0, kScatter = 1 };

enum MoeErr : int { kMoeOk = 0, kMoeGemmTimeout = 11, kMoeFlagTimeout = 12, kMoeOverflow = 13 };

struct RowMaps {
  CUtensorMap box[kRowBoxes];
};

struct GemmArgs {
  const int* rows;        // [n_experts] rows received per local expert
  const int* row_start;   // [n_experts] first row of each expert in the A buffer
  int n_experts;
  int n_tiles_w;          // N / 256
  int k_blocks;           // K / 64
  // kSwiGLU
  __nv_bfloat16* act;     // [capacity, act_ld]
  int act_ld;             // N / 2
  // kScatter
  const int* meta;        // [capacity] (src_rank << 20) | return slot on the source rank
  __nv_bfloat16* comb[kMaxRanks];  // per source rank: [tokens * topk, out_ld]
  int out_ld;             // N
  // cross-GPU flags (epoch valued).  wait_flags: this rank's array [n_ranks], all must reach
  // `epoch` before the first tile is loaded.  done_flags[r]: rank r's array, slot my_rank is
  // raised by the last CTA of this launch.
  const uint32_t* wait_flags;
  uint32_t* done_flags[kMaxRanks];
  int n_ranks, my_rank;
  uint32_t epoch;
  unsigned* ticket;       // zero before launch; left at zero
  unsigned* next_tile;    // tiles taken beyond the first of every pair; zero before launch, left at zero
  int* status;            // first error code
  unsigned long long timeout_ns;
  // fused dispatch (FUSED kernels only): this rank's rows are sent while the tensor cores
  // work; an expert's tiles start once `arrived[e]` reached `arrive_target[e]`.  With
  // send_ctas == 0 warps 6-9 of every CTA send; with send_ctas > 0 (even: whole pairs) the last
  // `send_ctas` CTAs of the grid do nothing but send (all their warps) and the others only run
  // tiles.
  const __nv_bfloat16* x;        // [tokens, hidden] local hidden states
  const int* send_pair;          // [n_send] (local expert << 20) | pair index, in send order
  const int* send_target;        // [n_send] (rank << 24) | row, or -1
  const int* pair_slot;          // [pairs] return slot of every pair
  const int* n_send;             // number of send positions
  const int* arrive_target;      // [n_experts] cumulative rows expected per local expert
  __nv_bfloat16* recv_x[kMaxRanks];
  int* recv_meta[kMaxRanks];
  uint32_t* arrived[kMaxRanks];  // per rank: [n_experts] cumulative rows landed
  int topk, hidden;
  int send_ctas;
  unsigned long long* debug;     // optional [gridDim.x * 4] ns: kernel start, senders done, producer wait, end
};

constexpr int kSendWarps = 4;        // sender warps per CTA when every CTA also runs tiles
constexpr int kFusedThreads = 512;   // a dedicated sender CTA uses all 16 warps
constexpr int kFusedWarps = kFusedThreads / 32;

// One warp copies a row of `n_vec` 16-byte words with U independent loads in flight per lane.
template <int U>
__device__ __forceinline__ void copy_row(const uint4* __restrict__ src, uint4* __restrict__ dst, int n_vec, int lane) {
  int v = lane;
  for (; v + 32 * (U - 1) < n_vec; v += 32 * U) {
    uint4 q[U];
#pragma unroll
    for (int i = 0; i < U; ++i) q[i] = __ldg(&src[v + 32 * i]);
#pragma unroll
    for (int i = 0; i < U; ++i) dst[v + 32 * i] = q[i];
  }
  for (; v < n_vec; v += 32) dst[v] = __ldg(&src[v]);
}

// Sender role of the fused kernel: warp `gw` of `n_gw` streams blocks of eight consecutive
// send positions.  After a block, every lane fences its stores at system scope, the warp
// re-converges, and one lane per row bumps the target expert's arrival counter on the
// receiving GPU, which is what the receiver's TMA producer polls.
template <int U>
__device__ __forceinline__ void send_rows(const GemmArgs& a, int gw, int n_gw, int lane) {
  const int n_send = *a.n_send;
  const int vec_per_row = a.hidden / 8;
  for (int blk = gw; blk * 8 < n_send; blk += n_gw) {
    const int pos0 = blk * 8, cnt = min(8, n_send - pos0);
    int my_pair = -1, my_tgt = -1;
    if (lane < cnt) {
      my_pair = a.send_pair[pos0 + lane];
      my_tgt = a.send_target[pos0 + lane];
    }
    for (int j = 0; j < cnt; ++j) {
      const int pr = __shfl_sync(0xffffffffu, my_pair, j), tg = __shfl_sync(0xffffffffu, my_tgt, j);
      if (tg < 0) continue;
      const int pair = pr & 0xFFFFF, dr = tg >> 24, row = tg & 0xFFFFFF;
      const uint4* src = reinterpret_cast<const uint4*>(a.x + (size_t)(pair / a.topk) * a.hidden);
      uint4* dst = reinterpret_cast<uint4*>(a.recv_x[dr] + (size_t)row * a.hidden);
      copy_row<U>(src, dst, vec_per_row, lane);
      if (lane == 0) a.recv_meta[dr][row] = (a.my_rank << 20) | a.pair_slot[pair];
    }
    __threadfence_system();
    __syncwarp();
    if (lane < cnt && my_tgt >= 0) {
      uint32_t* ctr = a.arrived[my_tgt >> 24] + (my_pair >> 20);
      asm volatile("red.relaxed.sys.global.add.u32 [%0], 1;" ::"l"(ctr) : "memory");
    }
  }
}

// Walks the tile list: expert by expert, received rows fastest, so that the pairs at work at any
// moment share few weight tiles.  An expert's rows, in steps of kStepN, are split evenly over its
// tiles: tiles of one size keep the pairs that share operands in step.  (Tiles of 512 rows, two
// accumulators side by side, load a quarter less but lose more to the shallower ring and the
// uncovered epilogue: first GEMM at 8192 tokens 3170 us against 2906 us.)
struct TileCursor {
  int expert = 0, first_tile = 0;  // first tile id of `expert`
  int w = 0, row0 = 0, n = 0;      // the tile: weight tile, first row within the expert, rows rounded up to kStepN
  static __device__ __forceinline__ int steps_of(int rows) { return (rows + kStepN - 1) / kStepN; }
  static __device__ __forceinline__ int tiles_of(int steps) { return (steps + kBN / kStepN - 1) / (kBN / kStepN); }
  // Advance to tile `t`; returns false when t is past the last tile.
  __device__ __forceinline__ bool seek(int t, const int* rows, const GemmArgs& a) {
    for (; expert < a.n_experts; ++expert) {
      const int steps = steps_of(rows[expert]), tiles = tiles_of(steps);
      if (t < first_tile + tiles * a.n_tiles_w) {
        const int local = t - first_tile;
        w = local / tiles;
        const int i = local - w * tiles, base = steps / tiles, extra = steps - base * tiles;
        row0 = (i * base + min(i, extra)) * kStepN;
        n = (base + (i < extra)) * kStepN;
        return true;
      }
      first_tile += tiles * a.n_tiles_w;
    }
    return false;
  }
};

__device__ __forceinline__ float silu(float x) { return x / (1.f + __expf(-x)); }

__device__ __forceinline__ void st_global_v4(void* p, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.global.v4.b32 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

// tmap_w: weights (kSwiGLU: five dimensions, see gate_up_map; kScatter: boxes of 128 rows);
// rows: received rows in boxes of 128, 64, 32 and 16.  Issuing a box takes the producer some 55
// cycles whatever its size: in boxes of 16 rows, eight per K block, it held up the tensor cores.
template <int EPI, bool FUSED = false>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(FUSED ? kFusedThreads : kGemmThreads, 1)
grouped_gemm_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ RowMaps rows,
                    const GemmArgs args) {
  using namespace sm100;
  extern __shared__ uint8_t smem_raw[];
  // 1024-byte alignment is required by the 128-byte swizzle atoms; the offset is the same in both
  // CTAs of a pair, which the pair's matrix instructions rely on
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kRingBytes);
  uint8_t* smem_turn = smem + kRingBytes + kBarBytes;  // 2 x kTurnBytes, 256-byte aligned
  // bars: full[kMaxStages], empty[kMaxStages], tmem_full[2], tmem_empty[2], tile[kTileSlots]; full
  // and tmem_empty are used in the pair's first CTA only, the others in both
  const uint32_t bar_full = smem_u32(bars), bar_empty = smem_u32(bars + kMaxStages);
  const uint32_t bar_tfull = smem_u32(bars + 2 * kMaxStages), bar_tempty = smem_u32(bars + 2 * kMaxStages + 2);
  const uint32_t bar_tile = smem_u32(bars + 2 * kMaxStages + 4);
  static_assert((2 * kMaxStages + 4 + kTileSlots) * 8 <= kBarBytes, "barriers");
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  __shared__ int s_flags_ok;
  __shared__ int s_tile[kTileSlots];
  __shared__ int s_rows[kMaxLocalExperts], s_start[kMaxLocalExperts];
  __shared__ unsigned long long s_dst[EPI == kScatter ? 2 * kBN : 1];

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int half = (int)cluster_cta_rank();  // which CTA of the pair
  // CTAs [0, n_gemm) run tiles; in the fused kernel the rest (if any) only send rows
  const int n_gemm = FUSED ? (int)gridDim.x - args.send_ctas : (int)gridDim.x;
  const int n_pairs = n_gemm / 2, pair = (int)blockIdx.x / 2;
  const bool sender_cta = FUSED && (int)blockIdx.x >= n_gemm;
  unsigned long long* dbg = FUSED && args.debug ? args.debug + 4 * blockIdx.x : nullptr;

  allow_successor();
  const unsigned long long started = dbg ? timer_ns() : 0;
  if (threadIdx.x == 0) {
    abort_flag = 0;
    s_flags_ok = 1;
    for (int s = 0; s < kMaxStages; ++s) {
      mbar_init(bar_full + 8 * s, 1);
      mbar_init(bar_empty + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(bar_tfull + 8 * b, 1);
      mbar_init(bar_tempty + 8 * b, 8);  // four epilogue warps of either CTA
    }
    for (int s = 0; s < kTileSlots; ++s) mbar_init(bar_tile + 8 * s, 1);
    fence_barrier_init();
    tma_prefetch_desc(&tmap_w);
    for (int b = 0; b < kRowBoxes; ++b) tma_prefetch_desc(&rows.box[b]);
  }
  if (warp == 1) tmem_alloc(smem_u32(&tmem_slot), kTmemCols);
  wait_predecessors();
  if (threadIdx.x == 0) {
    if (dbg) dbg[0] = started;
    // every source rank must have finished writing this launch's A rows
    if (args.wait_flags != nullptr) {
      const uint64_t t0 = timer_ns();
      for (int r = 0; r < args.n_ranks; ++r) {
        for (;;) {
          uint32_t v;
          asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(args.wait_flags + r) : "memory");
          if ((int32_t)(v - args.epoch) >= 0) break;
          if (timer_ns() - t0 > args.timeout_ns) {
            s_flags_ok = 0;
            atomicCAS(args.status, 0, kMoeFlagTimeout);
            break;
          }
          __nanosleep(200);
        }
      }
    }
  }
  for (int e = threadIdx.x; e < args.n_experts; e += blockDim.x) {
    s_rows[e] = args.rows[e];
    s_start[e] = args.row_start[e];
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync();  // the peer's barriers are initialised and its tensor memory is allocated
  tc_fence_after_sync();
  const uint32_t tmem_base = tmem_slot;
  volatile int* abort = &abort_flag;
  const uint64_t budget = args.timeout_ns;
  const bool go = s_flags_ok != 0;
  TileCursor cur;
  int largest = 1;  // steps of the launch's largest tile
  for (int e = lane; e < args.n_experts; e += 32) {
    const int steps = TileCursor::steps_of(s_rows[e]), tiles = TileCursor::tiles_of(steps);
    if (tiles > 0) largest = max(largest, (steps + tiles - 1) / tiles);
  }
  largest = __reduce_max_sync(0xffffffffu, largest);
  const uint32_t stage_bytes = kStageBytesW + largest * (kStepN / 2) * kBK * 2;
  const uint32_t stages = min((uint32_t)kMaxStages, kRingBytes / stage_bytes);
  // Number of this pair's i-th tile, for every role but the one that hands them out; past the end
  // of the list (which ends the role) when the wait was given up.
  auto tile_number = [&](uint32_t i) -> int {
    if (i == 0) return pair;
    const uint32_t slot = i % kTileSlots;
    if (!mbar_wait_cluster(bar_tile + 8 * slot, ((i / kTileSlots) & 1) ^ (slot == 0), abort, budget)) return 0x7fffffff;
    return *(volatile int*)&s_tile[slot];
  };
  auto find = [&](int t) { return cur.seek(t, s_rows, args); };

  if (sender_cta) {
    // ---------------- dedicated sender CTA (never waits on anything) ----------------
    send_rows<7>(args, ((int)blockIdx.x - n_gemm) * kFusedWarps + warp, args.send_ctas * kFusedWarps, lane);
    if (dbg && lane == 0) atomicMax(&dbg[1], (unsigned long long)timer_ns());
  } else if (go && warp == 0) {
    // ---------------- TMA producer ----------------
    if (elect_one()) {
      // Peers wrote the received rows with ordinary stores, seen through thread 0's acquire of their
      // flags; the TMA loads below are another proxy.
      if (args.wait_flags != nullptr) fence_proxy_async_global();
      const uint32_t lead_full = map_to_rank(bar_full, 0);
      uint32_t s = 0, ph = 0;  // stage and its phase, running over all tiles of this pair
      int ready_expert = -1, t = pair;
      for (uint32_t i = 0; find(t) && !*abort;) {
        ++i;
        if (half == 0) {  // the pair's next tile, fetched while this one is loaded
          t = n_pairs + (int)atomicAdd(args.next_tile, 1u);
          const uint32_t slot = i % kTileSlots;
          for (uint32_t r = 0; r < 2; ++r) {
            st_cluster(map_to_rank(smem_u32(&s_tile[slot]), r), t);
            mbar_arrive_remote(map_to_rank(bar_tile + 8 * slot, r));
          }
        }
        if (FUSED && cur.expert != ready_expert) {
          // all rows of this expert must have landed (senders on every GPU count them in)
          const uint32_t* ctr = args.arrived[args.my_rank] + cur.expert;
          const uint32_t want = (uint32_t)args.arrive_target[cur.expert];
          const uint64_t t0 = timer_ns();
          for (;;) {
            uint32_t v;
            asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(ctr) : "memory");
            if ((int32_t)(v - want) >= 0) break;
            if (*abort || timer_ns() - t0 > budget) {
              *abort = 1;
              atomicCAS(args.status, 0, kMoeFlagTimeout);
              break;
            }
            __nanosleep(100);
          }
          if (dbg) dbg[2] += timer_ns() - t0;
          if (*abort) break;
          fence_proxy_async_global();
          ready_expert = cur.expert;
        }
        const int mine = cur.n / 2;  // received rows that this CTA stages
        const int row_t = s_start[cur.expert] + cur.row0 + half * mine;
        const int w_tile = cur.expert * args.n_tiles_w + cur.w;
        const uint32_t pair_bytes = 2 * (kStageBytesW + (uint32_t)mine * kBK * 2);
        for (int kb = 0; kb < args.k_blocks; ++kb) {
          if (!mbar_wait(bar_empty + 8 * s, ph ^ 1, abort, budget)) break;
          const uint32_t full = lead_full + 8 * s;
          if (half == 0) mbar_expect_tx(bar_full + 8 * s, pair_bytes);
          uint32_t dst = smem_u32(smem) + s * stage_bytes;
          if constexpr (EPI == kSwiGLU)
            tma_pair_load_5d(dst, &tmap_w, full, kb * kBK, half * (kCtaM / (2 * kGateRows)), w_tile);
          else
            tma_pair_load_2d(dst, &tmap_w, full, kb * kBK, w_tile * kBM + half * kCtaM);
          dst += kStageBytesW;
          int row = row_t;
#pragma unroll
          for (int b = 0; b < kRowBoxes; ++b) {
            const int n = kBN / 2 >> b;
            if (mine & n) {
              tma_pair_load_2d(dst, &rows.box[b], full, kb * kBK, row);
              dst += n * kBK * 2;
              row += n;
            }
          }
          if (++s == stages) s = 0, ph ^= 1;
        }
        if (half != 0) t = tile_number(i);
      }
    }
  } else if (go && warp == 1) {
    // ---------------- MMA issuer, for both CTAs ----------------
    if (half == 0 && elect_one()) {
      uint32_t s = 0, ph = 0;
      for (uint32_t tile_n = 0; find(tile_number(tile_n)) && !*abort; ++tile_n) {
        const uint32_t acc = tile_n & 1, acc_ph = (tile_n >> 1) & 1;
        if (!mbar_wait(bar_tempty + 8 * acc, acc_ph ^ 1, abort, budget)) break;
        tc_fence_after_sync();
        const uint32_t idesc = umma_idesc_bf16(kBM, cur.n);
        const uint32_t tmem_d = tmem_base + acc * kBN;
        bool ok = true;
        for (int kb = 0; kb < args.k_blocks; ++kb) {
          if (!mbar_wait(bar_full + 8 * s, ph, abort, budget)) {
            ok = false;
            break;
          }
          tc_fence_after_sync();
          const uint32_t base = smem_u32(smem) + s * stage_bytes;
          const uint64_t dw = umma_desc_sw128(base), dt = umma_desc_sw128(base + kStageBytesW);
#pragma unroll
          for (int k = 0; k < kBK / kUmmaK; ++k) {
            // advance 16 elements = 32 bytes along K inside the swizzled 128-byte row
            umma_pair_bf16(tmem_d, dw + (uint64_t)(k * kUmmaK * 2 >> 4), dt + (uint64_t)(k * kUmmaK * 2 >> 4), idesc,
                           (kb | k) != 0);
          }
          umma_pair_commit(bar_empty + 8 * s);  // stage reusable, in both CTAs, once these MMAs have read it
          if (++s == stages) s = 0, ph ^= 1;
        }
        if (!ok) break;
        umma_pair_commit(bar_tfull + 8 * acc);  // accumulator complete, in both CTAs
      }
    }
  } else if (FUSED && warp >= 6) {
    // ---------------- sender warps beside the tile roles (never wait on anything) ----------------
    if (args.send_ctas == 0 && warp < 6 + kSendWarps) {
      send_rows<4>(args, blockIdx.x * kSendWarps + (warp - 6), gridDim.x * kSendWarps, lane);
      if (dbg && lane == 0) atomicMax(&dbg[1], (unsigned long long)timer_ns());
    }
  } else if (go && warp >= 2) {
    // ---------------- epilogue ----------------
    const int quarter = warp & 3;  // TMEM lanes 32*quarter .. +31 are the ones this warp may read
    const int et = threadIdx.x - 64;
    uint32_t turn = 0;
    for (uint32_t tile_n = 0;; ++tile_n) {
      // All four warps leave the loop together: they meet at barriers below, and tcgen05.ld is a
      // whole-warp instruction.  A thread that gave up a wait finds no tile.
      const bool more = find(tile_number(tile_n));
      if (!epilogue_all(more && !*abort)) break;
      const uint32_t acc = tile_n & 1, acc_ph = (tile_n >> 1) & 1;
      const int left = s_rows[cur.expert] - cur.row0;  // rows of the expert from this tile's first on
      const size_t row0 = (size_t)s_start[cur.expert] + cur.row0;
      if constexpr (EPI == kScatter) {  // where every row of the tile goes
        for (int r = et; r < cur.n; r += 128) {
          unsigned long long to = 0;
          if (r < left) {
            const int mt = args.meta[row0 + r];
            to = reinterpret_cast<unsigned long long>(args.comb[(mt >> 20) & (kMaxRanks - 1)] +
                                                      (size_t)(mt & 0xFFFFF) * args.out_ld);
          }
          s_dst[acc * kBN + r] = to;
        }
      }
      if (!epilogue_all(mbar_wait(bar_tfull + 8 * acc, acc_ph, abort, budget))) break;
      tc_fence_after_sync();
      const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * kBN;
      for (int c0 = 0; c0 < cur.n; c0 += kStepN, turn ^= 1) {
        uint8_t* stage = smem_turn + turn * kTurnBytes;
        const uint32_t mine = smem_u32(stage);
        // fragments: thread l holds lanes l/4 and l/4 + 8 of a 16-lane half, columns 8j + 2(l%4) and the next
        uint32_t a[16], b[16];
        __syncwarp();
        tmem_ld_16x32(taddr + c0, a);                // lanes 0-15
        tmem_ld_16x32(taddr + (16u << 16) + c0, b);  // lanes 16-31
        tmem_ld_wait();
        if constexpr (EPI == kSwiGLU) {
          uint32_t o[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float v0 = silu(__uint_as_float(a[2 * j])) * __uint_as_float(b[2 * j]);
            const float v1 = silu(__uint_as_float(a[2 * j + 1])) * __uint_as_float(b[2 * j + 1]);
            o[j] = pack_bf16(v0, v1);
          }
#pragma unroll
          for (int h = 0; h < 2; ++h)  // 8 features each; 128-byte rows, 16-byte chunks swizzled by row
            stmatrix_trans(mine + lane * 128 + (((2 * quarter + h) ^ (lane & 7)) << 4), o[h], o[2 + h], o[4 + h], o[6 + h]);
          epilogue_sync();
          __nv_bfloat16* dst = args.act + (row0 + c0) * args.act_ld + (size_t)cur.w * (kBM / 2) + half * (kCtaM / 2);
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int r = (et >> 3) + 16 * i, chunk = et & 7;
            const uint4 v = *reinterpret_cast<const uint4*>(stage + r * 128 + ((chunk ^ (r & 7)) << 4));
            if (c0 + r < left) st_global_v4(dst + (size_t)r * args.act_ld + chunk * 8, v.x, v.y, v.z, v.w);
          }
        } else {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const uint32_t row = mine + lane * 256;
            stmatrix_trans(row + (((4 * quarter + h) ^ (lane & 7)) << 4),
                           pack_bf16(__uint_as_float(a[2 * h]), __uint_as_float(a[2 * h + 1])),
                           pack_bf16(__uint_as_float(a[4 + 2 * h]), __uint_as_float(a[5 + 2 * h])),
                           pack_bf16(__uint_as_float(a[8 + 2 * h]), __uint_as_float(a[9 + 2 * h])),
                           pack_bf16(__uint_as_float(a[12 + 2 * h]), __uint_as_float(a[13 + 2 * h])));
            stmatrix_trans(row + (((4 * quarter + 2 + h) ^ (lane & 7)) << 4),
                           pack_bf16(__uint_as_float(b[2 * h]), __uint_as_float(b[2 * h + 1])),
                           pack_bf16(__uint_as_float(b[4 + 2 * h]), __uint_as_float(b[5 + 2 * h])),
                           pack_bf16(__uint_as_float(b[8 + 2 * h]), __uint_as_float(b[9 + 2 * h])),
                           pack_bf16(__uint_as_float(b[12 + 2 * h]), __uint_as_float(b[13 + 2 * h])));
          }
          epilogue_sync();
          // 16 lanes write 256 contiguous bytes of a row (they cross NVLink)
          const size_t col = ((size_t)cur.w * kBM + half * kCtaM) * 2;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int r = (et >> 4) + 8 * i, chunk = et & 15;
            const uint4 v = *reinterpret_cast<const uint4*>(stage + r * 256 + ((chunk ^ (r & 7)) << 4));
            const unsigned long long to = s_dst[acc * kBN + c0 + r];
            if (to != 0) st_global_v4(reinterpret_cast<void*>(to + col + (size_t)chunk * 16), v.x, v.y, v.z, v.w);
          }
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive_remote(map_to_rank(bar_tempty + 8 * acc, 0));
    }
  }

  // ---------------- teardown ----------------
  if (*abort) {
    // A role gave up.  Give copies that may still be in flight a bounded time to land before
    // shared memory and TMEM are released.
    const uint64_t t0 = timer_ns();
    while (timer_ns() - t0 < 200000) __nanosleep(1000);
    if (threadIdx.x == 0) atomicCAS(args.status, 0, kMoeGemmTimeout);
  }
  if constexpr (EPI == kScatter) __threadfence_system();  // rows stored to peers are visible before the flag
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync();  // neither CTA leaves while the other may still signal it or read its operands
  if (warp == 1) tmem_dealloc(tmem_base, kTmemCols);
  if (dbg && threadIdx.x == 0) dbg[3] = timer_ns();
  if (threadIdx.x == 0 && args.ticket != nullptr) {
    __threadfence();
    if (atomicAdd(args.ticket, 1u) == gridDim.x - 1) {
      *args.ticket = 0;
      *args.next_tile = 0;  // every pair has taken its last number
      if constexpr (EPI == kScatter) {
        __threadfence_system();
        for (int r = 0; r < args.n_ranks; ++r)
          asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(args.done_flags[r] + args.my_rank), "r"(args.epoch)
                       : "memory");
      }
    }
  }
}

}  // namespace moe
}  // namespace lplb
