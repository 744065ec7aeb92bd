// Interior-point solver for LP groups of up to 64 ranks on double-precision matrix
// instructions (sm_100a).
//
// Same LP, same Mehrotra predictor-corrector iterates and same warm-start rule as the solvers
// in lp_solver.cuh and lp_block_solver.cuh.  What bounds a solve is one chain of dependent
// operations, so everything here is arranged by its latency (measured, cycles: multiply-add
// 8, shuffle 24, shared-memory store + load 36, mma.m8n8k4.f64 26, maximum of two doubles 24,
// integer maximum over a warp 22):
//
//   * The normal matrix lives in 8 x 8 tiles in the accumulator layout of mma.m8n8k4.f64 (lane
//     4 r + c: row r, columns 2 c and 2 c + 1).  The same two registers serve as operand A of the
//     tile, and as operand B of its transpose, when k runs over 0, 2, 4, 6 and then 1, 3, 5, 7:
//     no data moves between products.
//   * It is inverted in place by symmetric block sweeps instead of being factored: one multiply
//     by the inverse, a few matrix instructions, replaces each pair of substitutions.  Inside a
//     tile a sweep takes two pivots at a time (one reciprocal, of the 2 x 2 determinant); between
//     tiles it takes a whole 8 x 8 tile, and the warp that owns the next pivot tile inverts it
//     while the others still update theirs.
//   * Warp I holds tile row I and is the ranks 8 I .. 8 I + 7, four lanes each; a lane is one of the
//     rank's edges, so that no instruction is spent once per edge (8 ranks 11.3 -> 10.3 us with
//     the sweep below, before the refinement).  With one warp there is no barrier.
//   * Sums over ranks are two matrix instructions by a matrix of ones for two sums at a time
//     (65 cycles; three rounds of shuffles take 96 for one).
//   * Maxima are taken on integers that order like the doubles they stand for.
//   * Whatever does not depend on the centring parameter is done before it is known: the
//     corrector's step is linear in it.
//   * A product with an inverse is not as good as a substitution, so the step is refined once (kDamping).
//
// Solve kernel, two replicas per rank, unrelated instances, us a call back to back (the warp solver
// for 8 ranks, the thread-block solver above -> this one): 8 ranks 22.6 -> 10.4, 64 groups of 8 ranks
// 26.2 -> 12.3, 16 ranks 40.6 -> 17.9, 32 ranks 64.4 -> 24.8, 64 ranks 147 -> 46.  An iteration: 8 ranks 3.5 -> 1.4,
// 64 ranks 22.5 -> 6.6 us.
#pragma once

#include "lp_solver.cuh"

namespace lplb {

constexpr int kTileMaxGroup = 64;  // one warp per tile row, eight warps
constexpr int kTileMaxDup = 4;     // beyond, the per-rank state no longer fits the registers

// Near the optimum the normal matrix M Theta M^T + diag(s / y) is almost singular: its first term grows like 1 / mu and is
// singular (its columns sum to zero, among the ranks of every connected part), and s / y of a loaded rank shrinks like
// mu.  A factorisation survives that, since what it solves is a system next to the right one; an inverse does
// not: a product with it leaves a residual of machine precision times the condition number, and that residual is the
// next iterate's primal infeasibility.  So the inverse is that of a slightly heavier matrix (the diagonal of
// the first term grows by this much of itself, which bounds the condition number), and the step is refined once
// against the true equations.  17280 warm-started solves of groups of 8 ranks with some 30 tokens an expert: without
// the two 74 run into the iteration cap, with them none, and the iterations are those of a factorisation (mean 3.096 both);
// with a tolerance of 1e-6 it was two solves in three.  Shares are within 1e-7 of the norm of those of a factorisation,
// without the two within 1e-5; with 1e-9 here and no refinement it was 1e-3, with refinement and no addition a
// tolerance of 1e-6 still failed one time in five.  It costs 0.2 us an iteration with 8 ranks (64 groups 10.5 -> 11.4 us a
// call); left out while mu is above 1e-3 the branch costs the fused step more than the skipped work gives.
constexpr double kDamping = 1.0 / (1ull << 40);

// Warps (= tile rows, and tiles per row) that solve a group of g ranks.
__host__ __device__ constexpr int tile_rows(int g) { return g <= 8 ? 1 : (g <= 16 ? 2 : (g <= 32 ? 4 : 8)); }

#ifdef LPLB_HOST_SIM
using lplb_sim::double2;
#endif

// ---- primitives ---------------------------------------------------------------------------
// D = A B + C for an 8 x 4 by 4 x 8 product: lane 4 r + c passes A[r][c] and B[c][r] and holds
// columns 2 c, 2 c + 1 of row r of C and D.
__device__ __forceinline__ void mma8(double& d0, double& d1, double a, double b, double c0, double c1) {
#ifdef LPLB_HOST_SIM
  lplb_sim::mma8(d0, d1, a, b, c0, c1);
#else
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%4, %5};"
      : "=d"(d0), "=d"(d1)
      : "d"(a), "d"(b), "d"(c0), "d"(c1));
#endif
}

// The hardware's approximation of 1/x.  By the PTX manual it reads the upper 32 bits of x, of them 20 of the
// mantissa, and returns as many, so its relative error is near 2^-20; subnormals count as zeros.
__device__ __forceinline__ double rcp_seed(double x) {
#ifdef LPLB_HOST_SIM
  return lplb_sim::rcp_approx(x);
#else
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  return r;
#endif
}
// 1/x to a few ulp: one step of Householder's method of third order, r (1 + e + e^2) with e = 1 - x r.
// Three dependent operations where two Newton steps take four.
__device__ __forceinline__ double rcp3(double x) {
  const double r = rcp_seed(x), e = fma(-x, r, 1.0);
  return fma(r, fma(e, e, e), r);
}
// 1/x to about 2^-38, one Newton step: enough for the 26 bits of a step length, where the approximation
// alone is not.
__device__ __forceinline__ double rcp2(double x) {
  const double r = rcp_seed(x);
  return fma(r, fma(-x, r, 1.0), r);
}

#ifdef LPLB_HOST_SIM
inline int lowest_bit(unsigned x) { return __builtin_ctz(x); }
#else
__device__ __forceinline__ int lowest_bit(unsigned x) { return __ffs((int)x) - 1; }
#endif

#ifdef LPLB_HOST_SIM
using lplb_sim::from_words;
using lplb_sim::hi_word;
using lplb_sim::lo_word;
#else
__device__ __forceinline__ int hi_word(double x) { return __double2hiint(x); }
__device__ __forceinline__ int lo_word(double x) { return __double2loint(x); }
__device__ __forceinline__ double from_words(int hi, int lo) { return __hiloint2double(hi, lo); }
#endif

// A step of length 1 / x, or `limit` / x, keeps one variable at its bound; only the largest x counts,
// and only if it is above `limit`.  x in [1/2, 2^63) as an unsigned integer that orders like it, with 26
// bits behind the binary point, the rest cut off (the float ratios of the other solvers carry 23).
// Anything below 1/2, negative numbers too, becomes at most 63, which stands for a step of 1; anything from
// 2^63 on, infinity too, one of the 64 largest keys, which stand for next to none.
__device__ __forceinline__ unsigned step_key(double x) {
  const unsigned hi = (unsigned)min(max(hi_word(x), 0x3FE00000), 0x43DFFFFF) - 0x3FE00000u;
  return (hi << 6) | ((unsigned)lo_word(x) >> 26);
}
// min(limit / (the number behind `key`), 1)
__device__ __forceinline__ double step_from_key(unsigned key, double limit) {
  const double x = from_words((int)((key >> 6) + 0x3FE00000u), (int)(key << 26));
  const double a = limit * rcp2(x);
  return hi_word(a) >= 0x3FF00000 ? 1.0 : a;
}
// What a step length of one does to a variable x > 0, in units of x: the ratio that becomes a key.
__device__ __forceinline__ double step_ratio(double x, double dx) { return -dx * rcp2(x); }
// min(max(x, 0), 1)
__device__ __forceinline__ double clamp01(double x) {
  const int hi = hi_word(x);
  return hi < 0 ? 0.0 : (hi >= 0x3FF00000 ? 1.0 : x);
}
__device__ __forceinline__ double negative_part(double x) { return hi_word(x) < 0 ? x : 0.0; }

__device__ __forceinline__ double lane_get(double v, int lane) { return __shfl_sync(0xffffffffu, v, lane); }

// Largest of the lanes' values, exactly; the largest must be positive.
__device__ __forceinline__ double warp_max_positive(double x) {
  const int hi = __reduce_max_sync(0xffffffffu, hi_word(x));
  const unsigned lo = __reduce_max_sync(0xffffffffu, hi_word(x) == hi ? (unsigned)lo_word(x) : 0u);
  return from_words(hi, (int)lo);
}

// In: a symmetric positive definite 8 x 8 matrix, one tile.  Out: minus its inverse.  Four symmetric
// sweeps of two pivots each; with P the inverse of the 2 x 2 pivot block and U the two columns of
// the pivots, a sweep turns the block into -P, U into U P and the rest N into N - U P U^T.  One
// matrix instruction does all three: rows of the pivots pass P as operand A and all others
// -U P, columns of the pivots pass -1 at their own place as operand B and all others U, and
// the accumulator is zero in both.  (k = 2, 3 of the instruction stay empty.)  A pivot block
// that rounding drove singular counts as infinite: its unknowns become zero in the solves.
//
// A sweep is one dependent chain: block, determinant, reciprocal, matrix instruction.  The tile goes
// through shared memory, where every lane reads just the elements that it needs, zeros and ones
// included, because the ten shuffles and the selections between their results take longer:
// 641 cycles for the four sweeps, with shuffles 715 to 930, with the next pivot block computed ahead of
// the matrix instruction 710 to 1000 (more instructions on the same warp).
// `scratch`: kSweepScratch doubles per warp, prepared by sweep_scratch_init.
constexpr int kSweepZero = 128, kSweepOne = 144, kSweepScratch = 146;
__device__ __forceinline__ void sweep_scratch_init(double* scratch, int lane) {
  if (lane < kSweepScratch - kSweepZero) scratch[kSweepZero + lane] = lane == kSweepOne - kSweepZero ? -1.0 : 0.0;
  __syncwarp();
}
__device__ __forceinline__ void sweep_tile(double& n0, double& n1, int lane, double* scratch) {
  const int r = lane >> 2, c = lane & 3;
  const bool odd = c & 1, used = c < 2, own = (r & 1) == (c & 1);
  // offsets in `scratch` of this lane's element of U in its own column, of the other one, of the opposite
  // diagonal element of the pivot block, and of what replaces the first two in the pivots' rows
  const int mine_at = used ? 2 * (lane & 28) + odd : kSweepZero, other_at = used ? 2 * (lane & 28) + !odd : kSweepZero;
  const int opposite_at = odd ? 0 : 9;
  const int mine_pivot = kSweepOne + !(used && own), other_pivot = kSweepOne + !(used && !own);
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    const int copy = (h & 1) * 64;
    double* tile = scratch + copy;
    *reinterpret_cast<double2*>(tile + 2 * lane) = double2{n0, n1};
    __syncwarp();
    const bool pivot = (r >> 1) == h;
    const double2 ab = *reinterpret_cast<const double2*>(tile + 18 * h);  // the block is a b / b d
    const double d = tile[18 * h + 9], opposite = tile[18 * h + opposite_at];
    const double mine = scratch[pivot ? mine_pivot : mine_at + 2 * h + (used ? copy : 0)];
    const double other = scratch[pivot ? other_pivot : other_at + 2 * h + (used ? copy : 0)];
    const double det = fma(ab.x, d, -(ab.y * ab.y)), inv = rcp3(det);
    const bool ok = (unsigned)(hi_word(det) - 0x01000000) < 0x7E000000u;  // a positive, finite number
    const double num = fma(other, ab.y, -(mine * opposite));
    const double scale = from_words(ok ? hi_word(inv) : 0, lo_word(inv));  // finite, and times zero if not ok
    const bool fresh = pivot || c == h;
    mma8(n0, n1, (ok ? num : 0.0) * scale, mine, fresh ? 0.0 : n0, fresh ? 0.0 : n1);
  }
}

// ---- exchange between ranks -----------------------------------------------------------------
// Every rank has up to four lanes; lane c is its edge c % L, L = 1, 2 or 4 (of three edges the fourth is
// a dummy that carries no load).  With one warp a value of another rank is a shuffle away;
// otherwise it is published in a shared-memory vector, one vector per use so that one barrier
// per use suffices.
enum TileVec : int { kVecY, kVecG, kVecG1, kVecX, kVecX1, kVecBorder, kVecG0, kVecX0, kVecCount };  // per rank
enum TileEdgeVec : int { kEdgeF, kEdgeCw, kEdgeRhs, kEdgeOne, kEdgeCor, kEdgeCount };               // per edge
enum TileSum : int { kSumStart, kSumCold, kSumMu, kSumDual, kSumX, kSumX1, kSumAffine, kSumX0, kSumCount };
enum TileMax : int { kMaxLoad, kMaxDown, kMaxCount };
constexpr int kTileKeys = 4;

constexpr int kRoundsFrom = 8;  // tile rows from which on pivots go in rounds, see sweep_matrix

struct TileLayout {
  int sweep, rows_mat, u, pi, vec, edge, sums, maxes, keys, total;  // in doubles; every part starts on 16 bytes
};
__host__ __device__ constexpr TileLayout tile_layout(int nb, int d) {
  TileLayout l{};
  const int n = 8 * nb, many = nb > 1;
  int o = 0;
  l.sweep = o, o += nb * kSweepScratch;
  l.rows_mat = o, o += many * nb * nb * 64;  // normal matrix, tile by tile; during the inversion what is left of the pivots' columns
  l.u = o, o += (many && nb < kRoundsFrom) * 2 * nb * 64;  // pivot columns, two alternating copies
  l.pi = o, o += many * nb * 64;             // minus the inverses of the pivot tiles
  l.vec = o, o += many * kVecCount * n;
  l.edge = o, o += many * kEdgeCount * d * n;
  l.sums = o, o += many * kSumCount * nb * 2;
  l.maxes = o, o += many * kMaxCount * nb;
  l.keys = o, o += many * kTileKeys * nb / 2;  // unsigned
  l.total = o;
  return l;
}
// Shared memory of `teams` groups solved side by side by one CTA.
__host__ __device__ inline size_t tile_solver_smem_bytes(int g, int d, int teams = 1) {
  return sizeof(double) * (size_t)tile_layout(tile_rows(g), d).total * teams;
}

template <int NB, int D>
struct TileTeam {
  static constexpr int kRanks = 8 * NB, kLanes = D == 3 ? 4 : D;  // distinct lanes per rank
  static constexpr TileLayout kLay = tile_layout(NB, D);
  int warp, lane, r, c, edge, rank;
  double* sm;
  __device__ __forceinline__ TileTeam(int warp_, int lane_, double* sm_)
      : warp(warp_), lane(lane_), r(lane_ >> 2), c(lane_ & 3), edge(lane_ & (kLanes - 1)), rank(8 * warp_ + (lane_ >> 2)), sm(sm_) {}
  __device__ __forceinline__ double* sweep() const { return sm + kLay.sweep + warp * kSweepScratch; }
  __device__ __forceinline__ double* vec(int v) const { return sm + kLay.vec + v * kRanks; }
  __device__ __forceinline__ double* edges(int v) const { return sm + kLay.edge + (v * D + (edge < D ? edge : 0)) * kRanks; }
  __device__ __forceinline__ double2* sums(int v) const { return reinterpret_cast<double2*>(sm + kLay.sums) + v * NB; }
  __device__ __forceinline__ double* maxes(int v) const { return sm + kLay.maxes + v * NB; }
  __device__ __forceinline__ unsigned* keys(int v) const { return reinterpret_cast<unsigned*>(sm + kLay.keys) + v * NB; }
  __device__ __forceinline__ double2* mat() const { return mat(warp); }  // the warp's tile row
  __device__ __forceinline__ double2* mat(int row) const { return reinterpret_cast<double2*>(sm + kLay.rows_mat) + row * NB * 32; }
  __device__ __forceinline__ double2* pivot_col(int parity) const { return reinterpret_cast<double2*>(sm + kLay.u) + parity * NB * 32; }
  __device__ __forceinline__ double2* pivot_inv(int p) const { return reinterpret_cast<double2*>(sm + kLay.pi) + p * 32; }

  __device__ __forceinline__ void sync() const {
    if constexpr (NB > 1) {
#ifdef LPLB_HOST_SIM
      lplb_sim_named_barrier(NB * 32);
#else
      asm volatile("bar.sync 1, %0;" ::"n"(NB * 32) : "memory");
#endif
    }
  }
  __device__ __forceinline__ void put(int v, double x) const {
    if constexpr (NB > 1) {
      if (c == 0) vec(v)[rank] = x;
    }
  }
  __device__ __forceinline__ double get(int v, double mine, int of) const {
    if constexpr (NB > 1) return vec(v)[of];
    else return lane_get(mine, 4 * of);
  }
  // the same edge of another rank
  __device__ __forceinline__ void put_edge(int v, double x) const {
    if constexpr (NB > 1) {
      if (c < D) edges(v)[rank] = x;
    }
  }
  __device__ __forceinline__ double get_edge(int v, double mine, int of) const {
    if constexpr (NB > 1) return edges(v)[of];
    else return lane_get(mine, 4 * of + c);
  }
  // Several warps: the inverse, held as its negative's tiles, times a published vector.
  __device__ __forceinline__ double times_inverse(int v, const double (&n0)[NB], const double (&n1)[NB]) const {
    const double2* g = reinterpret_cast<const double2*>(vec(v));
    double p0 = 0.0, p1 = 0.0, x, same;
#pragma unroll
    for (int j = 0; j < NB; ++j) {
      const double2 a = g[4 * j + c];
      p0 = fma(n0[j], a.x, p0);
      p1 = fma(n1[j], a.y, p1);
    }
    mma8(x, same, p0 + p1, -1.0, 0.0, 0.0);
    return x;
  }
  // Sum over the rank's edges, on all its lanes.
  __device__ __forceinline__ double edge_sum(double x) const {
    if constexpr (D == 1) return x;
    double sum, same;
    mma8(sum, same, x, c < D ? 1.0 : 0.0, 0.0, 0.0);
    return sum;
  }
  // Sums over all lanes of all ranks (copies of an edge count once) of two values, in two halves around a barrier.
  __device__ __forceinline__ void sum_put(int slot, double& a, double& b) const {
    double d0, d1, s;
    if constexpr (kLanes <= 2) {
      // lanes with copies pass b instead: even rows of the product are the ranks' a, odd rows their b
      const int half = kLanes == 1 ? c : c >> 1;
      mma8(d0, d1, half == (r & 1) ? 1.0 : 0.0, (half & 1) ? b : a, 0.0, 0.0);
      s = d0 + d1;
    } else {
      double e0, e1;
      mma8(d0, d1, 1.0, a, 0.0, 0.0);
      mma8(e0, e1, 1.0, b, 0.0, 0.0);
      s = (r & 1) ? e0 + e1 : d0 + d1;
    }
    mma8(a, b, 1.0, s, 0.0, 0.0);
    if constexpr (NB > 1) {
      if (lane == 0) sums(slot)[warp] = double2{a, b};
    }
  }
  __device__ __forceinline__ void sum_put(int slot, double& a) const {
    double none = 0.0;
    sum_put(slot, a, none);
  }
  __device__ __forceinline__ void sum_get(int slot, double& a) const {
    double none = 0.0;
    sum_get(slot, a, none);
  }
  __device__ __forceinline__ void sum_get(int slot, double& a, double& b) const {
    if constexpr (NB > 1) {
      double2 v[NB];
#pragma unroll
      for (int k = 0; k < NB; ++k) v[k] = sums(slot)[k];
#pragma unroll
      for (int o = NB / 2; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < o; ++k) {
          v[k].x += v[k + o].x;
          v[k].y += v[k + o].y;
        }
      a = v[0].x;
      b = v[0].y;
    }
  }
  // Largest value, exactly; it must be positive.
  __device__ __forceinline__ double max_put(int slot, double x) const {
    x = warp_max_positive(x);
    if constexpr (NB > 1) {
      if (lane == 0) maxes(slot)[warp] = x;
    }
    return x;
  }
  __device__ __forceinline__ double max_get(int slot, double x) const {
    if constexpr (NB > 1) x = warp_max_positive(maxes(slot)[lane % NB]);
    return x;
  }
  __device__ __forceinline__ unsigned key_put(int slot, unsigned key) const {
    key = __reduce_max_sync(0xffffffffu, key);
    if constexpr (NB > 1) {
      if (lane == 0) keys(slot)[warp] = key;
    }
    return key;
  }
  __device__ __forceinline__ unsigned key_get(int slot, unsigned key) const {
    if constexpr (NB > 1) key = __reduce_max_sync(0xffffffffu, keys(slot)[lane % NB]);
    return key;
  }
  __device__ __forceinline__ bool all(int slot, bool ok) const {  // several warps: key_put(slot, !ok) and a barrier before
    if constexpr (NB == 1) return __all_sync(0xffffffffu, ok);
    else return key_get(slot, 0) == 0;
  }
};

// The order in which the tiles of the diagonal become pivots, from the topology.  Pivots that are not coupled at their turn
// do not touch each other's rows, so they go in one round: of a torus's ring of eight tile rows 0, 2, 4, 6, then 1, 5, then
// 3, then 7.  Byte r of `rounds` is the set of round r, byte p of `near` the rows that are coupled to pivot p at its turn, those
// of earlier pivots included.
// Edges (i, to[i * d + k]) of both tables; entries outside of the group are skipped.
inline TilePlan plan_tiles(int g, int d, const int* const (&tables)[2]) {
  const int nb = tile_rows(g);
  unsigned coupled[8] = {};
  for (const int* to : tables)
    for (int i = 0; i < g; ++i)
      for (int k = 0; k < d; ++k) {
        const int j = to[i * d + k];
        if (j < 0 || j >= g || j / 8 == i / 8) continue;
        coupled[i / 8] |= 1u << (j / 8);
        coupled[j / 8] |= 1u << (i / 8);
      }
  TilePlan plan;
  unsigned left = (1u << nb) - 1u;
  for (int r = 0; left != 0; ++r) {
    unsigned set = 0, blocked = 0;
    for (int p = 0; p < nb; ++p)
      if (((left & ~blocked) >> p) & 1u) {
        set |= 1u << p;
        blocked |= coupled[p];
      }
    for (int p = 0; p < nb; ++p) {
      if (!((set >> p) & 1u)) continue;
      plan.near |= (unsigned long long)coupled[p] << (8 * p);
      for (int i = 0; i < nb; ++i)  // a sweep couples all that its pivot is coupled to
        if ((coupled[p] >> i) & 1u) coupled[i] |= coupled[p] & ~(1u << i);
    }
    plan.rounds |= (unsigned long long)set << (8 * r);
    left &= ~set;
  }
  return plan;
}

// The inverse of the normal matrix, one tile row per warp: on entry n[j] is tile (I, j) of the
// matrix, on return minus the inverse's tile.  Block sweeps over the tiles of the diagonal: with P the
// pivot tile's inverse and U_I the tiles of its column, tile (I, J) becomes N_IJ - U_I P U_J^T, the
// pivot's column U_I P, its row P U_J^T and the pivot itself -P.  What bounds it is the chain of tile inversions, a round of
// pivots each, so as many pivots go at once as the topology leaves uncoupled, and tiles that are zero are left out.  (64 ranks
// of a torus in four rounds instead of eight pivots one after the other: a call 52.0 -> 49.3 us; 40 ranks of a ring with the line
// before scratch_after 42.9 -> 35.3.)  A column is published in the matrix's place in shared memory, every tile by the warp that
// owns its row.  Up to four tile rows leave little to do at once, and the plain loop is faster (32 ranks 10.6 us for
// three iterations in rounds, 10.1 one after the other).
template <int NB, int D>
__device__ __forceinline__ void sweep_matrix(const TileTeam<NB, D>& tm, const TilePlan& plan, double (&n0)[NB], double (&n1)[NB]) {
  if constexpr (NB == 1) {
    sweep_tile(n0[0], n1[0], tm.lane, tm.sweep());
  } else if constexpr (NB < kRoundsFrom) {
    if (tm.warp == 0) {
      double p0 = n0[0], p1 = n1[0];
      sweep_tile(p0, p1, tm.lane, tm.sweep());
      tm.pivot_inv(0)[tm.lane] = double2{p0, p1};
    }
#pragma unroll 1
    for (int p = 0; p < NB; ++p) {
      double2* u = tm.pivot_col(p & 1);
      const bool pivot = tm.warp == p;
      u[tm.warp * 32 + tm.lane] = double2{n0[0], n1[0]};
      tm.sync();
      const double2 m = tm.pivot_inv(p & 1)[tm.lane];  // -P
      double l0 = 0.0, l1 = 0.0;                       // -U_I P
      mma8(l0, l1, n0[0], m.x, l0, l1);
      mma8(l0, l1, n1[0], m.y, l0, l1);
      const double a0 = pivot ? -m.x : l0, a1 = pivot ? -m.y : l1;
      const double f0 = pivot ? m.x : -l0, f1 = pivot ? m.y : -l1;
      auto update = [&](int j) {
        const double2 b = u[((p + j) & (NB - 1)) * 32 + tm.lane];
        double d0 = pivot ? 0.0 : n0[j], d1 = pivot ? 0.0 : n1[j];
        mma8(d0, d1, a0, b.x, d0, d1);
        mma8(d0, d1, a1, b.y, d0, d1);
        n0[j - 1] = d0;
        n1[j - 1] = d1;
      };
      update(1);
      if (tm.warp == p + 1) {
        // The next pivot tile is ready: invert it while the others update theirs.  (The other tiles of
        // this row are due to be replaced by P U_J^T, so they need no update.)
        double p0 = n0[0], p1 = n1[0];
        sweep_tile(p0, p1, tm.lane, tm.sweep());
        tm.pivot_inv((p + 1) & 1)[tm.lane] = double2{p0, p1};
      } else {
#pragma unroll
        for (int j = 2; j < NB; ++j) update(j);
      }
      n0[NB - 1] = f0;
      n1[NB - 1] = f1;
    }
  } else {
    double2* row = tm.mat();
    const double2 diag = row[tm.warp * 32 + tm.lane];
    double g0 = diag.x, g1 = diag.y;  // the row's own pivot tile
    constexpr int kAtOnce = NB < 4 ? NB : 4;
#pragma unroll 1
    for (unsigned long long rounds = plan.rounds; rounds != 0; rounds >>= 8) {
      const unsigned set = (unsigned)rounds & 0xFFu, next = (unsigned)(rounds >> 8) & 0xFFu;
      const bool turn = (set >> tm.warp) & 1u;
      if (turn) {
        sweep_tile(g0, g1, tm.lane, tm.sweep());
        tm.pivot_inv(tm.warp)[tm.lane] = double2{g0, g1};
      }
      // What the updates below add to is zero in the pivots' columns and in their rows, and in its own column a pivot
      // stands for minus the identity: so N_IJ + (-U_I P) U_J^T, U_I P and P U_J^T are all one product, without a choice.
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        if ((set >> j) & 1u) {
          if (j == tm.warp) row[j * 32 + tm.lane] = double2{tm.r == 2 * tm.c ? -1.0 : 0.0, tm.r == 2 * tm.c + 1 ? -1.0 : 0.0};
          else row[j * 32 + tm.lane] = double2{n0[j], n1[j]};
          n0[j] = n1[j] = 0.0;
        } else if (turn) {
          n0[j] = n1[j] = 0.0;
        }
      }
      tm.sync();
#pragma unroll 1
      for (unsigned pivots = set; pivots != 0; pivots &= pivots - 1) {
        const int p = lowest_bit(pivots);
        const unsigned near = (unsigned)(plan.near >> (8 * p)) & 0xFFu;
        const bool pivot = p == tm.warp;
        if (!pivot && !((near >> tm.warp) & 1u)) continue;
        const double2 m = tm.pivot_inv(p)[tm.lane];  // -P
        double a0 = -m.x, a1 = -m.y;
        if (!pivot) {
          const double2 u = row[p * 32 + tm.lane];
          a0 = a1 = 0.0;  // -U_I P
          mma8(a0, a1, u.x, m.x, a0, a1);
          mma8(a0, a1, u.y, m.y, a0, a1);
          mma8(g0, g1, a0, u.x, g0, g1);
          mma8(g0, g1, a1, u.y, g0, g1);
          // The other tiles of a row that holds a pivot of the next round are due to be replaced by P U_J^T, so they need no
          // update, and its pivot can be inverted at once.
          if ((next >> tm.warp) & 1u) continue;
        }
#pragma unroll
        for (int j0 = 0; j0 < NB; j0 += kAtOnce) {
          if ((((near | 1u << p) >> j0) & ((1u << kAtOnce) - 1u)) == 0) continue;
          double2 b[kAtOnce];
#pragma unroll
          for (int j = 0; j < kAtOnce; ++j) b[j] = tm.mat(j0 + j)[p * 32 + tm.lane];
#pragma unroll
          for (int j = 0; j < kAtOnce; ++j) mma8(n0[j0 + j], n1[j0 + j], a0, b[j].x, n0[j0 + j], n1[j0 + j]);
#pragma unroll
          for (int j = 0; j < kAtOnce; ++j) mma8(n0[j0 + j], n1[j0 + j], a1, b[j].y, n0[j0 + j], n1[j0 + j]);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < NB; ++j)
      if (j == tm.warp) {
        n0[j] = g0;
        n1[j] = g1;
      }
  }
}

// A lane's part of the saved iterate of its group, read whether it is valid or not (the slot is always
// allocated), so that whoever waits for the counts has the loads behind it by then.
struct TileStart {
  double f = 0.5, v = 0.5, z = 1.0, q = 1.0, s = 1.0, y = 0.0, t = 0.0;
  bool saved = false;
};
// `anchor`: the rank's slot, or null for a rank that does not take part; `group_anchor`: that of the group's first rank.
template <int D>
__device__ __forceinline__ TileStart load_tile_start(int edge, const double* anchor, const double* group_anchor,
                                                     const int* anchor_valid) {
  TileStart a;
  if (anchor != nullptr) {
    if (edge < D) {
      a.f = anchor[edge];
      a.v = anchor[D + edge];
      a.z = anchor[2 * D + edge];
      a.q = anchor[3 * D + edge];
    }
    a.s = anchor[4 * D];
    a.y = anchor[4 * D + 1];
  }
  if (group_anchor != nullptr) {
    a.t = group_anchor[4 * D + 2];
    a.saved = *anchor_valid != 0;
  }
  return a;
}

// One group of at most 8 NB ranks, solved by NB warps (all of them call; `warp` counts from 0 within the
// group).  Lane 4 r + c of warp I is edge c of rank 8 I + r (see above) and passes that bundle's load, the
// rank's non-replicated load, and the ranks whose bundle it holds (`src`) and that hold its own (`dst`); dummies
// and ranks from `rows` on, which do not take part, pass no load and themselves.  All four lanes of a
// rank pass `mine`, the rank's whole own load.  `sm`: tile_solver_smem_bytes of shared memory, 16-byte
// aligned.  `anchor`: the rank's slot of the warm-start state or null; `group_anchor` the slot of the group's first rank;
// `early`: what load_tile_start found there, or null.  The outcome is the same on every lane, the share is the lane's own.
template <int NB, int D>
__device__ __forceinline__ IpmOutcome ipm_solve_tiles(const int warp, const int lane, const int rows, const double w_in,
                                                      const double fixed, const double own_load, const int src,
                                                      const int dst, const IpmParams prm, double& f_out, const TileStart* early,
                                                      double* anchor, const double* group_anchor, int* anchor_valid, double* sm) {
  constexpr double kEta = 0.995;
  const TileTeam<NB, D> tm(warp, lane, sm);
  const int c = tm.c, rank = tm.rank;
  const bool live = rank < rows, real = tm.edge < D;
  const bool first = tm.edge == 0;  // the lane that adds the rank's own part to sums over lanes
  sweep_scratch_init(tm.sweep(), lane);
  // The saved iterate's loads are in flight while the scaling is computed, unless the caller has made them already.
  const TileStart start = early != nullptr ? *early : load_tile_start<D>(tm.edge, live ? anchor : nullptr, group_anchor, anchor_valid);
  const bool slot = anchor != nullptr && live;
  const double fa = start.f, va = start.v, za = start.z, qa = start.q, sa = start.s, ya = start.y, ta = start.t;
  const bool saved_before = start.saved;

  const double kcomp = (double)(rows + 2 * rows * D), inv_kcomp = rcp3(kcomp), inv_rows = rcp3((double)rows);

  // ---- where this lane's off-diagonal terms of the matrix go -----------------------------------
  // One warp: factors 0 or -1 of all the rank's terms for the lane's two columns.  Several: the places of the
  // lane's two terms in the tile row, written once per iteration.  Terms of a rank that share a
  // column are merged, in one order, so that whoever writes such a place writes the same.
  double cd[NB == 1 ? D : 1][2], cs[NB == 1 ? D : 1][2];
  double *place_dst = nullptr, *place_src = nullptr, *place_diag = nullptr;
  unsigned same_dst = 0, same_src = 0;  // bit 2 d: the dst term of edge d shares the column, bit 2 d + 1: its src term
  {
    int all_dst[D], all_src[D];
#pragma unroll
    for (int d = 0; d < D; ++d) {
      all_dst[d] = __shfl_sync(0xffffffffu, dst, (lane & 28) | d);
      all_src[d] = __shfl_sync(0xffffffffu, src, (lane & 28) | d);
    }
    if constexpr (NB == 1) {
#pragma unroll
      for (int d = 0; d < D; ++d)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          cd[d][e] = all_dst[d] == 2 * c + e ? -1.0 : 0.0;
          cs[d][e] = all_src[d] == 2 * c + e ? -1.0 : 0.0;
        }
    } else {
      double2* mat = tm.mat();
      if constexpr (NB < kRoundsFrom)
        for (int j = 0; j < NB; ++j) mat[j * 32 + lane] = double2{0.0, 0.0};
      auto at = [&](int col) { return reinterpret_cast<double*>(mat) + ((col >> 3) * 32 + 4 * tm.r + ((col & 7) >> 1)) * 2 + (col & 1); };
#pragma unroll
      for (int d = 0; d < D; ++d) {
        same_dst |= (all_dst[d] == dst ? 1u : 0u) << (2 * d) | (all_src[d] == dst ? 2u : 0u) << (2 * d);
        same_src |= (all_dst[d] == src ? 1u : 0u) << (2 * d) | (all_src[d] == src ? 2u : 0u) << (2 * d);
      }
      if (live && c < D) {  // a self edge has no terms
        if (dst != rank) place_dst = at(dst);
        if (src != rank) place_src = at(src);
      }
      if (c == 0) place_diag = at(rank);
      __syncwarp();
    }
  }

  // ---- scale so that the mean rank load is 1 ---------------------------------------
  double total = first && live ? own_load : 0.0;
  tm.put_edge(kEdgeF, w_in);
  tm.sum_put(kSumStart, total);
  tm.sync();
  tm.sum_get(kSumStart, total);
  const bool empty = !(total > 0.0);
  const double inv_scale = empty ? 0.0 : (double)rows * rcp3(total);
  const double base = (fixed + tm.edge_sum(tm.get_edge(kEdgeF, w_in, src))) * inv_scale;
  // a self edge moves no load: its column of M is zero, its load is already part of `base`
  const double w = dst == rank ? 0.0 : w_in * inv_scale, ww = w * w;

  // ---- warm start from the anchor, if it still fits the data -----------------------------
  bool cold;
  {
    const double x = w * fa;
    tm.put_edge(kEdgeCw, x);
    tm.sync();
    const double mfa = tm.edge_sum(x - tm.get_edge(kEdgeCw, x, src));
    const bool near = !slot || fabs(ta - base - mfa - sa) <= prm.guard;
    if constexpr (NB > 1) {
      tm.key_put(0, near ? 0u : 1u);
      tm.sync();
    }
    cold = !(tm.all(0, near) && saved_before && !empty);
  }
  // With one warp the rows past a smaller group's last rank take part; they save no iterate and start
  // cold beside a warm group.  A rank that does not take part keeps s = 1, y = 0 all along.
  const bool start_cold = cold || !slot;
  double f = start_cold ? 0.5 : fa, v = start_cold ? 0.5 : va, z = start_cold ? 1.0 : za, q = start_cold ? 1.0 : qa;
  double t = ta, s = start_cold ? 1.0 : sa, y = start_cold ? (live ? inv_rows : 0.0) : ya;
  if (NB == 1 ? __any_sync(0xffffffffu, live && start_cold) : cold) {  // feasible start
    const double x = 0.5 * w;
    tm.put_edge(kEdgeRhs, x);
    tm.sync();
    const double load = base + tm.edge_sum(x - tm.get_edge(kEdgeRhs, x, src));
    double lmax = tm.max_put(kMaxLoad, live ? load : -1.0);
    tm.sync();
    lmax = tm.max_get(kMaxLoad, lmax);
    double down = tm.max_put(kMaxDown, live ? (lmax + 1.0) - load : -1.0);
    tm.sync();
    const double lmin = (lmax + 1.0) - tm.max_get(kMaxDown, down);
    const double ct = lmax + 0.5 * (lmax - lmin) + 0.05;
    if (live && start_cold) s = ct - load;
    if (cold) t = ct;
    double sum = live && first ? (ct - load) * inv_rows : 0.0;
    tm.sum_put(kSumCold, sum);
    tm.sync();
    tm.sum_get(kSumCold, sum);
    if (start_cold) z = q = 2.0 * (sum * inv_rows);
  }
  bool saved = false, done = empty;
  int iters = 0;
  double gap = 1e300, gap_scale = 1.0;

#pragma unroll 1
  for (int it = 0;; ++it) {
    // ---- weights and residuals --------------------------------------------------------------
    const double fv = f * v, inv_fv = rcp3(fv), inv_y = rcp3(live ? y : 1.0);
    const double theta = fv * rcp3(fma(z, v, q * f));  // 1 / (z / f + q / v)
    const double cw = theta * ww, wf = w * f, wt = w * theta;
    const double inv_f = v * inv_fv, inv_v = f * inv_fv;
    tm.put_edge(kEdgeF, wf);
    tm.put_edge(kEdgeCw, cw);
    tm.put(kVecY, y);
    tm.sync();
    const double held = tm.get_edge(kEdgeCw, cw, src);
    const double load = base + tm.edge_sum(wf - tm.get_edge(kEdgeF, wf, src));
    const double wy = w * (y - tm.get(kVecY, y, dst));
    const double r_u = 1.0 - f - v;
    // right-hand sides: the predictor's, and the part of the corrector's that goes with sigma mu
    const double qv = q * inv_v, rd = fma(qv, r_u, -wy), x_rhs = wt * rd, x_one = wt * (inv_f - inv_v);
    tm.put_edge(kEdgeRhs, x_rhs);
    tm.put_edge(kEdgeOne, x_one);
    // gap, complementarity and feasibility
    double mu = real ? fma(z, f, q * v) : 0.0, dual_sum = real ? negative_part(z - q - wy) - q : 0.0, sum_y = 0.0;
    if (first) {
      mu = fma(s, y, mu);
      dual_sum = fma(y, base, dual_sum);
      sum_y = y;
    }
    if (!live) mu = dual_sum = 0.0;
    const bool feasible = !live || !real || fabs(r_u) <= prm.tol;
    tm.sum_put(kSumMu, mu, sum_y);
    tm.sum_put(kSumDual, dual_sum);
    double primal = tm.max_put(kMaxLoad, live ? load : -1.0);
    if constexpr (NB > 1) tm.key_put(0, feasible ? 0u : 1u);
    // ---- normal matrix ----------------------------------------------------------------------
    double n0[NB], n1[NB];
    {
      double val[2 * D], moved = 0.0;  // the rank's terms: theta w^2 of its own and of the held bundles
#pragma unroll
      for (int d = 0; d < D; ++d) {
        val[2 * d] = D == 1 ? cw : lane_get(cw, (lane & 28) | d);
        val[2 * d + 1] = D == 1 ? held : lane_get(held, (lane & 28) | d);
        moved += val[2 * d] + val[2 * d + 1];
      }
      const double diag = live ? fma(moved, 1.0 + kDamping, s * inv_y) : 1.0;
      if constexpr (NB == 1) {
        double e0 = rank == 2 * c ? diag : 0.0, e1 = rank == 2 * c + 1 ? diag : 0.0, h0 = 0.0, h1 = 0.0;
#pragma unroll
        for (int d = 0; d < D; ++d) {
          e0 = fma(cd[d][0], val[2 * d], e0);
          e1 = fma(cd[d][1], val[2 * d], e1);
          h0 = fma(cs[d][0], val[2 * d + 1], h0);
          h1 = fma(cs[d][1], val[2 * d + 1], h1);
        }
        n0[0] = e0 + h0;
        n1[0] = e1 + h1;
      } else {
        double at_dst = 0.0, at_src = 0.0;
#pragma unroll
        for (int k = 0; k < 2 * D; ++k) {
          at_dst -= (same_dst >> k) & 1u ? val[k] : 0.0;
          at_src -= (same_src >> k) & 1u ? val[k] : 0.0;
        }
        if constexpr (NB >= kRoundsFrom) {  // the last inversion has left its columns here; several barriers are behind it
          double2* mat = tm.mat();
#pragma unroll
          for (int j = 0; j < NB; ++j) mat[j * 32 + lane] = double2{0.0, 0.0};
          __syncwarp();
        }
        if (place_dst != nullptr) *place_dst = at_dst;
        if (place_src != nullptr) *place_src = at_src;
        if (place_diag != nullptr) *place_diag = diag;
      }
    }
    tm.sync();
    const double g_edges = tm.edge_sum(x_rhs - tm.get_edge(kEdgeRhs, x_rhs, src));
    const double o_edges = tm.edge_sum(x_one - tm.get_edge(kEdgeOne, x_one, src));
    const double g = live ? load - t + g_edges : 0.0, g_one = live ? inv_y + o_edges : 0.0;
    // ---- stopping test ------------------------------------------------------------------------
    tm.sum_get(kSumMu, mu, sum_y);
    tm.sum_get(kSumDual, dual_sum);
    primal = tm.max_get(kMaxLoad, primal);
    mu *= inv_kcomp;
    const double r_t = 1.0 - sum_y;
    const bool all_feasible = tm.all(0, feasible);
    if (!done) {
      gap = primal - dual_sum;  // absolute here, made relative once at the end
      gap_scale = fabs(primal);
      // at mu ~ 1e-13 the iterate is optimal to machine precision: stop instead of dividing by it
      if ((gap <= prm.tol * gap_scale && all_feasible && fabs(r_t) <= prm.tol) || mu <= 1e-13) done = true;
    }
    // A cold solve leaves its first iterate at or below snap_mu behind as the next anchor.
    if (cold && !saved && !empty && mu <= prm.snap_mu) {
      if (slot && c < D) {
        anchor[c] = f;
        anchor[D + c] = v;
        anchor[2 * D + c] = z;
        anchor[3 * D + c] = q;
        if (c == 0) {
          anchor[4 * D] = s;
          anchor[4 * D + 1] = y;
          anchor[4 * D + 2] = t;
          if (rank == 0) *anchor_valid = 1;
        }
      }
      saved = true;
    }
    if (done || it >= prm.max_iters) break;
    ++iters;

    // ---- inverse, and its products with (g, g_one) and with ones: the border column of sum(dy) = r_t --------
    if constexpr (NB > 1) {
      const double2* mat = tm.mat();
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        const double2 e = mat[j * 32 + lane];
        n0[j] = e.x;
        n1[j] = e.y;
      }
    }
    tm.put(kVecG, g);
    tm.put(kVecG1, g_one);
    sweep_matrix<NB, D>(tm, prm.plan, n0, n1);  // with several warps its barriers also publish the right-hand sides
    double x, x1, border, same;
    {
      double rs = 0.0;
#pragma unroll
      for (int j = 0; j < NB; ++j) rs += n0[j] + n1[j];
      mma8(border, same, rs, -1.0, 0.0, 0.0);
      if constexpr (NB == 1) {
        // even columns of the product carry g, odd ones g_one: lane 4 r + c fetches the element of ranks
        // 2 c and 2 c + 1 from a lane that holds the one that column r is made of
        const double pick = (c & 1) ? g_one : g;
        const int from = 8 * c + (tm.r & 1);
        const double b0 = lane_get(pick, from), b1 = lane_get(pick, from + 4);
        mma8(x, x1, -n0[0], b0, 0.0, 0.0);
        mma8(x, x1, -n1[0], b1, x, x1);
      } else {
        const double2* gv = reinterpret_cast<const double2*>(tm.vec(kVecG));
        const double2* ov = reinterpret_cast<const double2*>(tm.vec(kVecG1));
        double p0 = 0.0, p1 = 0.0, o0 = 0.0, o1 = 0.0;
#pragma unroll
        for (int j = 0; j < NB; ++j) {
          const double2 a = gv[4 * j + c], b = ov[4 * j + c];
          p0 = fma(n0[j], a.x, p0);
          p1 = fma(n1[j], a.y, p1);
          o0 = fma(n0[j], b.x, o0);
          o1 = fma(n1[j], b.y, o1);
        }
        mma8(x, same, p0 + p1, -1.0, 0.0, 0.0);
        mma8(x1, same, o0 + o1, -1.0, 0.0, 0.0);
      }
    }
    if (!live) border = 0.0;
    tm.put(kVecX, x);
    tm.put(kVecX1, x1);
    tm.put(kVecBorder, border);
    double sum_x = first ? x : 0.0, sum_b = first ? border : 0.0, sum_x1 = first ? x1 : 0.0;
    tm.sum_put(kSumX, sum_x, sum_b);
    tm.sum_put(kSumX1, sum_x1);
    tm.sync();
    tm.sum_get(kSumX, sum_x, sum_b);
    tm.sum_get(kSumX1, sum_x1);
    const double inv_sum_b = rcp3(sum_b), inv_mu = rcp3(kcomp * mu);
    // ---- predictor ---------------------------------------------------------------------------
    // df = theta (rd - w (dy - dy_dst)) with dy = x - dt border, as e + dt e_b
    const double e = fma(-wt, x - tm.get(kVecX, x, dst), theta * rd);
    const double e_b = wt * (border - tm.get(kVecBorder, border, dst));
    const double e_1 = fma(-wt, x1 - tm.get(kVecX1, x1, dst), theta * (inv_f - inv_v));
    const double si = s * inv_y, zi = z * inv_f;
    double dt = (sum_x - r_t) * inv_sum_b;
    double dy = fma(-dt, border, x), ds = fma(-si, dy, -s);
    double df = fma(dt, e_b, e), dv = r_u - df, dz = fma(-zi, df, -z), dq = fma(-qv, dv, -q);
    // the predictor takes every complementarity product to zero, so dz / z = -1 - df / f, and so on
    const double tf = -df * inv_f, tv = -dv * inv_v, ty = -dy * inv_y;
    unsigned key_p = max(step_key(1.0 - ty), max(step_key(tf), step_key(tv)));
    unsigned key_d = max(step_key(ty), max(step_key(1.0 - tf), step_key(1.0 - tv)));
    double c_p = real ? fma(z, df, q * dv) : 0.0, c_pd = real ? fma(df, dz, dv * dq) : 0.0;
    if (first) {
      c_p = fma(y, ds, c_p);
      c_pd = fma(ds, dy, c_pd);
    }
    const double p_f = dz * -tf, p_v = dq * -tv, p_s = ds * -ty;  // dz df / f, dq dv / v, ds dy / y
    const double rc = rd - p_f + p_v, x_cor = wt * rc;
    tm.put_edge(kEdgeCor, x_cor);
    if (!live) c_p = c_pd = 0.0;
    key_p = tm.key_put(0, live && real ? key_p : 0u);
    key_d = tm.key_put(1, live && real ? key_d : 0u);
    tm.sum_put(kSumAffine, c_p, c_pd);
    tm.sync();
    // ---- corrector ---------------------------------------------------------------------------
    const double c_edges = tm.edge_sum(x_cor - tm.get_edge(kEdgeCor, x_cor, src));
    const double g0 = live ? load - t - p_s + c_edges : 0.0;
    tm.put(kVecG0, g0);
    tm.sum_get(kSumAffine, c_p, c_pd);
    const double ap0 = step_from_key(tm.key_get(0, key_p), 1.0), ad0 = step_from_key(tm.key_get(1, key_d), 1.0);
    // complementarity after the affine step; sum x dz = -kcomp mu - sum z dx
    const double comp_aff = fma(ap0 * ad0, c_pd, fma(ap0 - ad0, c_p, kcomp * mu * (1.0 - ad0)));
    const double ratio = clamp01(comp_aff * inv_mu);
    const double sig_mu = ratio * ratio * ratio * mu;
    double x0;
    if constexpr (NB == 1) {
      const double b0 = lane_get(g0, 8 * c), b1 = lane_get(g0, 8 * c + 4);
      mma8(x0, same, -n0[0], b0, 0.0, 0.0);
      mma8(x0, same, -n1[0], b1, x0, same);
    } else {
      tm.sync();
      x0 = tm.times_inverse(kVecG0, n0, n1);
      tm.put(kVecX0, x0);
    }
    double sum_x0 = first ? x0 : 0.0;
    tm.sum_put(kSumX0, sum_x0);
    tm.sync();
    tm.sum_get(kSumX0, sum_x0);
    const double e0 = fma(-wt, x0 - tm.get(kVecX0, x0, dst), theta * rc);
    dt = (fma(sig_mu, sum_x1, sum_x0) - r_t) * inv_sum_b;
    dy = fma(-dt, border, fma(sig_mu, x1, x0));
    ds = fma(-si, dy, fma(sig_mu, inv_y, -s - p_s));
    df = fma(dt, e_b, fma(sig_mu, e_1, e0));
    // ---- refinement: what the step leaves of t - load - s = 0 is put right by a second product ----------
    // (through vectors and a sum whose last readers are behind a barrier by then)
    {
      const double moved = w * df;
      tm.put_edge(kEdgeCor, moved);
      tm.sync();
      const double m_edges = tm.edge_sum(moved - tm.get_edge(kEdgeCor, moved, src));
      const double left = live ? (load - t - dt) + (s + ds) + m_edges : 0.0;
      tm.put(kVecG0, left);
      double fix;
      if constexpr (NB == 1) {
        const double b0 = lane_get(left, 8 * c), b1 = lane_get(left, 8 * c + 4);
        mma8(fix, same, -n0[0], b0, 0.0, 0.0);
        mma8(fix, same, -n1[0], b1, fix, same);
      } else {
        tm.sync();
        fix = tm.times_inverse(kVecG0, n0, n1);
        tm.put(kVecX0, fix);
      }
      double sum_fix = first ? fix : 0.0;
      tm.sum_put(kSumX0, sum_fix);
      tm.sync();
      tm.sum_get(kSumX0, sum_fix);
      const double more = sum_fix * inv_sum_b;
      df = fma(more, e_b, fma(-wt, fix - tm.get(kVecX0, fix, dst), df));
      fix = fma(-more, border, fix);
      dt += more;
      dy += fix;
      ds = fma(-si, fix, ds);
    }
    dv = r_u - df;
    dz = fma(-zi, df, fma(sig_mu, inv_f, -z - p_f));
    dq = fma(-qv, dv, fma(sig_mu, inv_v, -q - p_v));
    key_p = max(step_key(step_ratio(s, ds)), max(step_key(-df * inv_f), step_key(-dv * inv_v)));
    key_d = max(step_key(-dy * inv_y), max(step_key(step_ratio(z, dz)), step_key(step_ratio(q, dq))));
    key_p = tm.key_put(2, live && real ? key_p : 0u);
    key_d = tm.key_put(3, live && real ? key_d : 0u);
    tm.sync();
    const double ap = step_from_key(tm.key_get(2, key_p), kEta), ad = step_from_key(tm.key_get(3, key_d), kEta);
    t = fma(ap, dt, t);
    if (live) {
      s = fma(ap, ds, s);
      y = fma(ad, dy, y);
    }
    if (live && real) {
      f = fma(ap, df, f);
      v = fma(ap, dv, v);
      z = fma(ad, dz, z);
      q = fma(ad, dq, q);
    }
  }

  const bool ok = !live || !real || (f == f && fabs(f) < 1e300);
  f_out = fmin(fmax(f, 0.0), 1.0);
  if constexpr (NB > 1) {
    tm.sync();  // every warp is through with key 0
    tm.key_put(0, ok ? 0u : 1u);
    tm.sync();
  }
  const bool finite = tm.all(0, ok);
  if (!finite) f_out = 0.5;
  if (empty) f_out = 1.0;  // nothing to balance: keep everything on the origin
  IpmOutcome out;
  out.iters = iters;
  out.converged = done && finite;
  out.finite = finite;
  out.gap = empty ? 0.0 : gap * rcp3(gap_scale > 1e-300 ? gap_scale : 1e-300);
  return out;
}

}  // namespace lplb
