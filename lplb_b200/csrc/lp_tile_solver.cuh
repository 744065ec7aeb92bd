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
//   * Warp I holds tile row I and is the ranks 8 I .. 8 I + 7, four lanes each with the same
//     values.  With one warp nothing goes through shared memory and there is no barrier.
//   * Sums over ranks are two matrix instructions by a matrix of ones for two sums at a time
//     (65 cycles; three rounds of shuffles take 96 for one).
//   * Maxima are taken on integers that order like the doubles they stand for.
//   * Whatever does not depend on the centring parameter is done before it is known: the
//     corrector's step is linear in it.
//
// Solve kernel, two replicas per rank, unrelated instances, us a call back to back (the warp solver
// for 8 ranks, the thread-block solver above -> this one): 8 ranks 22.6 -> 11.3, 64 groups of 8 ranks
// 26.2 -> 13.1, 16 ranks 40.6 -> 16.9, 32 ranks 64.4 -> 27.4, 64 ranks 147 -> 63.  An iteration: 8 ranks 3.5 -> 1.5,
// 64 ranks 22.5 -> 9.4 us.
#pragma once

#include "lp_solver.cuh"

namespace lplb {

constexpr int kTileMaxGroup = 64;  // one warp per tile row, eight warps
constexpr int kTileMaxDup = 4;     // beyond, the per-rank state no longer fits the registers

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

// The hardware's approximation of 1/x, relative error about 2^-23.
__device__ __forceinline__ double rcp_seed(double x) {
#ifdef LPLB_HOST_SIM
  return 1.0 / x;
#else
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  return r;
#endif
}
// 1/x to a few ulp: one third-order step on the approximation, r (1 + e + e^2) with e = 1 - x r.
// Three dependent operations where two Newton steps take four.
__device__ __forceinline__ double rcp3(double x) {
  const double r = rcp_seed(x), e = fma(-x, r, 1.0);
  return fma(r, fma(e, e, e), r);
}

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
// bits behind the binary point, the rest cut off (the float ratios of the other solvers carry 23);
// anything below 1/2, negative numbers too, becomes 0.  Three integer instructions.
__device__ __forceinline__ unsigned step_key(double x) {
  const unsigned hi = (unsigned)max(hi_word(x), 0x3FE00000) - 0x3FE00000u;
  return (hi << 6) | ((unsigned)lo_word(x) >> 26);
}
// min(limit / (the number behind `key`), 1)
__device__ __forceinline__ double step_from_key(unsigned key, double limit) {
  const double x = from_words((int)((key >> 6) + 0x3FE00000u), (int)(key << 26));
  const double r = rcp_seed(x), a = limit * fma(r, fma(-x, r, 1.0), r);
  return hi_word(a) >= 0x3FF00000 ? 1.0 : a;
}
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
__device__ __forceinline__ void sweep_tile(double& n0, double& n1, int lane) {
  const int r = lane >> 2, c = lane & 3;
  const bool odd = c & 1, used = c < 2;
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    const double u0 = lane_get(n0, (lane & 28) | h), u1 = lane_get(n1, (lane & 28) | h);
    const double a = lane_get(n0, 9 * h), b = lane_get(n1, 9 * h), d = lane_get(n1, 9 * h + 4);
    const double det = fma(a, d, -(b * b));
    const double inv = rcp3(det);
    const bool ok = (unsigned)(hi_word(det) - 0x01000000) < 0x7E000000u;  // a positive, finite number
    const bool pivot = (r >> 1) == h, own = (r & 1) == (c & 1);
    const double mine = odd ? u1 : u0, other = odd ? u0 : u1, p = odd ? a : d;
    double num = fma(other, b, -(mine * p));
    if (pivot) num = own ? p : -b;
    double bop = pivot ? (own ? -1.0 : 0.0) : mine;
    num = used ? num : 0.0;
    bop = used ? bop : 0.0;
    const bool fresh = pivot || c == h;
    mma8(n0, n1, num * (ok ? inv : 0.0), bop, fresh ? 0.0 : n0, fresh ? 0.0 : n1);
  }
}

// ---- exchange between ranks -----------------------------------------------------------------
// With one warp a value of another rank is a shuffle away; otherwise it is published in a
// shared-memory vector, one vector per use so that one barrier per use suffices.
enum TileVec : int {  // after the D-fold vectors
  kVecY, kVecComp, kVecDual, kVecLoad, kVecG, kVecG1, kVecX, kVecX1, kVecBorder, kVecCp, kVecCpd, kVecG0, kVecX0, kVecMisc, kVecCount
};
constexpr int kTileFold = 5;  // D-fold vectors: w f, theta w^2, and the products of the three right-hand sides

struct TileLayout {
  int rows_mat, u, pi, vec, keys, total;  // in doubles
};
__host__ __device__ constexpr TileLayout tile_layout(int nb, int d) {
  TileLayout l{};
  if (nb == 1) return l;
  const int n = 8 * nb;
  int o = 0;
  l.rows_mat = o, o += nb * nb * 64;  // normal matrix, tile by tile (16-byte aligned)
  l.u = o, o += 2 * nb * 64;          // pivot columns, two alternating copies
  l.pi = o, o += 2 * 64;              // minus the inverse of the pivot tile, likewise
  l.vec = o, o += (kTileFold * d + kVecCount) * n;
  l.keys = o, o += 2 * nb;         // unsigned: four keys per warp
  l.total = o;
  return l;
}
__host__ __device__ inline size_t tile_solver_smem_bytes(int g, int d) {
  return sizeof(double) * (size_t)tile_layout(tile_rows(g), d).total;
}

template <int NB, int D>
struct TileTeam {
  int warp, lane, r, c, rank;
  double* sm;
  static constexpr int kRanks = 8 * NB;
  __device__ __forceinline__ TileTeam(int warp_, int lane_, double* sm_)
      : warp(warp_), lane(lane_), r(lane_ >> 2), c(lane_ & 3), rank(8 * warp_ + (lane_ >> 2)), sm(sm_) {}
  __device__ __forceinline__ double* vec(int v) const { return sm + tile_layout(NB, D).vec + (kTileFold * D + v) * kRanks; }
  __device__ __forceinline__ double* fold(int v, int d) const { return sm + tile_layout(NB, D).vec + (v * D + d) * kRanks; }
  __device__ __forceinline__ unsigned* keys() const { return reinterpret_cast<unsigned*>(sm + tile_layout(NB, D).keys); }
  __device__ __forceinline__ double2* mat() const { return reinterpret_cast<double2*>(sm + tile_layout(NB, D).rows_mat) + warp * NB * 32; }
  __device__ __forceinline__ double2* pivot_col(int parity) const { return reinterpret_cast<double2*>(sm + tile_layout(NB, D).u) + parity * NB * 32; }
  __device__ __forceinline__ double2* pivot_inv(int parity) const { return reinterpret_cast<double2*>(sm + tile_layout(NB, D).pi) + parity * 32; }

  __device__ __forceinline__ void sync() const {
    if constexpr (NB > 1) {
#ifdef LPLB_HOST_SIM
      lplb_sim_named_barrier(NB * 32);
#else
      asm volatile("bar.sync 1, %0;" ::"n"(NB * 32) : "memory");
#endif
    }
  }
  __device__ __forceinline__ void put(double* where, double v) const {
    if constexpr (NB > 1) {
      if (c == 0) where[rank] = v;
    }
  }
  __device__ __forceinline__ double get(const double* where, double mine, int of) const {
    if constexpr (NB > 1) return where[of];
    else return lane_get(mine, 4 * of);
  }
  // Sums over the ranks of two values; (va, vb) hold them where they have been published.
  __device__ __forceinline__ void sum2(const double* va, double a, const double* vb, double b, double& sa, double& sb) const {
    double d0, d1;
    if constexpr (NB == 1) {
      // lanes of one rank hold the same values: every other one passes b
      mma8(d0, d1, c == (r & 1) ? 1.0 : 0.0, (c & 1) ? b : a, 0.0, 0.0);  // even rows: all ranks' a, odd rows: their b
      mma8(sa, sb, 1.0, d0 + d1, 0.0, 0.0);
    } else {
      const double* v = (r & 1) ? vb : va;
      const int first = (r >> 1) * 4 + c;
      double acc = v[first];
#pragma unroll
      for (int k = 16; k < kRanks; k += 16) acc += v[first + k];
      mma8(d0, d1, 1.0, acc, 0.0, 0.0);
      mma8(sa, sb, 1.0, (r & 1) ? d1 : d0, 0.0, 0.0);
    }
  }
  __device__ __forceinline__ double max_positive(const double* where, double x) const {
    if constexpr (NB > 1) {
      x = where[lane % kRanks];
      if constexpr (kRanks > 32) {
        const double other = where[lane + 32];
        // positive doubles order like their bit patterns, negative ones lie below
        const bool more = hi_word(other) > hi_word(x) ||
                          (hi_word(other) == hi_word(x) && (unsigned)lo_word(other) > (unsigned)lo_word(x));
        x = more ? other : x;
      }
    }
    return warp_max_positive(x);
  }
  // Largest key over the ranks, in two halves around a barrier.
  __device__ __forceinline__ unsigned key_put(int slot, unsigned key) const {
    key = __reduce_max_sync(0xffffffffu, key);
    if constexpr (NB > 1) {
      if (lane == 0) keys()[slot * NB + warp] = key;
    }
    return key;
  }
  __device__ __forceinline__ unsigned key_get(int slot, unsigned key) const {
    if constexpr (NB > 1) key = __reduce_max_sync(0xffffffffu, keys()[slot * NB + lane % NB]);
    return key;
  }
  __device__ __forceinline__ bool all(int slot, bool ok) const {  // several warps: key_put(slot, !ok) and a barrier before
    if constexpr (NB == 1) return __all_sync(0xffffffffu, ok);
    else return key_get(slot, 0) == 0;
  }
};

// The inverse of the normal matrix, one tile row per warp: on entry n[j] is tile (I, j) of the
// matrix, on return minus the inverse's tile.  Block sweeps over the tiles of the diagonal: with P the
// pivot tile's inverse and U_I the tiles of its column, tile (I, J) becomes N_IJ - U_I P U_J^T, the
// pivot's column U_I P, its row P U_J^T and the pivot itself -P.  The tiles of a row are kept rotated, so
// that the pivot's column is always the first and the loop over pivots stays rolled.
template <int NB, int D>
__device__ __forceinline__ void sweep_matrix(const TileTeam<NB, D>& tm, double (&n0)[NB], double (&n1)[NB]) {
  if constexpr (NB == 1) {
    sweep_tile(n0[0], n1[0], tm.lane);
  } else {
    if (tm.warp == 0) {
      double p0 = n0[0], p1 = n1[0];
      sweep_tile(p0, p1, tm.lane);
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
      if (tm.warp == p + 1) {  // the next pivot tile is ready: invert it beside the other updates
        double p0 = n0[0], p1 = n1[0];
        sweep_tile(p0, p1, tm.lane);
#pragma unroll
        for (int j = 2; j < NB; ++j) update(j);
        tm.pivot_inv((p + 1) & 1)[tm.lane] = double2{p0, p1};
      } else {
#pragma unroll
        for (int j = 2; j < NB; ++j) update(j);
      }
      n0[NB - 1] = f0;
      n1[NB - 1] = f1;
    }
  }
}

// One group of at most 8 NB ranks, solved by NB warps (all of them call; `warp` counts from 0 within the
// group).  Lane 4 r + c of warp I is rank 8 I + r and passes that rank's data, as in ipm_solve_segment;
// ranks from `rows` on do not take part (w = 0, fixed = 0, src = dst = the rank itself, no anchor).
// `sm`: tile_solver_smem_bytes of shared memory, 16-byte aligned (one warp: unused).  `anchor`:
// the rank's slot of the warm-start state or null; `group_anchor` the slot of the group's first rank.
// The outcome is the same on every lane.
template <int NB, int D>
__device__ __forceinline__ IpmOutcome ipm_solve_tiles(const int warp, const int lane, const int rows,
                                                      const double (&w_in)[D], const double fixed,
                                                      const int (&src_in)[D], const int (&dst_in)[D],
                                                      const IpmParams prm, double (&f_out)[D], double* anchor,
                                                      const double* group_anchor, int* anchor_valid, double* sm) {
  constexpr double kEta = 0.995;
  const TileTeam<NB, D> tm(warp, lane, sm);
  const int c = tm.c, rank = tm.rank;
  const bool live = rank < rows;
  int src[D], dst[D];
#pragma unroll
  for (int d = 0; d < D; ++d) {
    src[d] = src_in[d];
    dst[d] = dst_in[d];
  }
  // The saved iterate is read first, valid or not (the slot is always allocated): its loads are
  // in flight while the scaling is computed.
  double fa[D], va[D], za[D], qa[D], sa = 1.0, ya = 0.0, ta = 0.0;
  const bool slot = anchor != nullptr && live;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    fa[d] = slot ? anchor[d] : 0.5;
    va[d] = slot ? anchor[D + d] : 0.5;
    za[d] = slot ? anchor[2 * D + d] : 1.0;
    qa[d] = slot ? anchor[3 * D + d] : 1.0;
  }
  if (slot) {
    sa = anchor[4 * D];
    ya = anchor[4 * D + 1];
  }
  if (group_anchor != nullptr) ta = group_anchor[4 * D + 2];
  const bool saved_before = group_anchor != nullptr && *anchor_valid != 0;

  const double kcomp = (double)(rows + 2 * rows * D), inv_kcomp = rcp3(kcomp), inv_rows = rcp3((double)rows);

  // ---- where this lane's off-diagonal terms of the matrix go -----------------------------------
  // One warp: factors 0 or -1 for the lane's two columns.  Several: places in the tile row, written
  // once per iteration; terms that share a column are merged (the first collects the later ones).
  double cd[NB == 1 ? D : 1][2], cs[NB == 1 ? D : 1][2];
  double* place[NB > 1 ? 2 * D : 1];
  unsigned merge = 0;  // bit a * 2 D + b: term b > a goes to term a's place
  double* diag_place = nullptr;
  if constexpr (NB == 1) {
#pragma unroll
    for (int d = 0; d < D; ++d)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        cd[d][e] = dst[d] == 2 * c + e ? -1.0 : 0.0;
        cs[d][e] = src[d] == 2 * c + e ? -1.0 : 0.0;
      }
  } else {
    static_assert(kTileMaxDup <= 4, "the pairs of terms share one word: (2 D)^2 bits with a < b");
    double2* mat = tm.mat();
    for (int j = 0; j < NB; ++j) mat[j * 32 + lane] = double2{0.0, 0.0};
    auto at = [&](int col) { return reinterpret_cast<double*>(mat) + ((col >> 3) * 32 + 4 * tm.r + ((col & 7) >> 1)) * 2 + (col & 1); };
    int col[2 * D];
#pragma unroll
    for (int d = 0; d < D; ++d) {
      col[2 * d] = dst[d];
      col[2 * d + 1] = src[d];
    }
    int bit = 0;
#pragma unroll
    for (int a = 0; a < 2 * D; ++a) {
      bool first = col[a] != rank && live && c == 0;
#pragma unroll
      for (int b = 0; b < a; ++b)
        if (col[b] == col[a]) first = false;
#pragma unroll
      for (int b = a + 1; b < 2 * D; ++b, ++bit)
        if (col[b] == col[a]) merge |= 1u << bit;
      place[a] = first ? at(col[a]) : nullptr;
    }
    if (c == 0) diag_place = at(rank);
    __syncwarp();
  }

  // ---- scale so that the mean rank load is 1 ---------------------------------------
  double mine = fixed;
#pragma unroll
  for (int d = 0; d < D; ++d) mine += w_in[d];
  if (!live) mine = 0.0;
#pragma unroll
  for (int d = 0; d < D; ++d) tm.put(tm.fold(0, d), w_in[d]);
  tm.put(tm.vec(kVecMisc), mine);
  tm.sync();
  double total, unused;
  tm.sum2(tm.vec(kVecMisc), mine, tm.vec(kVecMisc), mine, total, unused);
  const bool empty = !(total > 0.0);
  const double inv_scale = empty ? 0.0 : (double)rows * rcp3(total);
  double w[D], base = fixed;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    base += tm.get(tm.fold(0, d), w_in[d], src[d]);
    // a self edge moves no load: its column of M is zero, its load is already part of `base`
    w[d] = dst[d] == rank ? 0.0 : w_in[d] * inv_scale;
  }
  base *= inv_scale;

  // ---- warm start from the anchor, if it still fits the data -----------------------------
  bool cold;
  {
    double mfa = 0.0;
#pragma unroll
    for (int d = 0; d < D; ++d) tm.put(tm.fold(1, d), w[d] * fa[d]);
    tm.sync();
#pragma unroll
    for (int d = 0; d < D; ++d) mfa += w[d] * fa[d] - tm.get(tm.fold(1, d), w[d] * fa[d], src[d]);
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
  double f[D], v[D], z[D], q[D], t = ta, s = 1.0, y = live ? inv_rows : 0.0;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    f[d] = start_cold ? 0.5 : fa[d];
    v[d] = start_cold ? 0.5 : va[d];
    z[d] = start_cold ? 1.0 : za[d];
    q[d] = start_cold ? 1.0 : qa[d];
  }
  if (!start_cold) {
    s = sa;
    y = ya;
  }
  if (NB == 1 ? __any_sync(0xffffffffu, live && start_cold) : cold) {  // feasible start
    double load = base;
#pragma unroll
    for (int d = 0; d < D; ++d) tm.put(tm.fold(2, d), 0.5 * w[d]);
    tm.sync();
#pragma unroll
    for (int d = 0; d < D; ++d) load += 0.5 * w[d] - tm.get(tm.fold(2, d), 0.5 * w[d], src[d]);
    tm.put(tm.vec(kVecLoad), live ? load : -1.0);
    tm.sync();
    const double lmax = tm.max_positive(tm.vec(kVecLoad), live ? load : -1.0);
    const double down = live ? (lmax + 1.0) - load : -1.0;
    tm.put(tm.vec(kVecDual), down);
    tm.sync();
    const double lmin = (lmax + 1.0) - tm.max_positive(tm.vec(kVecDual), down);
    const double ct = lmax + 0.5 * (lmax - lmin) + 0.05;
    if (live && start_cold) s = ct - load;
    if (cold) t = ct;
    const double sy = live ? (ct - load) * inv_rows : 0.0;
    tm.put(tm.vec(kVecComp), sy);
    tm.sync();
    double sum, same;
    tm.sum2(tm.vec(kVecComp), sy, tm.vec(kVecComp), sy, sum, same);
    const double mu0 = sum * inv_rows;
    if (start_cold) {
#pragma unroll
      for (int d = 0; d < D; ++d) z[d] = q[d] = 2.0 * mu0;
    }
    tm.sync();  // the vectors are used again below
  }
  bool saved = false, done = empty;
  int iters = 0;
  double gap = 1e300, gap_scale = 1.0;

#pragma unroll 1
  for (int it = 0;; ++it) {
    if (prm.stop != nullptr && __any_sync(0xffffffffu, *prm.stop != 0)) break;
    // ---- weights, residuals, gap, stopping test ----------------------------------------------
    double wf[D], cw[D], theta[D], inv_f[D], inv_v[D];
    const double inv_y = rcp3(live ? y : 1.0);
#pragma unroll
    for (int d = 0; d < D; ++d) {
      wf[d] = w[d] * f[d];
      const double fv = f[d] * v[d], inv_fv = rcp3(fv);
      theta[d] = fv * rcp3(fma(z[d], v[d], q[d] * f[d]));  // 1 / (z / f + q / v)
      cw[d] = theta[d] * (w[d] * w[d]);
      inv_f[d] = v[d] * inv_fv;
      inv_v[d] = f[d] * inv_fv;
      tm.put(tm.fold(0, d), wf[d]);
      tm.put(tm.fold(1, d), cw[d]);
    }
    tm.put(tm.vec(kVecY), y);
    tm.sync();
    double load = base, diag = s * inv_y, held[D], wy[D], r_u[D];
    double comp = s * y, dual = y * base;
    bool feasible = true;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      load += wf[d] - tm.get(tm.fold(0, d), wf[d], src[d]);
      held[d] = tm.get(tm.fold(1, d), cw[d], src[d]);
      wy[d] = w[d] * (y - tm.get(tm.vec(kVecY), y, dst[d]));
      diag += cw[d] + held[d];
      r_u[d] = 1.0 - f[d] - v[d];
      comp = fma(z[d], f[d], fma(q[d], v[d], comp));
      dual += negative_part(z[d] - q[d] - wy[d]) - q[d];
      feasible = feasible && fabs(r_u[d]) <= prm.tol;
    }
    if (!live) comp = dual = 0.0;
    tm.put(tm.vec(kVecComp), comp);
    tm.put(tm.vec(kVecDual), dual);
    tm.put(tm.vec(kVecLoad), live ? load : -1.0);
    // right-hand sides: the predictor's, and the part of the corrector's that goes with sigma mu
    double qv[D], rd[D], wt[D], x_rhs[D], x_one[D];
#pragma unroll
    for (int d = 0; d < D; ++d) {
      qv[d] = q[d] * inv_v[d];
      rd[d] = fma(qv[d], r_u[d], -wy[d]);
      wt[d] = w[d] * theta[d];
      x_rhs[d] = wt[d] * rd[d];
      x_one[d] = wt[d] * (inv_f[d] - inv_v[d]);
      tm.put(tm.fold(2, d), x_rhs[d]);
      tm.put(tm.fold(3, d), x_one[d]);
    }
    if constexpr (NB > 1) tm.key_put(0, live && !feasible ? 1u : 0u);
    tm.sync();
    double mu, sum_y, dual_sum, same;
    tm.sum2(tm.vec(kVecComp), comp, tm.vec(kVecY), y, mu, sum_y);
    tm.sum2(tm.vec(kVecDual), dual, tm.vec(kVecDual), dual, dual_sum, same);
    mu *= inv_kcomp;
    const double r_t = 1.0 - sum_y;
    const double primal = tm.max_positive(tm.vec(kVecLoad), live ? load : -1.0);
    const bool all_feasible = tm.all(0, !live || feasible);
    if (!done) {
      gap = primal - dual_sum;  // absolute here, made relative once at the end
      gap_scale = fabs(primal);
      // at mu ~ 1e-13 the iterate is optimal to machine precision: stop instead of dividing by it
      if ((gap <= prm.tol * gap_scale && all_feasible && fabs(r_t) <= prm.tol) || mu <= 1e-13) done = true;
    }
    // A cold solve leaves its first iterate at or below snap_mu behind as the next anchor.
    if (cold && !saved && !empty && mu <= prm.snap_mu) {
      if (slot && c == 0) {
#pragma unroll
        for (int d = 0; d < D; ++d) {
          anchor[d] = f[d];
          anchor[D + d] = v[d];
          anchor[2 * D + d] = z[d];
          anchor[3 * D + d] = q[d];
        }
        anchor[4 * D] = s;
        anchor[4 * D + 1] = y;
        anchor[4 * D + 2] = t;
        if (rank == 0) *anchor_valid = 1;
      }
      saved = true;
    }
    if (done || it >= prm.max_iters) break;
    ++iters;

    // ---- normal matrix and its inverse ---------------------------------------------------------
    double n0[NB], n1[NB];
    if (!live) diag = 1.0;
    if constexpr (NB == 1) {
      double e0 = rank == 2 * c ? diag : 0.0, e1 = rank == 2 * c + 1 ? diag : 0.0;
      double h0 = 0.0, h1 = 0.0;
#pragma unroll
      for (int d = 0; d < D; ++d) {
        e0 = fma(cd[d][0], cw[d], e0);
        e1 = fma(cd[d][1], cw[d], e1);
        h0 = fma(cs[d][0], held[d], h0);
        h1 = fma(cs[d][1], held[d], h1);
      }
      n0[0] = e0 + h0;
      n1[0] = e1 + h1;
    } else {
      double val[2 * D];
#pragma unroll
      for (int d = 0; d < D; ++d) {
        val[2 * d] = cw[d];
        val[2 * d + 1] = held[d];
      }
      int bit = 0;
#pragma unroll
      for (int a = 0; a < 2 * D; ++a) {
        double acc = val[a];
#pragma unroll
        for (int b = a + 1; b < 2 * D; ++b, ++bit)
          if ((merge >> bit) & 1u) acc += val[b];
        if (place[a] != nullptr) *place[a] = -acc;
      }
      if (diag_place != nullptr) *diag_place = diag;
      __syncwarp();
      const double2* mat = tm.mat();
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        const double2 e = mat[j * 32 + lane];
        n0[j] = e.x;
        n1[j] = e.y;
      }
    }
    double g = load - t, g_one = inv_y;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      g += x_rhs[d] - tm.get(tm.fold(2, d), x_rhs[d], src[d]);
      g_one += x_one[d] - tm.get(tm.fold(3, d), x_one[d], src[d]);
    }
    if (!live) g = g_one = 0.0;
    tm.put(tm.vec(kVecG), g);
    tm.put(tm.vec(kVecG1), g_one);
    sweep_matrix<NB, D>(tm, n0, n1);  // with several warps its barriers also publish the right-hand sides

    // inverse times (g, g_one), and times a vector of ones: the border column that carries sum(dy) = r_t
    double x, x1, border;
    {
      double rs = 0.0, same_b;
#pragma unroll
      for (int j = 0; j < NB; ++j) rs += n0[j] + n1[j];
      mma8(border, same_b, rs, -1.0, 0.0, 0.0);
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
        double p0 = 0.0, p1 = 0.0, o0 = 0.0, o1 = 0.0, unused_x;
#pragma unroll
        for (int j = 0; j < NB; ++j) {
          const double2 a = gv[4 * j + c], b = ov[4 * j + c];
          p0 = fma(n0[j], a.x, p0);
          p1 = fma(n1[j], a.y, p1);
          o0 = fma(n0[j], b.x, o0);
          o1 = fma(n1[j], b.y, o1);
        }
        mma8(x, unused_x, p0 + p1, -1.0, 0.0, 0.0);
        mma8(x1, unused_x, o0 + o1, -1.0, 0.0, 0.0);
      }
    }
    if (!live) border = 0.0;
    tm.put(tm.vec(kVecX), x);
    tm.put(tm.vec(kVecX1), x1);
    tm.put(tm.vec(kVecBorder), border);
    tm.sync();
    double sum_x, sum_b, sum_x1;
    tm.sum2(tm.vec(kVecX), x, tm.vec(kVecBorder), border, sum_x, sum_b);
    tm.sum2(tm.vec(kVecX1), x1, tm.vec(kVecX1), x1, sum_x1, same);
    const double inv_sum_b = rcp3(sum_b);
    const double inv_mu = rcp3(kcomp * mu);
    // ---- predictor ---------------------------------------------------------------------------
    // df = theta (rd - w (dy - dy_dst)) with dy = x - dt border, as e + dt e_b
    double e[D], e_b[D], e_1[D];
#pragma unroll
    for (int d = 0; d < D; ++d) {
      e[d] = fma(-wt[d], x - tm.get(tm.vec(kVecX), x, dst[d]), theta[d] * rd[d]);
      e_b[d] = wt[d] * (border - tm.get(tm.vec(kVecBorder), border, dst[d]));
      e_1[d] = fma(-wt[d], x1 - tm.get(tm.vec(kVecX1), x1, dst[d]), theta[d] * (inv_f[d] - inv_v[d]));
    }
    double dt = (sum_x - r_t) * inv_sum_b;
    double dy = fma(-dt, border, x);
    const double si = s * inv_y;
    double ds = fma(-si, dy, -s);
    double df[D], dv[D], dz[D], dq[D], zi[D], p_f[D], p_v[D], x_cor[D], rc[D];
    // the predictor takes every complementarity product to zero, so dz / z = -1 - df / f, and so on
    const double ty = -dy * inv_y;
    unsigned key_p = step_key(1.0 - ty), key_d = step_key(ty);
    double c_p = y * ds, c_pd = ds * dy;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      zi[d] = z[d] * inv_f[d];
      df[d] = fma(dt, e_b[d], e[d]);
      dv[d] = r_u[d] - df[d];
      dz[d] = fma(-zi[d], df[d], -z[d]);
      dq[d] = fma(-qv[d], dv[d], -q[d]);
      const double tf = -df[d] * inv_f[d], tv = -dv[d] * inv_v[d];
      key_p = max(key_p, max(step_key(tf), step_key(tv)));
      key_d = max(key_d, max(step_key(1.0 - tf), step_key(1.0 - tv)));
      c_p = fma(z[d], df[d], fma(q[d], dv[d], c_p));
      c_pd = fma(df[d], dz[d], fma(dv[d], dq[d], c_pd));
      p_f[d] = dz[d] * -tf;  // dz df / f
      p_v[d] = dq[d] * -tv;
      rc[d] = rd[d] - p_f[d] + p_v[d];
      x_cor[d] = wt[d] * rc[d];
      tm.put(tm.fold(4, d), x_cor[d]);
    }
    if (!live) {
      c_p = c_pd = 0.0;
      key_p = key_d = 0;
    }
    const double p_s = ds * -ty;  // ds dy / y
    key_p = tm.key_put(0, key_p);
    key_d = tm.key_put(1, key_d);
    tm.put(tm.vec(kVecCp), c_p);
    tm.put(tm.vec(kVecCpd), c_pd);
    tm.sync();
    // ---- corrector ---------------------------------------------------------------------------
    double g0 = load - t - p_s;
#pragma unroll
    for (int d = 0; d < D; ++d) g0 += x_cor[d] - tm.get(tm.fold(4, d), x_cor[d], src[d]);
    if (!live) g0 = 0.0;
    tm.put(tm.vec(kVecG0), g0);
    double sum_cp, sum_cpd;
    tm.sum2(tm.vec(kVecCp), c_p, tm.vec(kVecCpd), c_pd, sum_cp, sum_cpd);
    const double ap0 = step_from_key(tm.key_get(0, key_p), 1.0), ad0 = step_from_key(tm.key_get(1, key_d), 1.0);
    // complementarity after the affine step; sum x dz = -kcomp mu - sum z dx
    const double comp_aff = fma(ap0 * ad0, sum_cpd, fma(ap0 - ad0, sum_cp, kcomp * mu * (1.0 - ad0)));
    const double ratio = clamp01(comp_aff * inv_mu);
    const double sig_mu = ratio * ratio * ratio * mu;
    double x0;
    if constexpr (NB == 1) {
      const double b0 = lane_get(g0, 8 * c), b1 = lane_get(g0, 8 * c + 4);
      mma8(x0, same, -n0[0], b0, 0.0, 0.0);
      mma8(x0, same, -n1[0], b1, x0, same);
    } else {
      tm.sync();
      const double2* gv = reinterpret_cast<const double2*>(tm.vec(kVecG0));
      double p0 = 0.0, p1 = 0.0;
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        const double2 a = gv[4 * j + c];
        p0 = fma(n0[j], a.x, p0);
        p1 = fma(n1[j], a.y, p1);
      }
      mma8(x0, same, p0 + p1, -1.0, 0.0, 0.0);
      tm.put(tm.vec(kVecX0), x0);
      tm.sync();
    }
    double sum_x0;
    tm.sum2(tm.vec(kVecX0), x0, tm.vec(kVecX0), x0, sum_x0, same);
    dt = (fma(sig_mu, sum_x1, sum_x0) - r_t) * inv_sum_b;
    dy = fma(-dt, border, fma(sig_mu, x1, x0));
    ds = fma(-si, dy, fma(sig_mu, inv_y, -s - p_s));
    key_p = step_key(-ds * rcp_seed(s));
    key_d = step_key(-dy * inv_y);
#pragma unroll
    for (int d = 0; d < D; ++d) {
      const double e0 = fma(-wt[d], x0 - tm.get(tm.vec(kVecX0), x0, dst[d]), theta[d] * rc[d]);
      df[d] = fma(dt, e_b[d], fma(sig_mu, e_1[d], e0));
      dv[d] = r_u[d] - df[d];
      dz[d] = fma(-zi[d], df[d], fma(sig_mu, inv_f[d], -z[d] - p_f[d]));
      dq[d] = fma(-qv[d], dv[d], fma(sig_mu, inv_v[d], -q[d] - p_v[d]));
      key_p = max(key_p, max(step_key(-df[d] * inv_f[d]), step_key(-dv[d] * inv_v[d])));
      key_d = max(key_d, max(step_key(-dz[d] * rcp_seed(z[d])), step_key(-dq[d] * rcp_seed(q[d]))));
    }
    if (!live) key_p = key_d = 0;
    key_p = tm.key_put(2, key_p);
    key_d = tm.key_put(3, key_d);
    tm.sync();
    const double ap = step_from_key(tm.key_get(2, key_p), kEta), ad = step_from_key(tm.key_get(3, key_d), kEta);
    t = fma(ap, dt, t);
    if (live) {
      s = fma(ap, ds, s);
      y = fma(ad, dy, y);
#pragma unroll
      for (int d = 0; d < D; ++d) {
        f[d] = fma(ap, df[d], f[d]);
        v[d] = fma(ap, dv[d], v[d]);
        z[d] = fma(ad, dz[d], z[d]);
        q[d] = fma(ad, dq[d], q[d]);
      }
    }
  }

  bool ok = true;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    ok = ok && (f[d] == f[d]) && fabs(f[d]) < 1e300;
    f_out[d] = fmin(fmax(f[d], 0.0), 1.0);
  }
  if constexpr (NB > 1) {
    tm.sync();  // every warp is through with key 0
    tm.key_put(0, live && !ok ? 1u : 0u);
    tm.sync();
  }
  const bool finite = tm.all(0, !live || ok);
  if (!finite) {
#pragma unroll
    for (int d = 0; d < D; ++d) f_out[d] = 0.5;
  }
  if (empty) {  // nothing to balance: keep everything on the origin
#pragma unroll
    for (int d = 0; d < D; ++d) f_out[d] = 1.0;
  }
  IpmOutcome out;
  out.iters = iters;
  out.converged = done && finite;
  out.finite = finite;
  out.gap = empty ? 0.0 : gap * rcp3(gap_scale > 1e-300 ? gap_scale : 1e-300);
  return out;
}

}  // namespace lplb
