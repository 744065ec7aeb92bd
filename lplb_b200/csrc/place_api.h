// Host-side launch interface of the placement kernel.  Plain C++, no torch headers.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

namespace lplb {

enum PlaceReport : int {
  kPlacePending = -1,   // what the host sets before the launch
  kPlaceOk = 0,
  kPlaceInexact = 1,    // loads of expert groups beyond 2^53: their sums depend on the order of adding; no table was written
  kPlaceUncovered = 2,  // some expert does not sit in exactly one of the ranks' own slots; the tables are not usable
};

// r2o and o2r: each the inverse of the other, which the caller has checked.
struct PlaceArgs {
  const void* history;  // [n_logical] int32/int64 loads; null = natural order
  int is64;
  const int *r2o, *o2r;  // [g, dup]
  int n_logical, ep_size, n_group, g, dup, combined, n_nodes;
  // results, and the engine's own copies of them (which keep their addresses)
  int *phy2log, *log2phy, *logcnt, *log2edge;
  int* report;  // host memory: the outcome, written when everything else is
  int* anchor_valid;  // [n_anchor] cleared: a new placement is a new LP; may be null
  int n_anchor;
  int *table_phy2log, *table_log2phy, *table_log2edge, *table_log2slot;
};

size_t place_shared_bytes(const PlaceArgs& a);
cudaError_t launch_place(const PlaceArgs& a, cudaStream_t stream);

}  // namespace lplb
