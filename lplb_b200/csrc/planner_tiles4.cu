// Tile solver, 4 warps per group.
#include "planner_shapes_impl.cuh"

LPLB_INSTANTIATE(-4, 1)
LPLB_INSTANTIATE(-4, 2)
LPLB_INSTANTIATE(-4, 3)
LPLB_INSTANTIATE(-4, 4)
