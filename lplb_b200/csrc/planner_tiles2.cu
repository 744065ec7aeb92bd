// Tile solver, 2 warps per group.
#include "planner_shapes_impl.cuh"

LPLB_INSTANTIATE(-2, 1)
LPLB_INSTANTIATE(-2, 2)
LPLB_INSTANTIATE(-2, 3)
LPLB_INSTANTIATE(-2, 4)
