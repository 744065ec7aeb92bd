// Tile solver, 8 warps per group.
#include "planner_shapes_impl.cuh"

LPLB_INSTANTIATE(-8, 1)
LPLB_INSTANTIATE(-8, 2)
LPLB_INSTANTIATE(-8, 3)
LPLB_INSTANTIATE(-8, 4)
