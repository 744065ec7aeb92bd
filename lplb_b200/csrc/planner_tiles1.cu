// Tile solver, one warp per group.
#include "planner_shapes_impl.cuh"

LPLB_INSTANTIATE(-1, 1)
LPLB_INSTANTIATE(-1, 2)
LPLB_INSTANTIATE(-1, 3)
LPLB_INSTANTIATE(-1, 4)
