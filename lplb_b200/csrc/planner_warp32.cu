// Warp solver, groups of 32 ranks.
#include "planner_shapes_impl.cuh"

LPLB_INSTANTIATE(32, 1)
LPLB_INSTANTIATE(32, 2)
LPLB_INSTANTIATE(32, 3)
LPLB_INSTANTIATE(32, 4)
