// Thread-block solver.
#include "planner_shapes_impl.cuh"

LPLB_INSTANTIATE(0, 1)
LPLB_INSTANTIATE(0, 2)
LPLB_INSTANTIATE(0, 3)
LPLB_INSTANTIATE(0, 4)
LPLB_INSTANTIATE(0, 8)
