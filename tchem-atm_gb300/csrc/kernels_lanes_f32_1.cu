// One shape of the batched sparse-LU time advance: float, 1 sample per CTA.
#include "kernels_lanes_impl.cuh"

TCHEM_GB_LANE_SHAPE(f32_1, float, 1, 8, 1, false)
