// One shape of the batched sparse-LU time advance: float, 2 samples per CTA.
#include "kernels_lanes_impl.cuh"

TCHEM_GB_LANE_SHAPE(f32_2, float, 2, 16, 1, false)
