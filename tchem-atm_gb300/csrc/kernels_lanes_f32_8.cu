// One shape of the batched sparse-LU time advance: float, 8 samples per CTA.
#include "kernels_lanes_impl.cuh"

TCHEM_GB_LANE_SHAPE(f32_8, float, 8, 16, 1, false)
