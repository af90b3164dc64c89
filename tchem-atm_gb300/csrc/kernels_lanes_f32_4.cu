// One shape of the batched sparse-LU time advance: float, 4 samples per CTA.
#include "kernels_lanes_impl.cuh"

TCHEM_GB_LANE_SHAPE(f32_4, float, 4, 16, 1, false)
