// One shape of the batched sparse-LU time advance: float, 16 samples per CTA.
#include "kernels_lanes_impl.cuh"

TCHEM_GB_LANE_SHAPE(f32_16, float, 16, 16, 1, false)
