// One shape of the batched sparse-LU time advance: float, 16 samples per CTA, two CTAs per SM.
#include "kernels_lanes_impl.cuh"

TCHEM_GB_LANE_SHAPE(f32_16x2, float, 16, 8, 2, false)
