// One shape of the batched sparse-LU time advance: double, 16 samples per CTA, two CTAs per SM.
#include "kernels_lanes_impl.cuh"

TCHEM_GB_LANE_SHAPE(f64_16x2, double, 16, 8, 2, false)
