// One shape of the batched sparse-LU time advance: double, 8 samples per CTA.
#include "kernels_lanes_impl.cuh"

TCHEM_GB_LANE_SHAPE(f64_8, double, 8, 16, 1, false)
