// One shape of the batched sparse-LU time advance: double, 1 sample per CTA.
#include "kernels_lanes_impl.cuh"

TCHEM_GB_LANE_SHAPE(f64_1, double, 1, 8, 1, false)
