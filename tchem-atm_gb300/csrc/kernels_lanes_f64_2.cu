// One shape of the batched sparse-LU time advance: double, 2 samples per CTA.
#include "kernels_lanes_impl.cuh"

TCHEM_GB_LANE_SHAPE(f64_2, double, 2, 16, 1, false)
