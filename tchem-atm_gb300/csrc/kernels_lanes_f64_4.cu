// One shape of the batched sparse-LU time advance: double, 4 samples per CTA.
#include "kernels_lanes_impl.cuh"

TCHEM_GB_LANE_SHAPE(f64_4, double, 4, 16, 1, false)
