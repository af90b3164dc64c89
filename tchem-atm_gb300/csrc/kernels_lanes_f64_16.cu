// One shape of the batched sparse-LU time advance: double, 16 samples per CTA.
#include "kernels_lanes_impl.cuh"

TCHEM_GB_LANE_SHAPE(f64_16, double, 16, 16, 1, false)
