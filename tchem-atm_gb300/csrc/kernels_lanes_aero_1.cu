// One shape of the batched sparse-LU time advance: the gas-aerosol problem, 1 sample per CTA.
#include "kernels_lanes_impl.cuh"

TCHEM_GB_LANE_SHAPE(aero_1, double, 1, 8, 1, true)
