// One shape of the batched sparse-LU time advance: the gas-aerosol problem, 8 samples per CTA.
#include "kernels_lanes_impl.cuh"

TCHEM_GB_LANE_SHAPE(aero_8, double, 8, 16, 1, true)
