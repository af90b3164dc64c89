// One shape of the batched sparse-LU time advance: the gas-aerosol problem, 2 samples per CTA.
#include "kernels_lanes_impl.cuh"

TCHEM_GB_LANE_SHAPE(aero_2, double, 2, 16, 1, true)
