// Batched time advance over a static-order sparse LU: shapes and launch.
#include "kernels_lanes.hpp"

namespace tchem_gb {

#define TCHEM_GB_DECLARE_LANES(NAME)                                            \
  const void* lane_kernel_##NAME();                                           \
  cudaError_t launch_lanes_##NAME(const LaneParams&, int, cudaStream_t);
TCHEM_GB_DECLARE_LANES(f32_16x2)
TCHEM_GB_DECLARE_LANES(f32_16)
TCHEM_GB_DECLARE_LANES(f32_8)
TCHEM_GB_DECLARE_LANES(f32_4)
TCHEM_GB_DECLARE_LANES(f32_2)
TCHEM_GB_DECLARE_LANES(f32_1)
TCHEM_GB_DECLARE_LANES(f64_16x2)
TCHEM_GB_DECLARE_LANES(f64_16)
TCHEM_GB_DECLARE_LANES(f64_8)
TCHEM_GB_DECLARE_LANES(f64_4)
TCHEM_GB_DECLARE_LANES(f64_2)
TCHEM_GB_DECLARE_LANES(f64_1)
TCHEM_GB_DECLARE_LANES(aero_8)
TCHEM_GB_DECLARE_LANES(aero_4)
TCHEM_GB_DECLARE_LANES(aero_2)
TCHEM_GB_DECLARE_LANES(aero_1)
#undef TCHEM_GB_DECLARE_LANES

namespace {
struct Entry {
  const void* (*kernel)();
  cudaError_t (*launch)(const LaneParams&, int, cudaStream_t);
};
const Entry kEntries[kLaneForms][kLaneShapeCount] = {
    {{lane_kernel_f32_16x2, launch_lanes_f32_16x2},
     {lane_kernel_f32_16, launch_lanes_f32_16},
     {lane_kernel_f32_8, launch_lanes_f32_8},
     {lane_kernel_f32_4, launch_lanes_f32_4},
     {lane_kernel_f32_2, launch_lanes_f32_2},
     {lane_kernel_f32_1, launch_lanes_f32_1}},
    {{lane_kernel_f64_16x2, launch_lanes_f64_16x2},
     {lane_kernel_f64_16, launch_lanes_f64_16},
     {lane_kernel_f64_8, launch_lanes_f64_8},
     {lane_kernel_f64_4, launch_lanes_f64_4},
     {lane_kernel_f64_2, launch_lanes_f64_2},
     {lane_kernel_f64_1, launch_lanes_f64_1}},
    {{nullptr, nullptr},
     {nullptr, nullptr},
     {lane_kernel_aero_8, launch_lanes_aero_8},
     {lane_kernel_aero_4, launch_lanes_aero_4},
     {lane_kernel_aero_2, launch_lanes_aero_2},
     {lane_kernel_aero_1, launch_lanes_aero_1}}};
}  // namespace

const void* lane_kernel(int shape, LaneForm form) { return kEntries[form][shape].kernel(); }

cudaError_t launch_lanes(const LaneParams& P, int shape, LaneForm form, int grid, cudaStream_t stream) {
  return kEntries[form][shape].launch(P, grid, stream);
}

}  // namespace tchem_gb
