// Device copies of the batched sparse-LU kernel's instruction streams, one per kernel shape.
#pragma once

#include "device_tables.hpp"
#include "kernels_lanes.hpp"

namespace tchem_gb {

struct LaneTables {
  int device = -1;
  void* allocation = nullptr;
  bool valid[kLaneForms][kLaneShapeCount] = {};
  LaneDev dev[kLaneForms][kLaneShapeCount] = {};
};

// The box-model (and E3SM) problem of a mechanism, FP32 and FP64; null where it has no program of any
// shape (too large, or more than three factors).
LaneTables* upload_lane_tables(const HostTables& ht, int device, int max_smem);
// The gas-aerosol problem of a mechanism and an aerosol model (sizes and SIMPOL entries of A and
// simpol_index as in tchem_gb_aero_view).
LaneTables* upload_aero_lane_tables(const HostTables& ht, const AeroDev& A, const int32_t* simpol_index, int device,
                                    int max_smem);

// A form's shape for a batch and its launch (shape < 0: none).
struct LanePlan {
  int shape = -1, grid = 0;
  LaneForm form = LANE_F32;
  LaneSmem smem{};
  LaneDev dev{};
};
LanePlan plan_lanes(const LaneTables* t, LaneForm form, int ext, int sm_count, int max_smem, int nbatch, int slack);
// Whether the batched kernel is the faster default for a box-model batch of mechanisms with m species (E3SM columns
// and aerosol cells always take it).
bool lanes_pay_for_box(LaneForm form, int m, int sm_count, int nbatch);
void destroy_lane_tables(LaneTables* t);

}  // namespace tchem_gb
