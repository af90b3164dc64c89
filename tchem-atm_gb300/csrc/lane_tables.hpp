// Device copies of the batched sparse-LU kernel's instruction streams, one per kernel shape.
#pragma once

#include "device_tables.hpp"
#include "kernels_lanes.hpp"

namespace tchem_gb {

struct LaneTables {
  int device = -1;
  void* allocation = nullptr;
  bool valid[2][kLaneShapeCount] = {};  // [FP32, FP64]
  LaneDev dev[2][kLaneShapeCount] = {};
};

// Null where the mechanism has no program of any shape (too large, or more than three factors).
LaneTables* upload_lane_tables(const HostTables& ht, int device, int max_smem);
void destroy_lane_tables(LaneTables* t);

}  // namespace tchem_gb
