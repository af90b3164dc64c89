// Batched time advance over a static-order sparse LU (kernels_lanes_impl.cuh): launch interface.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>

#include "advance.hpp"
#include "kernels.hpp"

namespace tchem_gb {

// One mechanism's instruction streams for one kernel shape, on the device (lane_program.hpp).
// The streams in the order of their shared-memory places: what is read most often per round first.
enum LaneStreamId { LS_NET, LS_FORWARD, LS_BACKWARD, LS_REACTIONS, LS_FACTOR, LS_MATRIX, LS_COUNT };
struct LaneDev {
  int32_t m, R, Q, D;         // LaneInput
  int32_t nps, nrs, n_entries, n_t, tail, zero, vec, ms;  // ms: positions before the tail
  const int32_t* pos;         // [m] position of each species
  const int32_t* species;           // [nps][P] position | species << 16 (no species: m)
  const uint4* packets[LS_COUNT];
  int32_t packet_count[LS_COUNT];
  int32_t levels[LS_COUNT], level_at[LS_COUNT];  // of the scheduled streams: count, place in the table
  // small tables in one block: [LS_COUNT][warps] first packet and rounds (int32 each), [warps][4] ends of
  // the net production's segments (int32), then each scheduled stream's [level][warp] rounds (bytes)
  const uint4* table;
  int32_t table_bytes;              // a multiple of 16
  const double* emis;               // [m]
};

// Byte offsets of the CTA's shared-memory sections; every array is [...][S].
struct LaneSmem {
  uint32_t lu, x, v, q, ctl, tol, ext, prog, bytes;
  uint32_t stream[LS_COUNT];  // resident streams, 0: read from global memory
  uint32_t stage, stage_bytes;  // what is left, for chunks of the others
};

struct LaneParams {
  AdvanceParams a;
  LaneDev p;
  LaneSmem s;
  // gas-aerosol problem: rows [active gas, particles], the state row's constant gas species between them
  AeroDev aero;
  const double* number_conc;  // [B][nP]
  int32_t n_gas;              // gas species, active and constant
  int32_t* redo_count;  // samples left to the general kernel (status kStatusRedo)
};

// Kernel shapes: samples per CTA, warps per CTA, CTAs per SM (launch bounds); P = 32 warps / S slots.
struct LaneShape {
  int S, warps, ctas;
  int P() const { return 32 * warps / S; }
};
constexpr LaneShape kLaneShapes[] = {{16, 8, 2}, {16, 16, 1}, {8, 16, 1}, {4, 16, 1}, {2, 16, 1}, {1, 8, 1}};
constexpr int kLaneShapeCount = 6;

// Control block of the CTA: per sample 6 doubles and 18 ints, and two flags.
constexpr int kLaneControlDoubles = 6, kLaneControlInts = 18;
constexpr uint32_t lane_control_bytes(int S) {
  return (static_cast<uint32_t>(S) * (8 * kLaneControlDoubles + 4 * kLaneControlInts) + 16 + 15) & ~15u;
}

// The tail's published rows and columns: one sample's values side by side, samples this far apart (16-byte
// loads of eight samples then fall in distinct banks).
constexpr int lane_publish_stride(int n_t) { return n_t + 4; }
// m rows, Q rows of q, D slots of d; ext: doubles per sample of the aerosol problem (else 0).
inline LaneSmem lane_smem(int m, int Q, int D, int ext, int n_entries, int n_t, int table_bytes, int S, int P,
                          bool fp64) {
  auto up16 = [](size_t b) { return static_cast<uint32_t>((b + 15) & ~size_t(15)); };
  const size_t t = fp64 ? 8 : 4;
  LaneSmem s{};
  uint32_t o = 0;
  s.lu = o;
  o += up16(t * S * n_entries);
  s.x = o;
  o += up16(sizeof(double) * S * (m + 1));
  s.v = o;
  if (!fp64) o += up16(sizeof(double) * S * (m + 1));
  // q and, in its place at other times, the factor-slot derivatives, the tail's pivot rows and
  // columns (two of each, double-buffered), and the warps' sums of the two norms
  s.q = o;
  o += up16(S * std::max(std::max(sizeof(double) * (Q + 1), t * (D + 1)),
                         std::max(t * 8 * lane_publish_stride(n_t), sizeof(double) * (2 * (P * S / 32) + 1))));
  s.ctl = o;
  o += lane_control_bytes(S);
  s.tol = o;  // step tolerances by position, the same for every sample
  o += up16(2 * sizeof(double) * m);
  s.ext = o;
  o += up16(sizeof(double) * S * ext);
  s.prog = o;  // LaneDev::table
  o += static_cast<uint32_t>(table_bytes);
  s.bytes = o;
  return s;
}
// Gives the streams, in order, the shared memory that the other sections leave: a packet
// from shared memory is there in tens of cycles, one from L2 in hundreds, and the short levels of the
// substitutions cannot hide that.
// Shared memory of one of `ctas` CTAs on an SM (228 KB, 1 KB of it per CTA).
inline uint32_t lane_room(int ctas, int max_smem) {
  return std::min<uint32_t>(static_cast<uint32_t>(max_smem), 228u * 1024u / ctas - 1024u);
}
inline void lane_place_streams(LaneSmem& s, const LaneDev& d, uint32_t room) {
  for (int k = 0; k < LS_COUNT; ++k) {
    const uint32_t b = 16u * static_cast<uint32_t>(d.packet_count[k]);
    s.stream[k] = 0;
    if (s.bytes + b > room) continue;
    s.stream[k] = s.bytes;
    s.bytes += b;
  }
  s.stage = s.bytes;
  s.stage_bytes = 0;
  for (int k = 0; k < LS_COUNT; ++k)
    if (!s.stream[k]) s.stage_bytes = (room - s.bytes) & ~15u;
  s.bytes += s.stage_bytes;
}

enum LaneForm { LANE_F32 = 0, LANE_F64 = 1, LANE_AERO = 2 };  // the aerosol problem is FP64
constexpr int kLaneForms = 3;
inline bool lane_has_shape(LaneForm form, int shape) { return form != LANE_AERO || kLaneShapes[shape].S <= 8; }
const void* lane_kernel(int shape, LaneForm form);
cudaError_t launch_lanes(const LaneParams& P, int shape, LaneForm form, int grid, cudaStream_t stream);
// Doubles per sample of the aerosol problem's own section.
inline int lane_aero_doubles(const AeroDev& A) { return 4 * A.nS + 6 * A.nP + 4 * A.nP * A.nS + A.nP * A.nA; }

}  // namespace tchem_gb
