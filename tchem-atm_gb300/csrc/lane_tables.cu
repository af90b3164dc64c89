// Builds and uploads the instruction streams of the batched sparse-LU kernel (lane_program.hpp).
#include "lane_tables.hpp"

#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <stdexcept>
#include <string>
#include <vector>

#include "lane_program.hpp"

namespace tchem_gb {
namespace {

struct Arena {
  std::vector<unsigned char> host;
  template <typename T>
  size_t put(const T* v, size_t n) {
    const size_t o = (host.size() + 255) & ~size_t(255);
    host.resize(o + n * sizeof(T));
    if (n) std::memcpy(host.data() + o, v, n * sizeof(T));
    return o;
  }
  template <typename T>
  size_t put(const std::vector<T>& v) {
    return put(v.data(), v.size());
  }
};

// Streams of the forms [first, last] of one problem.
LaneTables* upload(const LaneInput& in, int ext, int first, int last, int device, int max_smem) {
  LanePattern pat;
  try {
    pat = build_lane_pattern(in);
  } catch (const std::domain_error&) {
    return nullptr;
  }
  struct Offsets {
    size_t species, table, packets[LS_COUNT];
  } at[kLaneForms][kLaneShapeCount] = {};
  LaneTables t;
  Arena arena;
  const size_t emis = arena.put(in.emis), pos = arena.put(pat.pos);
  bool any = false;
  for (int form = first; form <= last; ++form)
    for (int k = 0; k < kLaneShapeCount; ++k) {
      if (!lane_has_shape(static_cast<LaneForm>(form), k)) continue;
      const bool fp64 = form != LANE_F32;
      const LaneShape sh = kLaneShapes[k];
      const int n_t = lane_tail_size(in, pat, sh, fp64);
      LaneDev& d = t.dev[form][k];
      if (lane_smem(in.m, in.Q, in.D, ext, lane_entries(pat, sh.P(), n_t), n_t, 0, sh.S, sh.P(), fp64).bytes >
          lane_room(sh.ctas, max_smem))
        continue;
      LaneProgram lp;
      try {
        lp = build_lane_program(in, pat, sh.P(), sh.warps, n_t, fp64);
      } catch (const std::domain_error&) {
        continue;
      }
      Offsets& o = at[form][k];
      std::vector<int32_t> head(2 * LS_COUNT * sh.warps);
      std::vector<uint8_t> levels;
      const size_t level_base = 4 * (head.size() + lp.net_end.size());
      auto put = [&](int id, const LaneStream& s) {
        o.packets[id] = arena.put(s.packets);
        d.packet_count[id] = static_cast<int32_t>(s.packets.size());
        for (int w = 0; w < sh.warps; ++w) {
          head[2 * (id * sh.warps + w)] = s.first[w];
          head[2 * (id * sh.warps + w) + 1] = s.rounds[w];
        }
        d.levels[id] = s.levels;
        d.level_at[id] = static_cast<int32_t>(level_base + levels.size());
        levels.insert(levels.end(), s.level_rounds.begin(), s.level_rounds.end());
      };
      put(LS_NET, lp.net);
      put(LS_FORWARD, lp.forward);
      put(LS_BACKWARD, lp.backward);
      put(LS_REACTIONS, lp.reactions);
      put(LS_FACTOR, lp.factor);
      put(LS_MATRIX, lp.matrix);
      std::vector<unsigned char> table((level_base + levels.size() + 15) / 16 * 16, 0);
      std::memcpy(table.data(), head.data(), 4 * head.size());
      std::memcpy(table.data() + 4 * head.size(), lp.net_end.data(), 4 * lp.net_end.size());
      if (!levels.empty()) std::memcpy(table.data() + level_base, levels.data(), levels.size());
      d.table_bytes = static_cast<int32_t>(table.size());
      if (lane_smem(in.m, in.Q, in.D, ext, lp.n_entries, n_t, d.table_bytes, sh.S, sh.P(), fp64).bytes >
          lane_room(sh.ctas, max_smem))
        continue;
      o.table = arena.put(table);
      o.species = arena.put(lp.species);
      t.valid[form][k] = any = true;
      d.m = in.m;
      d.R = in.R;
      d.Q = in.Q;
      d.D = in.D;
      d.nps = lp.nps;
      d.nrs = lp.nrs;
      d.n_entries = lp.n_entries;
      d.n_t = lp.n_t;
      d.tail = lp.tail;
      d.zero = lp.zero;
      d.vec = lp.vec;
      d.ms = std::max(0, lp.m - lp.n_t);
    }
  if (!any) return nullptr;
  t.device = device;
  int prev = 0;
  cudaGetDevice(&prev);
  if (cudaSetDevice(device) != cudaSuccess) throw std::runtime_error("cudaSetDevice failed");
  cudaError_t e = cudaMalloc(&t.allocation, arena.host.size());
  if (e == cudaSuccess) e = cudaMemcpy(t.allocation, arena.host.data(), arena.host.size(), cudaMemcpyHostToDevice);
  cudaSetDevice(prev);
  if (e != cudaSuccess) {
    if (t.allocation) cudaFree(t.allocation);
    cudaGetLastError();
    throw std::runtime_error(std::string("instruction streams: ") + cudaGetErrorString(e));
  }
  const unsigned char* b = static_cast<const unsigned char*>(t.allocation);
  for (int form = first; form <= last; ++form)
    for (int k = 0; k < kLaneShapeCount; ++k) {
      if (!t.valid[form][k]) continue;
      const Offsets& o = at[form][k];
      LaneDev& d = t.dev[form][k];
      d.species = reinterpret_cast<const int32_t*>(b + o.species);
      d.table = reinterpret_cast<const uint4*>(b + o.table);
      for (int i = 0; i < LS_COUNT; ++i) d.packets[i] = reinterpret_cast<const uint4*>(b + o.packets[i]);
      d.emis = reinterpret_cast<const double*>(b + emis);
      d.pos = reinterpret_cast<const int32_t*>(b + pos);
    }
  return new LaneTables(t);
}

}  // namespace

LaneTables* upload_lane_tables(const HostTables& ht, int device, int max_smem) {
  return upload(lane_input(ht), 0, LANE_F32, LANE_F64, device, max_smem);
}

LaneTables* upload_aero_lane_tables(const HostTables& ht, const AeroDev& A, const int32_t* simpol_index, int device,
                                    int max_smem) {
  // Each (particle, SIMPOL entry) pair is two rows of q: what its transfer takes from the gas species and
  // gives to the aerosol species; and 2 (1 + nA) slots of d: the derivatives of the two by the gas species
  // and by each species of the particle. The kernel computes both (aero_transfers, aero_slots).
  LaneInput in = lane_input(ht);
  const int R = in.R, D = in.D, nA = A.nA;
  in.m = A.M;
  in.net.resize(A.M);
  in.emis.resize(A.M, 0.0);
  for (int ip = 0; ip < A.nP; ++ip)
    for (int is = 0; is < A.nS; ++is) {
      const int e = ip * A.nS + is, gas = simpol_index[3 * is + 1], aero = simpol_index[3 * is] + ip * nA;
      in.net[gas].push_back({R + 2 * e, 1.0});
      in.net[aero].push_back({R + 2 * e + 1, 1.0});
      for (int c = 0; c <= nA; ++c) {
        const int col = c == 0 ? gas : A.m_gas + ip * nA + c - 1, slot = D + 2 * (e * (1 + nA) + c);
        in.jac.push_back({gas, col, {{slot, 1.0}}});
        in.jac.push_back({aero, col, {{slot + 1, 1.0}}});
      }
    }
  in.Q = R + 2 * A.nP * A.nS;
  in.D = D + 2 * A.nP * A.nS * (1 + nA);
  return upload(in, lane_aero_doubles(A), LANE_AERO, LANE_AERO, device, max_smem);
}

// The batched sparse-LU kernel's shape for a batch: the fewest samples per CTA (the most slots per
// sample, the shortest round) whose lanes hold the batch at once, or `slack` times over, else the most
// that one CTA per SM holds (samples then follow each other through the lanes). Box samples differ in length, the
// longest taking about twice the mean, and the longest one's rounds are shorter with fewer samples beside it:
// FP32 with up to 64 species gains up to twice the room (51 species over 2 s: 2,432 samples 269 ms with
// 16 per CTA and 257 with 8, 620 samples 149 with two and 133 with four, 230 samples 104 with two and 92 with one; 310
// samples 93 with two and 100 with one), where a round's time depends on the samples in it more than that (FP64, larger
// matrices) up to three times (51 species FP64, 900 samples 155 ms with four and 141 with two; 120 species, 400 samples
// 144 ms with two and 131 with one; other sizes in between were not measured). E3SM columns and aerosol cells are alike
// in length and are held at once (FP64, 1,300 columns over 600 s: 12 ms with 8, 8 with 16). The shape with two CTAs per
// SM takes longer per round (51 species: 160 k cycles for 32 samples against 104 k for 16) and less per sample, so for
// boxes it pays when its lanes are filled several times over, from four times its room: 10,000 samples over 1 s 464 ms
// with one CTA per SM, 494 ms with two; 16,384 695 and 690 ms; 40,000 1,462 and 1,343 ms. E3SM columns follow the
// same line, though alike in length they would gain from it as soon as one CTA per SM does not hold them (FP64 over 600 s,
// 2,600 columns 14.7 ms with one CTA and 10.2 with two, 4,000 15.1 and 10.6).
LanePlan plan_lanes(const LaneTables* t, LaneForm form, int ext, int sm_count, int max_smem, int nbatch, int slack) {
  LanePlan p;
  p.form = form;
  long best = 0;
  for (int k = kLaneShapeCount - 1; t && k >= 0; --k) {
    if (!t->valid[form][k]) continue;
    const LaneShape sh = kLaneShapes[k];
    const long room = static_cast<long>(sm_count) * sh.ctas * sh.S;
    if (room <= best || (sh.ctas > 1 && nbatch < 4 * room && p.shape >= 0)) continue;
    best = room;
    p.shape = k;
    if (slack * room >= nbatch) break;
  }
  if (p.shape < 0) return p;
  const LaneShape sh = kLaneShapes[p.shape];
  p.dev = t->dev[form][p.shape];
  p.smem = lane_smem(p.dev.m, p.dev.Q, p.dev.D, ext, p.dev.n_entries, p.dev.n_t, p.dev.table_bytes, sh.S, sh.P(),
                     form != LANE_F32);
  lane_place_streams(p.smem, p.dev, lane_room(sh.ctas, max_smem));
  // the limit, not this plan's bytes: another group or thread may launch the same kernel with more
  cudaFuncSetAttribute(lane_kernel(p.shape, form), cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem);
  p.grid = std::min(sm_count * sh.ctas, (std::max(nbatch, 1) + sh.S - 1) / sh.S);
  return p;
}

// A round of the batched kernel has some 70 (FP32) to 175 (FP64) CTA barriers however small the matrix, which a
// one-warp or two-warp kernel on a matrix in registers does not pay: few species, or so many samples that the SMs
// hold that kernel's warps one beside the other, and the batched kernel is the slower one until the batch fills
// its two-CTA shape (128 samples per SM). Measured on 152 SMs, ms of the register kernel / of the batched one:
//  * FP32, up to 32 species (one warp, dense LU): 8 species over 1e-2 s, 150 samples 19.6 / 22.7, 1,000 22.5 / 29.9, 10,000
//    44 / 50, 20,000 74 / 50; 20 species over 1e-2 s, 150 samples 32 / 23, 600 32 / 33, 4,000 42 / 62, 20,000 88 / 85;
//    32 species over 1e-2 s, 1,000 samples 54 / 43, 2,000 63 / 60, 4,000 67 / 83, 20,000 146 / 135. The first crossing
//    goes with the square of the species: at 1.2, 3.3 and 8.5 samples per SM for 12, 20 and 32 species.
//  * FP32, 33 to 64 species (two warps, Gauss-Jordan): between 5.5 and 14 samples per SM. 51 species over 60 s, 800
//    samples 234 / 227, 900 231 / 237, 1,600 322 / 333, 2,432 413 / 400; over 1e-3 s, 800 48 / 45, 1,250 47 / 53,
//    1,900 55 / 58; 64 species over 1e-2 s, 900 samples 41 / 49, 1,900 48 / 56. Above it the batched kernel wins over
//    seconds and more (51 species over 60 s, 4,000 samples 588 / 520) and loses where a few samples need many times
//    the others' iterations (over 1e-3 s, 4,000 samples 62 / 68 to 87); the horizon is not known on the host.
//  * FP64, up to 3 species: over 1e-3 s, 150 samples 1.14 / 0.83, 1,000 1.17 / 1.97, 2,000 2.1 / 2.0.
bool lanes_pay_for_box(LaneForm form, int m, int sm_count, int nbatch) {
  const long B = nbatch, sms = sm_count;
  if (B >= 128 * sms) return true;
  if (form != LANE_F32) return m > 3 || B <= sms || B > 13 * sms;
  if (m <= 8) return false;
  if (m <= 32) return 120 * B <= sms * m * m;
  return m > 64 || 2 * B <= 11 * sms || B > 14 * sms;
}

void destroy_lane_tables(LaneTables* t) {
  if (!t) return;
  int prev = 0;
  cudaGetDevice(&prev);
  cudaSetDevice(t->device);
  cudaFree(t->allocation);
  cudaSetDevice(prev);
  delete t;
}

}  // namespace tchem_gb
