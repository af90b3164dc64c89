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

}  // namespace

LaneTables* upload_lane_tables(const HostTables& ht, int device, int max_smem) {
  LanePattern pat;
  try {
    pat = build_lane_pattern(ht);
  } catch (const std::domain_error&) {
    return nullptr;
  }
  struct Offsets {
    size_t species, table, packets[LS_COUNT];
  } at[2][kLaneShapeCount] = {};
  LaneTables t;
  Arena arena;
  const size_t emis = arena.put(reinterpret_cast<const double*>(ht.blob.data() + ht.L.off_emis),
                                static_cast<size_t>(ht.L.m));
  bool any = false;
  for (int fp64 = 0; fp64 < 2; ++fp64)
    for (int k = 0; k < kLaneShapeCount; ++k) {
      const LaneShape sh = kLaneShapes[k];
      const int n_t = lane_tail_size(ht.L, pat, sh, fp64 != 0);
      LaneDev& d = t.dev[fp64][k];
      if (lane_smem(ht.L, lane_entries(pat, sh.P(), n_t), n_t, 0, sh.S, sh.P(), fp64 != 0).bytes >
          lane_room(sh.ctas, max_smem))
        continue;
      LaneProgram lp;
      try {
        lp = build_lane_program(ht, pat, sh.P(), sh.warps, n_t, fp64 != 0);
      } catch (const std::domain_error&) {
        continue;
      }
      Offsets& o = at[fp64][k];
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
      if (lane_smem(ht.L, lp.n_entries, n_t, d.table_bytes, sh.S, sh.P(), fp64 != 0).bytes >
          lane_room(sh.ctas, max_smem))
        continue;
      o.table = arena.put(table);
      o.species = arena.put(lp.species);
      t.valid[fp64][k] = any = true;
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
  for (int fp64 = 0; fp64 < 2; ++fp64)
    for (int k = 0; k < kLaneShapeCount; ++k) {
      if (!t.valid[fp64][k]) continue;
      const Offsets& o = at[fp64][k];
      LaneDev& d = t.dev[fp64][k];
      d.species = reinterpret_cast<const int32_t*>(b + o.species);
      d.table = reinterpret_cast<const uint4*>(b + o.table);
      for (int i = 0; i < LS_COUNT; ++i) d.packets[i] = reinterpret_cast<const uint4*>(b + o.packets[i]);
      d.emis = reinterpret_cast<const double*>(b + emis);
    }
  return new LaneTables(t);
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
