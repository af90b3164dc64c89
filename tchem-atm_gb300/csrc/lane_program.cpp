// Order, schedule and packet streams of the batched time-advance kernel (see lane_program.hpp).
#include "lane_program.hpp"

#include <algorithm>
#include <cstring>
#include <numeric>
#include <queue>
#include <stdexcept>

namespace tchem_gb {
namespace {

// Host copies of the packed tables' sections (the plain form's CSR blob).
template <typename T>
const T* section(const HostTables& ht, int32_t off) {
  return reinterpret_cast<const T*>(ht.blob.data() + off);
}

constexpr int kProducts = 3;      // products per factor / solve packet
constexpr int kLevelPackets = 2;  // shortest level: packets per slot

struct Task {
  int dst = 0;
  int scale = -1;            // position of the scaling reciprocal
  uint32_t flags = 0;        // what the last packet does besides: LP_LCOL, LP_PIVOT
  std::vector<std::pair<int, int>> ops;
};

// List scheduling of tasks whose operands are entries (final from the start unless a task writes
// them). Emits the slots' packets level by level.
struct Scheduler {
  int P, warps, zero, one, pair;  // pair: rounds the kernel takes at a time
  std::vector<std::vector<Packet>> slot;  // packets of every slot so far
  int levels = 0;
  std::vector<uint8_t> level_rounds;

  Scheduler(int P_, int warps_, int zero_, int one_, int pair_)
      : P(P_), warps(warps_), zero(zero_), one(one_), pair(pair_), slot(P_) {}

  Packet nop() const {
    const uint32_t z = static_cast<uint32_t>(zero) | (static_cast<uint32_t>(zero) << 16);
    return Packet{{static_cast<uint32_t>(zero) | (static_cast<uint32_t>(one) << LP_SCALE_SHIFT), z, z, z}};
  }

  // The task's products as packets of slot s.
  void emit(int s, const Task& t, const std::pair<int, int>* ops, int n, bool end) {
    const uint32_t z = static_cast<uint32_t>(zero) | (static_cast<uint32_t>(zero) << 16);
    const int np = std::max(1, (n + kProducts - 1) / kProducts);
    for (int k = 0; k < np; ++k) {
      Packet p{};
      for (int q = 0; q < kProducts; ++q) {
        const int o = k * kProducts + q;
        p.w[1 + q] = o < n ? static_cast<uint32_t>(ops[o].first) | (static_cast<uint32_t>(ops[o].second) << 16) : z;
      }
      const int here = n - k * kProducts;
      const bool last = end && k == np - 1;
      p.w[0] = static_cast<uint32_t>(t.dst) | (k > 0 ? uint32_t(LP_CONT) : 0u) | (here > 1 ? uint32_t(LP_TWO) : 0u) |
               (here > 2 ? uint32_t(LP_THREE) : 0u) | (here > 0 ? uint32_t(LP_ONE) : 0u) |
               (last ? t.flags | (t.scale >= 0 ? uint32_t(LP_SCALED) : 0u) : 0u) |
               (static_cast<uint32_t>(last && t.scale >= 0 ? t.scale : one) << LP_SCALE_SHIFT);
      slot[s].push_back(p);
    }
  }

  // Pads the slots of each warp to its rounds of the level.
  void close_level(const std::vector<size_t>& begin) {
    const int spw = P / warps;
    for (int w = 0; w < warps; ++w) {
      size_t n = begin[w];
      for (int s = w * spw; s < (w + 1) * spw; ++s) n = std::max(n, slot[s].size());
      n += (n - begin[w]) % pair;
      for (int s = w * spw; s < (w + 1) * spw; ++s) slot[s].resize(n, nop());
      level_rounds.push_back(static_cast<uint8_t>(n - begin[w]));
    }
    ++levels;
  }

  void run(const std::vector<Task>& tasks, int n_entries) {
    const int n = static_cast<int>(tasks.size());
    std::vector<int> writer(n_entries, -1);
    for (int i = 0; i < n; ++i) writer[tasks[i].dst] = i;
    // heights: longest chain of tasks that wait for this one (diagonal reciprocals: entry = position)
    std::vector<std::vector<int>> users(n);
    std::vector<int> waits(n, 0);
    auto dep = [&](int entry, int user, std::vector<int>& seen) {
      const int w = writer[entry];
      if (w >= 0 && w != user && seen[w] != user) {
        seen[w] = user;
        users[w].push_back(user);
        ++waits[user];
      }
    };
    {
      std::vector<int> seen(n, -1);
      for (int i = 0; i < n; ++i) {
        for (const auto& o : tasks[i].ops) {
          dep(o.first, i, seen);
          dep(o.second, i, seen);
        }
        if (tasks[i].scale >= 0) dep(tasks[i].scale, i, seen);
      }
    }
    std::vector<int> topo, height(n, 0);
    {
      std::vector<int> left = waits;
      for (int i = 0; i < n; ++i)
        if (left[i] == 0) topo.push_back(i);
      for (size_t q = 0; q < topo.size(); ++q)
        for (int u : users[topo[q]])
          if (--left[u] == 0) topo.push_back(u);
      if (static_cast<int>(topo.size()) != n) throw std::logic_error("lane program: cyclic tasks");
      for (int q = n - 1; q >= 0; --q)
        for (int u : users[topo[q]]) height[topo[q]] = std::max(height[topo[q]], height[u] + 1);
    }
    // ready products: those whose operands are final
    std::vector<std::vector<std::pair<int, int>>> ready(n);
    std::vector<std::vector<std::pair<int, int>>> on(n_entries);  // (task, op) waiting for an entry
    std::vector<std::vector<char>> pending(n);
    std::vector<int> remaining(n), scale_wait(n, 0);
    std::vector<std::vector<int>> scaled_by(n_entries);
    std::vector<char> done(n, 0);
    for (int i = 0; i < n; ++i) {
      remaining[i] = static_cast<int>(tasks[i].ops.size());
      pending[i].assign(tasks[i].ops.size(), 0);
      for (size_t o = 0; o < tasks[i].ops.size(); ++o) {
        const int a = tasks[i].ops[o].first, b = tasks[i].ops[o].second;
        if (writer[a] >= 0) { ++pending[i][o]; on[a].push_back({i, static_cast<int>(o)}); }
        if (writer[b] >= 0) { ++pending[i][o]; on[b].push_back({i, static_cast<int>(o)}); }
        if (!pending[i][o]) ready[i].push_back(tasks[i].ops[o]);
      }
      if (tasks[i].scale >= 0 && writer[tasks[i].scale] >= 0) {
        scale_wait[i] = 1;
        scaled_by[tasks[i].scale].push_back(i);
      }
    }
    int left = n;
    std::vector<int> open(n);
    std::iota(open.begin(), open.end(), 0);
    while (left > 0) {
      // candidates: tasks that can end in this level, then those with whole packets of ready products
      std::vector<std::pair<int, int>> cand;  // (-priority, task)
      long total = 0;
      for (int i : open) {
        const int nr = static_cast<int>(ready[i].size());
        const bool whole = nr == remaining[i] && !scale_wait[i];
        if (!whole && nr < kProducts) continue;
        const int np = whole ? std::max(1, (nr + kProducts - 1) / kProducts) : nr / kProducts;
        total += np;
        cand.push_back({-(2 * height[i] + (whole ? 1 : 0)), i});
      }
      if (cand.empty()) throw std::logic_error("lane program: no task is ready");
      std::sort(cand.begin(), cand.end());
      // a level's rounds fit a byte
      const int cap =
          std::min(254, (std::max<int>(kLevelPackets, static_cast<int>((total + P - 1) / P)) + pair - 1) / pair * pair);
      std::vector<size_t> begin(warps);
      for (int w = 0; w < warps; ++w) begin[w] = slot[w * (P / warps)].size();
      std::priority_queue<std::pair<int, int>, std::vector<std::pair<int, int>>, std::greater<>> load;
      for (int s = 0; s < P; ++s) load.push({0, s});
      std::vector<int> ended;
      for (const auto& c : cand) {
        if (load.empty()) break;
        const int i = c.second;
        const auto top = load.top();
        const int room = cap - top.first;
        if (room <= 0) break;
        const int nr = static_cast<int>(ready[i].size());
        const bool whole = nr == remaining[i] && !scale_wait[i];
        const int need = whole ? std::max(1, (nr + kProducts - 1) / kProducts) : nr / kProducts;
        const int np = std::min(need, room);
        const bool end = whole && np == need;
        const int take = end ? nr : std::min(nr, np * kProducts);
        load.pop();
        emit(top.second, tasks[i], ready[i].data(), take, end);
        ready[i].erase(ready[i].begin(), ready[i].begin() + take);
        remaining[i] -= take;
        if (top.first + np < cap) load.push({top.first + np, top.second});
        if (end) ended.push_back(i);
      }
      close_level(begin);
      for (int i : ended) {
        done[i] = 1;
        --left;
        const int e = tasks[i].dst;
        for (const auto& w : on[e])
          if (--pending[w.first][w.second] == 0) ready[w.first].push_back(tasks[w.first].ops[w.second]);
        for (int t : scaled_by[e]) scale_wait[t] = 0;
      }
      open.erase(std::remove_if(open.begin(), open.end(), [&](int i) { return done[i] != 0; }), open.end());
    }
  }
};

// The slots' packets by warp and round, padded to pairs, with a spare pair.
LaneStream interleave(const std::vector<std::vector<Packet>>& slot, int warps, const Packet& nop, int pair = 2,
                      bool scheduled = false) {
  LaneStream st;
  const int spw = static_cast<int>(slot.size()) / warps;
  for (int w = 0; w < warps; ++w) {
    size_t n = 0;
    for (int s = w * spw; s < (w + 1) * spw; ++s) n = std::max(n, slot[s].size());
    n += n % pair;
    st.first.push_back(static_cast<int32_t>(st.packets.size()));
    st.rounds.push_back(static_cast<int32_t>(n));
    for (size_t k = 0; k < n + 2; ++k) {
      const size_t at = st.packets.size();
      uint32_t flags = 0;
      for (int s = w * spw; s < (w + 1) * spw; ++s) {
        st.packets.push_back(k < slot[s].size() ? slot[s][k] : nop);
        flags |= st.packets.back().w[0];
      }
      if (scheduled)
        for (size_t q = at; q < st.packets.size(); ++q)
          st.packets[q].w[0] |= (flags & kLaneWarpFlags) | ((flags & LP_PIVOT) ? uint32_t(LP_PIVOTS) : 0u);
    }
  }
  return st;
}

}  // namespace

LaneInput lane_input(const HostTables& ht) {
  const MechLayout& L = ht.L;
  LaneInput in;
  in.m = L.m;
  in.R = in.Q = L.R;
  in.D = L.NF;
  in.max_factors = L.max_factors;
  const int32_t* rf_ptr = section<int32_t>(ht, L.off_rf_ptr);
  const int16_t* rf_sp = section<int16_t>(ht, L.off_rf_sp);
  in.rf_ptr.assign(rf_ptr, rf_ptr + L.R + 1);
  in.rf_sp.assign(rf_sp, rf_sp + L.NF);
  const int32_t* pr_ptr = section<int32_t>(ht, L.off_pr_ptr);
  const int16_t* pr_r = section<int16_t>(ht, L.off_pr_r);
  const double* pr_nu = section<double>(ht, L.off_pr_nu);
  in.net.resize(L.m);
  for (int i = 0; i < L.m; ++i)
    for (int e = pr_ptr[i]; e < pr_ptr[i + 1]; ++e) in.net[i].push_back({pr_r[e], pr_nu[e]});
  const int32_t* rc = section<int32_t>(ht, L.off_jz_rc);
  const int32_t* jz_ptr = section<int32_t>(ht, L.off_jz_ptr);
  const int16_t* jc_f = section<int16_t>(ht, L.off_jc_f);
  const double* jc_nu = section<double>(ht, L.off_jc_nu);
  for (int z = 0; z < L.NZ; ++z) {
    LaneInput::Entry e{rc[z] >> 16, rc[z] & 0xffff, {}};
    for (int c = jz_ptr[z]; c < jz_ptr[z + 1]; ++c) e.terms.push_back({jc_f[c], jc_nu[c]});
    in.jac.push_back(std::move(e));
  }
  const double* emis = section<double>(ht, L.off_emis);
  in.emis.assign(emis, emis + L.m);
  return in;
}

LanePattern build_lane_pattern(const LaneInput& in) {
  const int m = in.m;
  if (m > kLaneMaxSpecies) throw std::domain_error("lane program: too many species");
  if (in.Q > 0xffff || in.D >= 0xffff) throw std::domain_error("lane program: too many rates");
  if (in.max_factors > 3) throw std::domain_error("lane program: more than three reactant factors");
  std::vector<char> A(static_cast<size_t>(m) * m, 0);
  auto at = [&](int i, int j) -> char& { return A[static_cast<size_t>(i) * m + j]; };
  for (int i = 0; i < m; ++i) at(i, i) = 1;
  for (const auto& e : in.jac) at(e.row, e.col) = 1;
  LanePattern p;
  p.m = m;
  // Greedy Markowitz on the diagonal, several independent pivots at a time: every remaining species
  // within half again of the smallest score that shares no entry with one taken in this pass. The
  // fill grows by under 1 % and the elimination tree gets lower (34 to 32 levels at 51 species).
  std::vector<char> left(m, 1);
  while (static_cast<int>(p.order.size()) < m) {
    std::vector<std::pair<long, int>> score;
    for (int j = 0; j < m; ++j) {
      if (!left[j]) continue;
      long r = 0, c = 0;
      for (int t = 0; t < m; ++t)
        if (left[t]) {
          r += at(j, t);
          c += at(t, j);
        }
      score.push_back({(r - 1) * (c - 1), j});
    }
    std::sort(score.begin(), score.end());
    const long low = score[0].first;
    const double thr = std::max(1.5 * low, low + (low < 4 ? 2.0 : 0.0));
    std::vector<char> blocked(m, 0);
    std::vector<int> take;
    for (const auto& s : score) {
      if (s.first > thr) break;
      if (blocked[s.second]) continue;
      take.push_back(s.second);
      for (int t = 0; t < m; ++t)
        if (left[t] && (at(s.second, t) || at(t, s.second))) blocked[t] = 1;
    }
    for (int k : take) {
      left[k] = 0;
      p.order.push_back(k);
      for (int i = 0; i < m; ++i) {
        if (!left[i] || !at(i, k)) continue;
        for (int j = 0; j < m; ++j)
          if (left[j] && at(k, j)) at(i, j) = 1;
      }
    }
  }
  p.pos.assign(m, 0);
  for (int k = 0; k < m; ++k) p.pos[p.order[k]] = k;
  p.fill.assign(static_cast<size_t>(m) * m, 0);
  for (int k = 0; k < m; ++k)
    for (int l = 0; l < m; ++l) p.fill[static_cast<size_t>(k) * m + l] = at(p.order[k], p.order[l]);
  return p;
}

int lane_entries(const LanePattern& pat, int P, int n_t) {
  const int m = pat.m, ms = std::max(0, m - n_t);
  int n = 0;
  for (int k = 0; k < m; ++k)
    for (int l = 0; l < m; ++l)
      if ((k < ms || l < ms) && pat.fill[static_cast<size_t>(k) * m + l]) ++n;
  return n + 1 + n_t * lane_tail_stride(P, n_t) + 1 + ms + std::max(n_t, m - ms);
}

// By the estimated cycles of one round's factorization and solves. Issue: a packet row is about 35
// instructions over four schedulers; latency: a level's barrier and dependent loads about 250 cycles, a
// tail pivot about 250 (measured with one pivot per step; steps take two now, which these choices do not use yet). The
// tables' size, not known before the program is built, is taken as 2,048 bytes, and as 704 with two CTAs per SM, what the
// 51-species sections leave there at a tail of 24; the program's own size is checked before a shape is offered. FP64
// has no tail: the inverse needs three times the products of the triangular factors, on a pipe of 2 per cycle (measured
// with 16 samples per CTA; with one the pipe idles, and a tail there has not been tried).
int lane_tail_size(const LaneInput& in, const LanePattern& pat, const LaneShape& shape, bool fp64) {
  if (fp64) return 0;
  const int S = shape.S, warps = shape.warps;
  const int m = pat.m, P = shape.P(), gr = lane_grid_rows(P), gc = lane_grid_cols(P);
  auto F = [&](int i, int j) { return pat.fill[static_cast<size_t>(i) * m + j] != 0; };
  std::vector<long> ops(m), level(m, 0);
  for (int k = 0; k < m; ++k) {
    long r = 0, c = 0;
    for (int t = k + 1; t < m; ++t) {
      r += F(t, k);
      c += F(k, t);
    }
    ops[k] = r * c;
    for (int j = 0; j < k; ++j)
      if (F(k, j) || F(j, k)) level[k] = std::max(level[k], level[j] + 1);
  }
  const double share = S / 32.0;  // warp rows per item
  const int solves = 3;
  int best = 0;
  double best_cost = 0.0;
  for (int c = -1; c < kLaneTiles; ++c) {
    const int tr = c < 0 ? 0 : lane_tile(P, warps, c), n_t = tr * gr, tc = n_t / gc, ms = std::max(0, m - n_t);
    if (c > 0 && lane_tile(P, warps, c - 1) * gr >= m) break;  // the smaller tail already holds everything
    long n_ops = 0, n_lv = 0, nnz = 0;
    for (int k = 0; k < ms; ++k) {
      n_ops += ops[k];
      n_lv = std::max(n_lv, level[k] + 1);
    }
    for (int i = 0; i < m; ++i)
      for (int j = 0; j < m; ++j) nnz += (i < ms || j < ms) && F(i, j);
    const double rows = share * (n_ops / 2.0 + solves * nnz / 2.0);
    const double step = tr * tc + 3.0 * (tr + tc) + 40.0;
    const double issue = (35.0 * rows + n_t * warps * step) / 4.0;
    const double latency = 250.0 * n_lv * (2 + 2 * solves) + 250.0 * n_t;
    const uint32_t bytes = lane_smem(in.m, in.Q, in.D, 0, lane_entries(pat, P, n_t), n_t, shape.ctas > 1 ? 704 : 2048, S, P, false).bytes;
    if (bytes > lane_room(shape.ctas, 227 * 1024) && c >= 0) continue;
    const double cost = issue + latency;
    if (c < 0 || cost < best_cost) {
      best = n_t;
      best_cost = cost;
    }
  }
  return best;
}

LaneProgram build_lane_program(const LaneInput& in, const LanePattern& pat, int P, int warps, int n_t, bool fp64) {
  const int m = in.m, R = in.R;
  const int ms = std::max(0, m - n_t);  // sparse positions; tail row i is position ms + i
  LaneProgram lp;
  lp.m = m;
  lp.R = R;
  lp.P = P;
  lp.n_t = n_t;
  lp.nps = (m + P - 1) / P;
  lp.nrs = (R + P - 1) / P;
  if (lp.nps > lane_species(P) || lp.nrs > lane_reactions(P)) throw std::domain_error("lane program: too few slots");
  // the entries' numbers
  std::vector<int32_t> entry(static_cast<size_t>(m) * m, -1);
  auto E = [&](int i, int j) -> int32_t& { return entry[static_cast<size_t>(i) * m + j]; };
  int ne = ms + 1;  // entry ms is the one
  for (int k = 0; k < m; ++k)
    for (int l = 0; l < m; ++l) {
      if (k >= ms && l >= ms) continue;
      if (k == l) E(k, l) = k;
      else if (pat.fill[static_cast<size_t>(k) * m + l]) E(k, l) = ne++;
    }
  lp.tail = ne;
  for (int k = ms; k < m; ++k)
    for (int l = ms; l < m; ++l) E(k, l) = ne + (k - ms) * lane_tail_stride(P, n_t) + (l - ms);
  ne += n_t * lane_tail_stride(P, n_t);
  lp.zero = ne;
  lp.vec = ne + 1;
  lp.n_entries = lp.vec + ms + std::max(n_t, m - ms);
  if (lp.n_entries >= kLaneMaxEntries || ms > 511) throw std::domain_error("lane program: too many entries");
  const int zero = lp.zero, vec = lp.vec, n_entries = lp.n_entries;

  // ---- reactions: most factors first, dealt to the slots in turn ----
  const std::vector<int32_t>&rf_ptr = in.rf_ptr, &rf_sp = in.rf_sp;
  std::vector<int> ro(R);
  std::iota(ro.begin(), ro.end(), 0);
  std::stable_sort(ro.begin(), ro.end(),
                   [&](int a, int b) { return rf_ptr[a + 1] - rf_ptr[a] > rf_ptr[b + 1] - rf_ptr[b]; });
  {
    const Packet none{{static_cast<uint32_t>(m) | (static_cast<uint32_t>(m) << 16), static_cast<uint32_t>(m), 0u,
                       static_cast<uint32_t>(R)}};
    std::vector<Packet> f(static_cast<size_t>(lp.nrs) * P, none);
    for (int q = 0; q < R; ++q) {
      const int r = ro[q], n = rf_ptr[r + 1] - rf_ptr[r];
      uint32_t a[3] = {static_cast<uint32_t>(m), static_cast<uint32_t>(m), static_cast<uint32_t>(m)};
      for (int k = 0; k < n; ++k) a[k] = static_cast<uint32_t>(pat.pos[rf_sp[rf_ptr[r] + k]]);
      f[q] = Packet{{a[0] | (a[1] << 16), a[2] | (static_cast<uint32_t>(n) << 16), static_cast<uint32_t>(rf_ptr[r]),
                     static_cast<uint32_t>(r)}};
    }
    std::vector<std::vector<Packet>> slot(P);
    for (size_t q = 0; q < f.size(); ++q) slot[q % P].push_back(f[q]);
    lp.reactions = interleave(slot, warps, none);
  }

  // ---- species: longest net-production lists first, dealt to the slots in turn and back ----
  std::vector<int> so(m);
  std::iota(so.begin(), so.end(), 0);
  std::stable_sort(so.begin(), so.end(),
                   [&](int a, int b) { return in.net[a].size() > in.net[b].size(); });
  std::vector<int> slot_species(static_cast<size_t>(lp.nps) * P, -1);
  lp.species.assign(static_cast<size_t>(lp.nps) * P, m);
  for (int q = 0; q < m; ++q) {
    const int k = q / P, s = q % P;
    // every other row runs back over the slots, so a slot's total stays even
    const size_t at = static_cast<size_t>(k) * P + (k % 2 ? P - 1 - s : s);
    slot_species[at] = so[q];
    lp.species[at] = pat.pos[so[q]] | (so[q] << 16);
  }
  {
    // one segment per species of the slot, as long as the warp's longest list, a multiple of 2
    const int spw = P / warps;
    std::vector<std::vector<Packet>> slot(P);
    const Packet none{{static_cast<uint32_t>(in.Q), 0u, 0u, 0u}};  // q[Q] = 0
    for (int w = 0; w < warps; ++w)
      for (int k = 0; k < kLaneSegments; ++k) {
        size_t n = 0;
        for (int s = w * spw; s < (w + 1) * spw && k < lp.nps; ++s) {
          const int sp = slot_species[static_cast<size_t>(k) * P + s];
          if (sp < 0) continue;
          for (const auto& t : in.net[sp]) {
            Packet p{};
            p.w[0] = static_cast<uint32_t>(t.first);
            std::memcpy(&p.w[2], &t.second, sizeof(double));
            slot[s].push_back(p);
          }
          n = std::max(n, in.net[sp].size());
        }
        n += n % 2;
        const size_t end = (k ? lp.net_end[w * kLaneSegments + k - 1] : 0) + n;
        for (int s = w * spw; s < (w + 1) * spw; ++s) slot[s].resize(end, none);
        lp.net_end.push_back(static_cast<int32_t>(end));
      }
    lp.net = interleave(slot, warps, none);
  }

  // ---- matrix: the nonzeros of J and the diagonal, longest contribution lists first ----
  {
    std::vector<std::vector<std::pair<int, double>>> list(zero);
    for (const auto& e : in.jac) {
      auto& l = list[E(pat.pos[e.row], pat.pos[e.col])];
      l.insert(l.end(), e.terms.begin(), e.terms.end());
    }
    std::vector<char> diag(zero, 0);
    for (int k = 0; k < ms; ++k) diag[k] = 1;
    for (int k = 0; k < n_t; ++k) diag[lp.tail + k * lane_tail_stride(P, n_t) + k] = 1;  // rows beyond the species: identity
    std::vector<int> eo(zero);
    std::iota(eo.begin(), eo.end(), 0);
    std::stable_sort(eo.begin(), eo.end(), [&](int a, int b) { return list[a].size() > list[b].size(); });
    const uint32_t dz = static_cast<uint32_t>(in.D);  // d[D] = 0
    const int per = fp64 ? 1 : 2;
    std::vector<std::vector<Packet>> slot(P);
    std::priority_queue<std::pair<int, int>, std::vector<std::pair<int, int>>, std::greater<>> load;
    for (int s = 0; s < P; ++s) load.push({0, s});
    for (int e : eo) {
      if (list[e].empty() && !diag[e]) continue;  // fill: zeroed by the kernel
      const auto top = load.top();
      load.pop();
      const int n = static_cast<int>(list[e].size()), np = std::max(1, (n + per - 1) / per);
      for (int k = 0; k < np; ++k) {
        Packet p{};
        p.w[0] = static_cast<uint32_t>(e) | (k == 0 ? uint32_t(LM_START) : 0u) | (k == np - 1 ? uint32_t(LM_END) : 0u) |
                 (diag[e] ? uint32_t(LM_DIAG) : 0u);
        if (!fp64) {
          uint32_t d[2] = {dz, dz};
          float nu[2] = {0.f, 0.f};
          for (int q = 0; q < 2; ++q)
            if (2 * k + q < n) {
              d[q] = static_cast<uint32_t>(list[e][2 * k + q].first);
              nu[q] = static_cast<float>(list[e][2 * k + q].second);
            }
          p.w[1] = d[0] | (d[1] << 16);
          std::memcpy(&p.w[2], nu, sizeof(nu));
        } else {
          double nu = 0.0;
          p.w[1] = dz;
          if (k < n) {
            p.w[1] = static_cast<uint32_t>(list[e][k].first);
            nu = list[e][k].second;
          }
          std::memcpy(&p.w[2], &nu, sizeof(nu));
        }
        slot[top.second].push_back(p);
      }
      load.push({top.first + np, top.second});
    }
    const Packet nop{{static_cast<uint32_t>(zero), dz | (fp64 ? 0u : dz << 16), 0u, 0u}};
    lp.matrix = interleave(slot, warps, nop);
  }

  // ---- factor and substitutions ----
  auto scheduled = [&](const Scheduler& sc) {
    LaneStream st = interleave(sc.slot, warps, sc.nop(), sc.pair, true);
    st.levels = sc.levels;
    st.level_rounds = sc.level_rounds;
    return st;
  };
  {
    // a pivot row without other entries is subtracted from no one: its column's multipliers only enter the substitution,
    // whatever their size
    std::vector<char> spreads(m, 0);
    for (int k = 0; k < ms; ++k)
      for (int l = k + 1; l < m; ++l) spreads[k] |= E(k, l) >= 0;
    std::vector<Task> tasks;
    for (int i = 0; i < m; ++i)
      for (int j = 0; j < m; ++j) {
        const int e = E(i, j);
        if (e < 0) continue;
        Task t;
        t.dst = e;
        const int lim = std::min(std::min(i, j), ms);
        for (int k = 0; k < lim; ++k)
          if (E(i, k) >= 0 && E(k, j) >= 0) t.ops.push_back({E(i, k), E(k, j)});
        if (i == j && i < ms) {
          t.flags = LP_PIVOT;
        } else if (i > j && j < ms) {
          t.flags = spreads[j] ? uint32_t(LP_LCOL) : 0u;
          t.scale = j;
        } else if (t.ops.empty()) {
          continue;  // final as assembled
        }
        tasks.push_back(std::move(t));
      }
    Scheduler sc(P, warps, zero, ms, fp64 ? 1 : 2);
    if (!tasks.empty()) sc.run(tasks, n_entries);
    lp.factor = scheduled(sc);
  }
  {
    Scheduler fw(P, warps, zero, ms, 1), bw(P, warps, zero, ms, 1);
    std::vector<Task> fwd, bwd;
    for (int i = 0; i < m; ++i) {
      Task t;
      t.dst = vec + i;
      for (int k = 0; k < std::min(i, ms); ++k)
        if (E(i, k) >= 0) t.ops.push_back({E(i, k), vec + k});
      if (!t.ops.empty()) fwd.push_back(std::move(t));
    }
    for (int i = ms - 1; i >= 0; --i) {
      Task t;
      t.dst = vec + i;
      t.scale = i;
      for (int k = i + 1; k < m; ++k)
        if (E(i, k) >= 0) t.ops.push_back({E(i, k), vec + k});
      bwd.push_back(std::move(t));
    }
    if (!fwd.empty()) fw.run(fwd, n_entries);
    if (!bwd.empty()) bw.run(bwd, n_entries);
    lp.forward = scheduled(fw);
    lp.backward = scheduled(bw);
  }
  return lp;
}

}  // namespace tchem_gb
