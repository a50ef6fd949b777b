// Host-side planning of the sparse pre-elimination (see elimination.hpp).
#include <algorithm>
#include <map>
#include <utility>

#include "elimination.hpp"

namespace sgdlm {

namespace {
// Stop when a level would eliminate fewer than this share of the active nodes.
constexpr double kMinLevelShare = 0.05;
}  // namespace

std::vector<int> gamma_order(int m, int P, const std::vector<unsigned> &sp) {
  const size_t mm = (size_t)m * m;
  std::vector<int> order;
  for (int e = 0; e < m * P; ++e)
    if ((size_t)sp[e] < mm) order.push_back(e);
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
    return sp[a] % (unsigned)m < sp[b] % (unsigned)m;
  });
  return order;
}

EliminationPlanHost plan_elimination(int m, int P, const std::vector<unsigned> &sp,
                                     int max_levels) {
  EliminationPlanHost pl;
  pl.m = m;
  pl.P = P;
  // current pattern: row r -> (col -> slot), col c -> (row -> slot)
  std::vector<std::map<int, int>> rows(m), cols(m);
  std::vector<int> diag(m);
  for (int r = 0; r < m; ++r) diag[r] = (int)kSlotDiag0 + r;
  int nv = (int)kSlotDiag0 + m;
  for (int e : gamma_order(m, P, sp)) {
    const unsigned pos = sp[e];
    const int r = (int)(pos % (unsigned)m), c = (int)(pos / (unsigned)m);
    rows[r][c] = nv;
    cols[c][r] = nv;
    pl.l0_e.push_back(e);
    ++nv;
  }
  pl.lev_piv.push_back(0);
  pl.lev_scale.push_back(0);
  pl.lev_chunk.push_back(0);
  pl.chunk_tofs.push_back(0);
  pl.lev_fwd_nodes.push_back(0);
  pl.fwd_ptr.push_back(0);
  pl.lev_bwd_nodes.push_back(0);
  pl.bwd_ptr.push_back(0);
  std::vector<char> active(m, 1);
  int n_active = m;
  // slot indices and node numbers are stored in 16 bits
  if (nv > kMaxSlots || m > 0xFFFF) max_levels = 0;

  for (int lev = 0; lev < max_levels; ++lev) {
    // greedy independent set, ascending degree in the symmetrised active graph
    std::vector<std::pair<int, int>> order;
    order.reserve(n_active);
    for (int r = 0; r < m; ++r) {
      if (!active[r]) continue;
      int d = 0;
      for (auto &kv : rows[r]) d += active[kv.first] ? 1 : 0;
      for (auto &kv : cols[r]) d += active[kv.first] ? 1 : 0;
      order.emplace_back(d, r);
    }
    std::sort(order.begin(), order.end());
    std::vector<char> blocked(m, 0), inS(m, 0);
    std::vector<int> S;
    for (auto &dr : order) {
      const int r = dr.second;
      if (blocked[r]) continue;
      S.push_back(r);
      inS[r] = 1;
      blocked[r] = 1;
      for (auto &kv : rows[r]) blocked[kv.first] = 1;
      for (auto &kv : cols[r]) blocked[kv.first] = 1;
    }
    if ((int)S.size() == n_active) S.pop_back();  // keep a non-empty dense core
    if (S.empty() || (double)S.size() < kMinLevelShare * n_active) break;
    std::sort(S.begin(), S.end());
    auto keep = [&](int v) { return active[v] && !inS[v]; };
    // terms of the updated entries, in a deterministic order
    std::map<std::pair<int, int>, std::vector<unsigned>> acc;
    for (int t : S)
      for (auto &rq : cols[t]) {
        if (!keep(rq.first)) continue;
        for (auto &cq : rows[t])
          if (keep(cq.first))
            acc[{rq.first, cq.first}].push_back(pack16((unsigned)rq.second, (unsigned)cq.second));
      }
    int fill = 0;
    for (auto &kv : acc) {
      const int r = kv.first.first, c = kv.first.second;
      if (r != c && !rows[r].count(c)) ++fill;
    }
    if (nv + fill > kMaxSlots) break;  // the slots would not fit 16 bits

    for (int t : S) pl.piv.push_back(diag[t]);
    for (int t : S)
      for (auto &rq : cols[t])
        if (keep(rq.first)) pl.scale.push_back(pack16((unsigned)rq.second, (unsigned)diag[t]));
    // forward program, grouped by the updated node
    std::map<int, std::vector<unsigned>> fwd_by_row;
    for (int t : S)
      for (auto &rq : cols[t])
        if (keep(rq.first)) fwd_by_row[rq.first].push_back(pack16((unsigned)rq.second, (unsigned)t));
    for (auto &kv : fwd_by_row) {
      pl.fwd_node.push_back(kv.first);
      for (unsigned f : kv.second) pl.fwd.push_back(f);
      pl.fwd_ptr.push_back((int)pl.fwd.size());
    }
    for (int t : S) {
      pl.bwd_node.push_back(t);
      pl.bwd_diag.push_back(diag[t]);
      for (auto &cq : rows[t])
        if (keep(cq.first)) pl.bwd.push_back(pack16((unsigned)cq.second, (unsigned)cq.first));
      pl.bwd_ptr.push_back((int)pl.bwd.size());
    }
    // entries: updated in place, or a fresh slot for fill-in (base = constant 0)
    struct Entry {
      unsigned out, base;
      const std::vector<unsigned> *terms;
    };
    std::vector<Entry> ents;
    ents.reserve(acc.size());
    for (auto &kv : acc) {
      const int r = kv.first.first, c = kv.first.second;
      int slot;
      unsigned base;
      if (r == c) {
        slot = diag[r];
        base = (unsigned)slot;
      } else {
        auto it = rows[r].find(c);
        if (it != rows[r].end()) {
          slot = it->second;
          base = (unsigned)slot;
        } else {
          slot = nv++;
          base = kSlotZero;
          rows[r][c] = slot;
          cols[c][r] = slot;
        }
      }
      ents.push_back(Entry{(unsigned)slot, base, &kv.second});
      pl.n_terms += kv.second.size();
    }
    // chunks of 32 lanes with similar term counts
    std::stable_sort(ents.begin(), ents.end(), [](const Entry &a, const Entry &b) {
      return a.terms->size() > b.terms->size();
    });
    for (size_t c0 = 0; c0 < ents.size(); c0 += 32) {
      size_t K = 0;
      for (size_t l = 0; l < 32 && c0 + l < ents.size(); ++l) K = std::max(K, ents[c0 + l].terms->size());
      const size_t tofs = pl.terms.size();
      pl.terms.resize(tofs + 32 * K, pack16(kSlotZero, kSlotZero));
      for (size_t l = 0; l < 32; ++l) {
        if (c0 + l < ents.size()) {
          const Entry &e = ents[c0 + l];
          pl.ent.push_back(pack16(e.out, e.base));
          for (size_t k = 0; k < e.terms->size(); ++k) pl.terms[tofs + 32 * k + l] = (*e.terms)[k];
        } else {
          pl.ent.push_back(pack16(kSlotNone, kSlotZero));
        }
      }
      pl.chunk_tofs.push_back((int)pl.terms.size());
    }
    for (int t : S) {
      active[t] = 0;
      --n_active;
    }
    pl.lev_piv.push_back((int)pl.piv.size());
    pl.lev_scale.push_back((int)pl.scale.size());
    pl.lev_chunk.push_back((int)pl.chunk_tofs.size() - 1);
    pl.lev_fwd_nodes.push_back((int)pl.fwd_node.size());
    pl.lev_bwd_nodes.push_back((int)pl.bwd_node.size());
    ++pl.nlev;
  }
  pl.nv = nv;
  pl.node_core.assign(m, -1);
  for (int r = 0; r < m; ++r)
    if (active[r]) {
      pl.node_core[r] = (int)pl.core_node.size();
      pl.core_node.push_back(r);
    }
  pl.core_n = (int)pl.core_node.size();
  pl.dp = std::max(32, (pl.core_n + 31) / 32 * 32);
  // renumber the slots: the constants, then the values the solve programs read,
  // then the rest (so that a solve needs only a prefix of the slot array)
  std::vector<int> remap(nv, -1);
  int next = 0;
  remap[kSlotZero] = next++;
  remap[kSlotOne] = next++;
  auto take = [&](int slot) {
    if (remap[slot] < 0) remap[slot] = next++;
  };
  for (unsigned f : pl.fwd) take((int)(f & 0xFFFFu));
  for (unsigned b : pl.bwd) take((int)(b & 0xFFFFu));
  for (int d : pl.bwd_diag) take(d);
  pl.n_solve = next;
  for (int v = 0; v < nv; ++v) take(v);
  auto lo_map = [&](unsigned w) { return pack16((unsigned)remap[w & 0xFFFFu], w >> 16); };
  auto both_map = [&](unsigned w) {
    return pack16((unsigned)remap[w & 0xFFFFu], (unsigned)remap[w >> 16]);
  };
  pl.diag_slot.resize(m);
  for (int r = 0; r < m; ++r) pl.diag_slot[r] = remap[(int)kSlotDiag0 + r];
  pl.l0_slot.resize(pl.l0_e.size());
  for (size_t k = 0; k < pl.l0_e.size(); ++k) pl.l0_slot[k] = remap[(int)kSlotDiag0 + m + (int)k];
  for (int &v : pl.piv) v = remap[v];
  for (unsigned &w : pl.scale) w = both_map(w);
  for (unsigned &w : pl.ent) {
    const unsigned out = w & 0xFFFFu;
    w = pack16(out == kSlotNone ? kSlotNone : (unsigned)remap[out], (unsigned)remap[w >> 16]);
  }
  for (unsigned &w : pl.terms) w = both_map(w);
  for (unsigned &w : pl.fwd) w = lo_map(w);
  for (unsigned &w : pl.bwd) w = lo_map(w);
  for (int &v : pl.bwd_diag) v = remap[v];
  for (int &v : diag) v = remap[v];
  for (int r = 0; r < m; ++r)
    for (auto &kv : rows[r]) kv.second = remap[kv.second];
  if (pl.nlev > 0) {
    const size_t dp = (size_t)pl.dp;
    pl.core_map.assign(dp * dp, (uint16_t)kSlotZero);
    for (int r : pl.core_node) {
      const int pr = pl.node_core[r];
      pl.core_map[pr + dp * pr] = (uint16_t)diag[r];
      for (auto &cq : rows[r])
        if (active[cq.first]) pl.core_map[pr + dp * pl.node_core[cq.first]] = (uint16_t)cq.second;
    }
    for (size_t pr = pl.core_n; pr < dp; ++pr) pl.core_map[pr + dp * pr] = (uint16_t)kSlotOne;
  }
  return pl;
}

LevelStreamHost level_stream(const EliminationPlanHost &pl, int lanes) {
  LevelStreamHost st;
  auto add_rows = [&](size_t n) {
    st.rows.resize(st.rows.size() + n * (size_t)lanes * 2, 0u);
    return st.rows.size() - n * (size_t)lanes * 2;
  };
  for (int l = 0; l < pl.nlev; ++l) {
    const int p0 = pl.lev_piv[l], np = pl.lev_piv[l + 1] - p0;
    const int s0 = pl.lev_scale[l], ns = pl.lev_scale[l + 1] - s0;
    const int first = (std::max(np, ns) + lanes - 1) / lanes;
    const size_t at = add_rows(first);
    for (int q = 0; q < np; ++q) st.rows[at + 2 * (size_t)q] = (unsigned)pl.piv[p0 + q];
    for (int q = 0; q < ns; ++q) st.rows[at + 2 * (size_t)q + 1] = pl.scale[s0 + q];
    st.n_first.push_back(first);
    // the level's entries, by decreasing term count: entry e on thread e % lanes, pass
    // after pass over those that have a k-th term
    std::vector<unsigned> ent, terms;  // entry e's terms: first_term[e] .. first_term[e + 1]
    std::vector<int> first_term;
    for (int ch = pl.lev_chunk[l]; ch < pl.lev_chunk[l + 1]; ++ch)
      for (int lane = 0; lane < 32; ++lane) {
        const unsigned e = pl.ent[(size_t)ch * 32 + lane];
        if ((e & 0xFFFFu) == kSlotNone) continue;
        ent.push_back(e);
        first_term.push_back((int)terms.size());
        for (int k = pl.chunk_tofs[ch]; k < pl.chunk_tofs[ch + 1]; k += 32)
          if (pl.terms[k + lane] != pack16(kSlotZero, kSlotZero)) terms.push_back(pl.terms[k + lane]);
      }
    first_term.push_back((int)terms.size());
    int second = 0;
    for (size_t k = 0;; ++k) {
      size_t n = 0;
      while (n < ent.size() && (size_t)(first_term[n + 1] - first_term[n]) > k) ++n;  // (decreasing term counts)
      if (n == 0) break;
      const int rows = (int)((n + lanes - 1) / lanes);
      const size_t a = add_rows(rows);
      for (size_t e = 0; e < n; ++e) {
        const unsigned out = ent[e] & 0xFFFFu;
        st.rows[a + 2 * e] = k == 0 ? ent[e] : pack16(out, out);
        st.rows[a + 2 * e + 1] = terms[first_term[e] + k];
      }
      second += rows;
    }
    st.n_second.push_back(second);
  }
  add_rows(kStreamAhead);
  return st;
}

namespace {
// A level takes the independent nodes whose Markowitz cost is at most kCostFactor
// times the smallest one plus kCostSlack (more per level: fewer levels and barriers,
// more fill); levels end once kDenseShare of the remaining cells are non-zero (from
// there on rank-8 updates in registers are cheaper per term than the indexed terms).
// 10 000 draws, ms at m = 400 / 200 / 100 (17 / 12 / 10 parents at most): share 0.7:
// 41.5 / 3.80 / 0.62, 0.85: 42.3 / 3.86 / 0.62, 0.95: 40.9 / 3.56 / 0.47; slack 16:
// 40.7 / 3.33 / 0.46; factor 1.5: 43.4 / 3.98 / 0.63, 4: 43.7 / 3.54 / 0.46.
constexpr double kCostFactor = 2.5;
constexpr int kCostSlack = 16;
// Beyond that share they go on only until the dense part fits the slots' space.
constexpr double kDenseShare = 0.95;
constexpr size_t kMaxTermWords = 1u << 19;
}  // namespace

LogdetPlanHost plan_logdet(int m, int P, const std::vector<unsigned> &sp, int max_slots) {
  LogdetPlanHost pl;
  pl.m = m;
  const size_t mm = (size_t)m * m;
  std::vector<int> slot(mm, -1), entry(mm, -1);  // of cell (r, c) at r + m c
  auto at = [&](int r, int c) -> size_t { return (size_t)r + (size_t)m * c; };
  std::vector<std::vector<int>> rows(m), cols(m);  // active off-diagonal columns / rows
  int nv = 1;  // slot 0: constant 0
  for (int r = 0; r < m; ++r) pl.diag_slot.push_back(slot[at(r, r)] = nv++);
  size_t nz = (size_t)m;
  for (int e : gamma_order(m, P, sp)) {
    const unsigned pos = sp[e];
    const int r = (int)(pos % (unsigned)m), c = (int)(pos / (unsigned)m);
    pl.l0_slot.push_back(slot[at(r, c)] = nv++);
    rows[r].push_back(c);
    cols[c].push_back(r);
    ++nz;
  }
  std::vector<int> active(m), free_slots;
  for (int r = 0; r < m; ++r) active[r] = r;
  pl.lev_piv.push_back(0);
  pl.lev_scale.push_back(0);
  pl.lev_chunk.push_back(0);
  pl.chunk_tofs.push_back(0);
  std::vector<char> blocked(m), in_s(m, 0);
  auto dense_cells = [&]() { return (active.size() | 1) * active.size(); };
  while (active.size() > 1 && (dense_cells() > (size_t)max_slots ||
                               (double)nz < kDenseShare * (double)active.size() * active.size())) {
    std::vector<std::pair<long, int>> order;
    for (int v : active) order.emplace_back((long)rows[v].size() * (long)cols[v].size(), v);
    std::sort(order.begin(), order.end());
    const double limit = kCostFactor * (double)order[0].first + kCostSlack;
    std::fill(blocked.begin(), blocked.end(), 0);
    std::vector<int> S;
    for (auto &cv : order) {
      if ((double)cv.first > limit || S.size() + 1 == active.size()) break;
      const int v = cv.second;
      if (blocked[v]) continue;
      S.push_back(v);
      in_s[v] = 1;
      for (int u : rows[v]) blocked[u] = 1;
      for (int u : cols[v]) blocked[u] = 1;
    }
    std::sort(S.begin(), S.end());
    // the updated cells and their terms, in order of first use
    struct Term {
      int entry;
      unsigned word;
    };
    std::vector<Term> list;
    std::vector<size_t> cell;   // of each entry
    std::vector<int> count;
    std::vector<unsigned> base;
    for (int t : S) {
      pl.piv.push_back(slot[at(t, t)]);
      for (int r : cols[t])
        pl.scale.push_back(pack16((unsigned)slot[at(r, t)], (unsigned)slot[at(t, t)]));
      for (int r : cols[t])
        for (int c : rows[t]) {
          const size_t x = at(r, c);
          if (entry[x] < 0) {
            entry[x] = (int)cell.size();
            cell.push_back(x);
            count.push_back(0);
          }
          ++count[entry[x]];
          list.push_back(Term{entry[x], pack16((unsigned)slot[at(r, t)], (unsigned)slot[at(t, c)])});
        }
    }
    for (size_t k = 0; k < cell.size(); ++k) {
      const size_t x = cell[k];
      base.push_back(slot[x] >= 0 ? (unsigned)slot[x] : kSlotZero);
      if (slot[x] < 0) {
        if (free_slots.empty()) {
          slot[x] = nv++;
        } else {
          slot[x] = free_slots.back();
          free_slots.pop_back();
        }
        const int r = (int)(x % (size_t)m), c = (int)(x / (size_t)m);
        rows[r].push_back(c);
        cols[c].push_back(r);
        ++nz;
      }
    }
    if (nv > max_slots || nv > kMaxSlots || pl.terms.size() > kMaxTermWords) return LogdetPlanHost{};
    pl.n_terms += list.size();
    // entries by decreasing term count (stable), 32 to a chunk
    std::vector<int> ord(cell.size()), place(cell.size()), at_count(S.size() + 2, 0);
    for (int c : count) ++at_count[S.size() - (size_t)c + 1];  // (a term per pivot at most)
    for (size_t c = 1; c < at_count.size(); ++c) at_count[c] += at_count[c - 1];
    for (size_t k = 0; k < ord.size(); ++k) ord[at_count[S.size() - (size_t)count[k]]++] = (int)k;
    for (size_t c0 = 0; c0 < ord.size(); c0 += 32) {
      const size_t tofs = pl.terms.size();
      pl.terms.resize(tofs + 32 * (size_t)count[ord[c0]], pack16(kSlotZero, kSlotZero));
      for (size_t l = 0; l < 32; ++l) {
        if (c0 + l < ord.size()) {
          const int k = ord[c0 + l];
          place[k] = (int)(tofs + l);
          pl.ent.push_back(pack16((unsigned)slot[cell[k]], base[k]));
        } else {
          pl.ent.push_back(pack16(kSlotNone, kSlotZero));
        }
      }
      pl.chunk_tofs.push_back((int)pl.terms.size());
    }
    for (const Term &t : list) {
      pl.terms[place[t.entry]] = t.word;
      place[t.entry] += 32;
    }
    for (size_t x : cell) entry[x] = -1;
    // the eliminated nodes' slots are free from the next level on
    for (int t : S) {
      free_slots.push_back(slot[at(t, t)]);
      for (int r : cols[t]) {
        free_slots.push_back(slot[at(r, t)]);
        rows[r].erase(std::find(rows[r].begin(), rows[r].end(), t));
      }
      for (int c : rows[t]) {
        free_slots.push_back(slot[at(t, c)]);
        cols[c].erase(std::find(cols[c].begin(), cols[c].end(), t));
      }
      nz -= 1 + cols[t].size() + rows[t].size();
    }
    active.erase(std::remove_if(active.begin(), active.end(), [&](int v) { return in_s[v]; }),
                 active.end());
    pl.lev_piv.push_back((int)pl.piv.size());
    pl.lev_scale.push_back((int)pl.scale.size());
    pl.lev_chunk.push_back((int)pl.chunk_tofs.size() - 1);
    ++pl.nlev;
  }
  pl.nv = nv;
  pl.core_n = (int)active.size();
  pl.ld = pl.core_n | 1;
  pl.core_map.assign((size_t)pl.ld * pl.core_n, (uint16_t)kSlotZero);
  for (int c = 0; c < pl.core_n; ++c)
    for (int r = 0; r < pl.core_n; ++r) {
      const int v = slot[at(active[r], active[c])];
      if (v >= 0) pl.core_map[(size_t)r + (size_t)pl.ld * c] = (uint16_t)v;
    }
  return pl;
}

}  // namespace sgdlm
