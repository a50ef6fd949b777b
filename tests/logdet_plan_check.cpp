// Test harness: evaluates the product's plan for log|det| of FP64 draws (plan_logdet) and
// the levels as a stream of words per thread (level_stream), gpusgdlm_gb300/csrc/
// elimination.cu, in FP64 on the host, and checks that what threads do between two barriers
// does not depend on their order.
#include <cmath>
#include <set>
#include <vector>

#include "../gpusgdlm_gb300/csrc/elimination.cu"

namespace {
int lo(unsigned w) { return (int)(w & 0xFFFFu); }
int hi(unsigned w) { return (int)(w >> 16); }

// The accesses of one phase, by "thread": a slot written by one is not touched by another.
struct Phase {
  std::vector<int> writer;                    // of each slot, -1: none
  std::vector<std::pair<int, int>> readers;   // (slot, thread)
  bool ok = true;
  explicit Phase(int slots) : writer(slots, -1) {}
  void read(int slot, int thread) { readers.emplace_back(slot, thread); }
  void write(int slot, int thread) {
    if (writer[slot] >= 0 && writer[slot] != thread) ok = false;
    writer[slot] = thread;
  }
  bool sound() const {
    for (auto &r : readers)
      if (writer[r.first] >= 0 && writer[r.first] != r.second) return false;
    return ok;
  }
};

double dense_log_det(std::vector<double> &A, int n) {
  double ld = 0.0;
  for (int k = 0; k < n; ++k) {
    int p = k;
    for (int r = k + 1; r < n; ++r)
      if (std::fabs(A[r + (size_t)n * k]) > std::fabs(A[p + (size_t)n * k])) p = r;
    for (int c = 0; c < n; ++c) std::swap(A[k + (size_t)n * c], A[p + (size_t)n * c]);
    ld += std::log(std::fabs(A[k + (size_t)n * k]));
    for (int r = k + 1; r < n; ++r) {
      const double l = A[r + (size_t)n * k] / A[k + (size_t)n * k];
      for (int c = k; c < n; ++c) A[r + (size_t)n * c] -= l * A[k + (size_t)n * c];
    }
  }
  return ld;
}
std::vector<double> gamma_values(int m, int P, const std::vector<unsigned> &sp, const double *theta) {
  std::vector<double> g;
  for (int e : sgdlm::gamma_order(m, P, sp)) g.push_back(theta[e]);
  return g;
}
}  // namespace

// info: core_n (0: no plan), levels, slots, 1 if every phase is sound and every slot exists
extern "C" double logdet_plan_check(int m, int P, const unsigned *sp_, const double *theta, int max_slots,
                                    int *info) {
  const std::vector<unsigned> sp(sp_, sp_ + (size_t)m * P);
  const sgdlm::LogdetPlanHost pl = sgdlm::plan_logdet(m, P, sp, max_slots);
  info[0] = pl.core_n, info[1] = pl.nlev, info[2] = pl.nv, info[3] = 1;
  if (pl.core_n == 0) return 0.0;
  std::vector<double> v(pl.nv, NAN);
  v[sgdlm::kSlotZero] = 0.0;
  for (int r = 0; r < m; ++r) v[pl.diag_slot[r]] = 1.0;
  const std::vector<double> g = gamma_values(m, P, sp, theta);
  for (size_t q = 0; q < g.size(); ++q) v[pl.l0_slot[q]] = -g[q];
  double ld = 0.0;
  bool sound = pl.nv <= max_slots && g.size() == pl.l0_slot.size() && pl.ld % 2 == 1;
  for (int lev = 0; lev < pl.nlev; ++lev) {
    Phase a(pl.nv), b(pl.nv), c(pl.nv);
    for (int q = pl.lev_piv[lev]; q < pl.lev_piv[lev + 1]; ++q) {
      ld += std::log(std::fabs(v[pl.piv[q]]));
      v[pl.piv[q]] = 1.0 / v[pl.piv[q]];
      a.write(pl.piv[q], q);
    }
    for (int q = pl.lev_scale[lev]; q < pl.lev_scale[lev + 1]; ++q) {
      v[lo(pl.scale[q])] *= v[hi(pl.scale[q])];
      b.read(hi(pl.scale[q]), q);
      b.write(lo(pl.scale[q]), q);
    }
    const std::vector<double> old = v;
    for (int ch = pl.lev_chunk[lev]; ch < pl.lev_chunk[lev + 1]; ++ch)
      for (int l = 0; l < 32; ++l) {
        const unsigned e = pl.ent[(size_t)ch * 32 + l];
        const int thread = ch * 32 + l;
        double x = old[hi(e)];
        c.read(hi(e), thread);
        for (int t = pl.chunk_tofs[ch] + l; t < pl.chunk_tofs[ch + 1]; t += 32) {
          x -= old[lo(pl.terms[t])] * old[hi(pl.terms[t])];
          c.read(lo(pl.terms[t]), thread);
          c.read(hi(pl.terms[t]), thread);
        }
        if ((unsigned)lo(e) == sgdlm::kSlotNone) continue;
        v[lo(e)] = x;
        c.write(lo(e), thread);
      }
    sound = sound && a.sound() && b.sound() && c.sound();
  }
  const int n = pl.core_n;
  std::vector<double> A((size_t)n * n);
  for (int c = 0; c < n; ++c)
    for (int r = 0; r < n; ++r) A[r + (size_t)n * c] = v[pl.core_map[r + (size_t)pl.ld * c]];
  info[3] = sound ? 1 : 0;
  return ld + dense_log_det(A, n);
}

// The levels of plan_elimination through level_stream(lanes), thread by thread in reverse
// order; info: core_n, levels, 0, 1 if sound
extern "C" double level_stream_check(int m, int P, const unsigned *sp_, const double *theta, int levels,
                                     int lanes, int *info) {
  const std::vector<unsigned> sp(sp_, sp_ + (size_t)m * P);
  const sgdlm::EliminationPlanHost pl = sgdlm::plan_elimination(m, P, sp, levels);
  const sgdlm::LevelStreamHost st = sgdlm::level_stream(pl, lanes);
  std::vector<double> v(pl.nv, 0.0);
  v[sgdlm::kSlotOne] = 1.0;
  for (int r = 0; r < m; ++r) v[pl.diag_slot[r]] = 1.0;
  const std::vector<double> g = gamma_values(m, P, sp, theta);
  for (size_t q = 0; q < g.size(); ++q) v[pl.l0_slot[q]] = -g[q];
  double ld = 0.0;
  bool sound = (int)st.n_first.size() == pl.nlev && (int)st.n_second.size() == pl.nlev;
  size_t row = 0;
  auto word = [&](size_t r, int t, int half) { return st.rows[(r * (size_t)lanes + t) * 2 + half]; };
  for (int lev = 0; sound && lev < pl.nlev; ++lev) {
    const int np = pl.lev_piv[lev + 1] - pl.lev_piv[lev];
    sound = sound && st.n_first[lev] <= 0xFFFF && st.n_second[lev] <= 0xFFFF && np <= 0xFFFF;
    Phase a(pl.nv), b(pl.nv);
    for (int t = lanes - 1; t >= 0; --t)
      for (int r = 0; r < st.n_first[lev]; ++r) {
        const unsigned x = word(row + r, t, 0), y = word(row + r, t, 1);
        if (x) {  // the level's pivots are its first words: where the kernels put their logarithms
          sound = sound && r * lanes + t < np;
          ld += std::log(std::fabs(v[x]));
          a.read((int)x, t);
        }
        if (y) {
          v[lo(y)] /= v[hi(y)];
          a.read(hi(y), t);
          a.write(lo(y), t);
        }
      }
    row += st.n_first[lev];
    for (int t = lanes - 1; t >= 0; --t)
      for (int r = 0; r < st.n_second[lev]; ++r) {
        const unsigned x = word(row + r, t, 0), y = word(row + r, t, 1);
        if (!lo(x)) continue;
        v[lo(x)] = v[hi(x)] - v[lo(y)] * v[hi(y)];
        b.read(hi(x), t);
        b.read(lo(y), t);
        b.read(hi(y), t);
        b.write(lo(x), t);
      }
    row += st.n_second[lev];
    sound = sound && a.sound() && b.sound();
  }
  sound = sound && st.rows.size() == (row + sgdlm::kStreamAhead) * (size_t)lanes * 2;
  const int n = pl.core_n;
  std::vector<double> A((size_t)n * n, 0.0);
  if (pl.nlev > 0) {
    for (int c = 0; c < n; ++c)
      for (int r = 0; r < n; ++r) A[r + (size_t)n * c] = v[pl.core_map[r + (size_t)pl.dp * c]];
  } else {
    for (int r = 0; r < m; ++r) A[r + (size_t)n * r] = 1.0;
    for (int e = 0; e < m * P; ++e)
      if ((size_t)sp[e] < (size_t)m * m) A[sp[e] % m + (size_t)n * (sp[e] / m)] = -theta[e];
  }
  info[0] = n, info[1] = pl.nlev, info[2] = 0, info[3] = sound ? 1 : 0;
  return ld + dense_log_det(A, n);
}
