// Sparse pre-elimination of (I - Gamma) before the dense LU.
//
// (I - Gamma) has a unit diagonal and at most max_p off-diagonal entries per
// row, at the same positions for every draw.  Once per parental-set change the
// host plans a sequence of elimination levels: at each level it picks a greedy
// independent set S of the current sparsity graph (no edge between two members
// of S, so the S x S block is diagonal) and eliminates it,
//   L[r][t]  = M[r][t] / M[t][t]                       (t in S, r not in S)
//   M'[r][c] = M[r][c] - sum_{t in S} L[r][t] M[t][c],
//   log|det M| = sum_{t in S} log|M[t][t]| + log|det M'|.
// This is a symmetric permutation plus exact block elimination, so |det| is
// unchanged; what is left (the "core") goes to the dense LU.  At m = 400 with
// ~8.5 parents per series four levels shrink the dense core from 400 to about
// 210 nodes.
//
// The plan is a small program over a per-draw array of value slots `vals`.
// Every matrix position owns one slot for its whole life: an entry that a level
// updates is overwritten in place, a fill-in entry gets a fresh slot, and a
// multiplier L[r][t] replaces M[r][t] in its slot.  Slot indices fit 16 bits.
//   slot 0             constant 0 (padding terms read it; never written)
//   slot 1             constant 1 (identity padding of the dense core)
//   slots 2 .. n_solve the values the forward / backward solve programs read
//                      (rows, columns and pivots of the eliminated nodes)
//   then everything else.
// Initial values: vals[diag_slot[r]] = 1, vals[l0_slot[k]] = -theta[l0_e[k]].
// A level runs as: pivots and multipliers (scale), barrier, new entries,
// barrier.  Entries are grouped in chunks of 32 (one per warp lane), sorted by
// term count so that a chunk's lanes do the same number of terms; a chunk's
// terms are stored term-major (term k of lane l at chunk_tofs + 32 k + l) so
// that each load of the program is one coalesced 128-byte line.
#pragma once
#include <cstdint>
#include <vector>

#include <cuda_runtime.h>

namespace sgdlm {

constexpr unsigned kSlotZero = 0, kSlotOne = 1, kSlotDiag0 = 2;
constexpr unsigned kSlotNone = 0xFFFFu;  // padding lane of a chunk: no store
constexpr int kMaxSlots = 0xFFFF;        // slots 0 .. 0xFFFE
constexpr int kMaxLevels = 16;           // levels a caller may ask for

inline unsigned pack16(unsigned lo, unsigned hi) { return (lo & 0xFFFFu) | (hi << 16); }

struct EliminationPlanHost {
  int m = 0, P = 0;
  int nlev = 0;
  int nv = 0;                        // slots per draw
  int n_solve = 2;                   // slots [0, n_solve) hold what the solves read
  std::vector<int> diag_slot;        // m initial diagonal slots (value 1)
  std::vector<int> l0_e;             // theta index e (j*max_p + k) of level-0 entry
  std::vector<int> l0_slot;          // its slot (value -theta[e])
  // per level (nlev + 1 offsets each)
  std::vector<int> lev_piv;          // -> piv
  std::vector<int> piv;              // slot of M[t][t] of the eliminated nodes
  std::vector<int> lev_scale;        // -> scale
  std::vector<unsigned> scale;       // (slot M[r][t] | slot M[t][t] << 16): M[r][t] /= M[t][t]
  std::vector<int> lev_chunk;        // -> chunks
  std::vector<int> chunk_tofs;       // #chunks + 1 offsets into terms (multiples of 32)
  std::vector<unsigned> ent;         // 32 per chunk: (out slot | base slot << 16)
  std::vector<unsigned> terms;       // (slot L[r][t] | slot M[t][c] << 16)
  // forward (right-hand side) program, grouped by the updated node r:
  //   z[r] -= sum_t L[r][t] z[t]
  std::vector<int> lev_fwd_nodes;    // -> fwd_node
  std::vector<int> fwd_node;         // r
  std::vector<int> fwd_ptr;          // term ranges per node (size #nodes + 1)
  std::vector<unsigned> fwd;         // (slot L[r][t] | t << 16)
  // backward program: y[t] = (z[t] - sum_c M[t][c] y[c]) / M[t][t]
  std::vector<int> lev_bwd_nodes;    // -> bwd_node
  std::vector<int> bwd_node;         // t
  std::vector<int> bwd_diag;         // slot M[t][t]
  std::vector<int> bwd_ptr;          // term ranges per node (size #nodes + 1)
  std::vector<unsigned> bwd;         // (slot M[t][c] | c << 16)
  // dense core
  int core_n = 0;
  int dp = 0;                        // core_n rounded up to 32
  std::vector<int> core_node;        // core position -> node
  std::vector<int> node_core;        // node -> core position or -1
  std::vector<uint16_t> core_map;    // dp x dp (column-major) slot of each core cell
  size_t n_terms = 0;                // unpadded term count (for reporting)
};

// The levels' program as rows of one 8-byte word per thread of a block of `lanes`
// threads, in the order in which they are worked off, so that a thread reads its words
// one after the other, ahead of the barriers between phases:
//   first phase of a level: x = slot of a pivot (0: none), y = a multiplier (slot
//     M[r][t] | slot M[t][t] << 16; 0: none);
//   second phase: x = out slot | base slot << 16 (out 0: none), y = slot L | slot U << 16:
//     vals[out] = vals[base] - vals[L] vals[U].  An entry's further terms follow in the
//     same thread's later rows, with the entry itself as base.
// Row t of phase p of level l: rows[(sum of the counts before + t) * lanes + thread];
// kStreamAhead empty rows at the end (they are read, never used).
constexpr int kStreamAhead = 3;
struct LevelStreamHost {
  std::vector<unsigned> rows;  // x, y pairs
  std::vector<int> n_first, n_second;
};
LevelStreamHost level_stream(const EliminationPlanHost &pl, int lanes);
struct LevelStream {
  const uint2 *rows;
  // rows of each phase and pivots of each level (a level's pivots are the first words
  // of its first phase's rows)
  unsigned short n_first[kMaxLevels], n_second[kMaxLevels], n_piv[kMaxLevels];
};

// Device copy of the plan (pointers into one allocation owned by the engine).
// core_map == nullptr means "no plan": the whole matrix is the dense core.
struct EliminationPlan {
  int m, P, nlev, nv, n_solve, nnz0, core_n;
  const int *diag_slot, *l0_e, *l0_slot;
  const int *lev_piv, *piv;
  const int *lev_scale;
  const unsigned *scale;
  const int *lev_chunk, *chunk_tofs;
  const unsigned *ent, *terms;
  const int *lev_fwd_nodes, *fwd_node, *fwd_ptr;
  const unsigned *fwd;
  const int *lev_bwd_nodes, *bwd_node, *bwd_diag, *bwd_ptr;
  const unsigned *bwd;
  const int *core_node;
  const uint16_t *core_map;
  // the solve programs (lev_fwd_nodes .. bwd) are one contiguous, 16-byte aligned
  // run of prog_len ints starting at prog, so that a kernel can stage them
  const int *prog;
  int prog_len;
  // for blocks of 128 threads (k_lu_small): the levels, and the slots of the core's
  // cells (row, 4 q) .. (row, 4 q + 3), 16 bits each, at small_map[128 q + row]
  LevelStream small_stream;
  const uint2 *small_map;
  LevelStream stream;  // the levels for blocks of 256 threads (k_lu, FP32 draws, log|det|)
};

// The theta indices e = j*max_p + k of the Gamma entries (sp[e] < m*m), row of (I - Gamma)
// by row, within a row in increasing e: the order of the draw-major Gamma copy and of
// both plans' level-0 entries.
std::vector<int> gamma_order(int m, int P, const std::vector<unsigned> &sp);

// Builds the plan from the parental sets (sp: max_p x m, entries < m*m address
// (I - Gamma) at row + m*col).  max_levels = 0, or parental sets with more than
// kMaxSlots values, give no levels (the plain dense LU of the whole matrix).
EliminationPlanHost plan_elimination(int m, int P, const std::vector<unsigned> &sp,
                                     int max_levels);

// ---- log|det| of FP64 draws ---------------------------------------------------
// FP64 arithmetic is the narrow unit of this GPU (one warp FMA per 64 cycles and SM
// sub-partition, 19 per SM), so for FP64 draws the plan spends indices to save
// operations: many more levels, each a set of independent nodes of low Markowitz
// cost (row count times column count), until the remaining nodes' matrix is nearly
// dense.  At m = 400 with ~8.5 parents per series that is 1.4e6 multiply-adds per
// draw (18 levels, 154 dense nodes) instead of the 3.8e6 of four greedy levels and a
// 224 x 224 core; at m = 100, 1.1e4 instead of 9e4.  A node's slots are handed on once
// it is eliminated (only log|det| is wanted, nothing is solved), so that the live
// values stay in shared memory.
//
// A level: pivots (the slot becomes the reciprocal), multipliers, new entries, as
// above; chunks of 32 entries, terms term-major.
struct LogdetPlanHost {
  int m = 0, nlev = 0, nv = 0;      // nv: slots per draw (slot 0: constant 0)
  int core_n = 0, ld = 0;           // dense part: nodes, leading dimension (odd: bank conflicts)
  std::vector<int> diag_slot, l0_slot;
  std::vector<int> lev_piv, piv, lev_scale;
  std::vector<unsigned> scale;
  std::vector<int> lev_chunk, chunk_tofs;
  std::vector<unsigned> ent, terms;
  std::vector<uint16_t> core_map;   // ld x core_n (column-major) slot of each dense cell
  size_t n_terms = 0;
};
struct LogdetPlan {
  int m, nnz0, nlev, nv, core_n, ld;
  const int *diag_slot, *l0_slot;
  const int *lev_piv, *piv, *lev_scale;
  const unsigned *scale;
  const int *lev_chunk, *chunk_tofs;
  const unsigned *ent, *terms;
  const uint16_t *core_map;
};
// core_n = 0: more than max_slots live values, or a dense part far above that: no plan.
LogdetPlanHost plan_logdet(int m, int P, const std::vector<unsigned> &sp, int max_slots);

}  // namespace sgdlm
