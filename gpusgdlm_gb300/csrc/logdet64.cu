// log|det(I - Gamma_i)| of FP64 draws (elimination.hpp, LogdetPlan).
//
// A block owns one draw: its live values are in shared memory, the levels' program
// comes from L2, and the nearly dense rest is factored in shared memory in panels of
// kW columns (LU without pivoting; the trailing update in 2 x 4 register tiles per
// lane, 16 x 16 per warp).  As the FP32 fast pass, it does not pivot: a draw with a
// multiplier above kPivotLimit, or a zero, subnormal or non-finite pivot, is appended
// to the redo list (k_lu_fallback).
//
// What bounds it: the FP64 pipe, 19 cycles per warp FMA and SM.  So the pivots are
// multiplied up (their product kept as a mantissa and an exponent) and one logarithm
// (30 FMAs) is taken per draw, reciprocals (5 FMAs) are taken once per pivot, and
// blocks are as small as the dense part allows (32 .. 512 threads): the levels' and
// columns' latencies of one draw are covered by the others on the SM.  A block takes
// its next draw from a counter: where several engines share the GPU, a block whose SM
// was held by another engine's kernel starts late and takes fewer (three engines' steps
// at m = 400 in turn: 62.3 ms a step with a fixed share per block, 56.0 ms).  10 000 draws:
// m = 400 40.6 ms (68 % of the FP64 pipe; one block per SM, so the panels' columns are
// not covered), 94.5 ms with four levels and the 224 x 224 core; m = 100 0.46 ms
// (13.0 ms); m = 200 3.3 ms.  Panels of 16 columns: 45.2 ms at m = 400.
#include <algorithm>
#include <cmath>

#include "elimination.hpp"
#include "kernels.hpp"

namespace sgdlm {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr double kPivotLimit = 8.0;  // the fast pass's limit (lu_kernels.cu)
constexpr int kW = 8;                // panel width
constexpr int kFlight = 8;           // chunks of a level in flight per warp
constexpr int kWarpsPerSm = 20;      // registers for so many warps per SM (96 per thread)

// A product of many factors: mant in [1, 2) times 2^exp2 (exact scaling).
struct Product {
  double mant = 1.0;
  int exp2 = 0;
  // false: v is zero, subnormal or not finite
  __device__ __forceinline__ bool mul(double v) {
    mant *= fabs(v);
    return norm() && fabs(v) <= 1.7e308;
  }
  __device__ __forceinline__ bool norm() {
    const int hi = __double2hiint(mant), e = (hi >> 20) & 0x7FF;
    exp2 += e - 1023;
    mant = __hiloint2double((hi & 0x000FFFFF) | 0x3FF00000, __double2loint(mant));
    return e != 0 && e != 0x7FF;
  }
};

template <int NT> __device__ __forceinline__ void group_sync() {
  if constexpr (NT == 32)
    __syncwarp();
  else
    __syncthreads();
}
__device__ __forceinline__ int lo16(unsigned w) { return (int)(w & 0xFFFFu); }
__device__ __forceinline__ int hi16(unsigned w) { return (int)(w >> 16); }

// One warp's 16 x 16 tile of A22 -= L21 U12: this lane's rows ra, ra + 8 and columns
// ca + 4y.
template <bool Full>
__device__ __forceinline__ void tile_update(double *M, int ld, int k0, int ra, int ca, int nc, int nr,
                                            int ncol) {
  int rb[2], cb[4];
#pragma unroll
  for (int x = 0; x < 2; ++x) rb[x] = Full ? ra + 8 * x : min(ra + 8 * x, nc - 1);
#pragma unroll
  for (int y = 0; y < 4; ++y) cb[y] = ld * (Full ? ca + 4 * y : min(ca + 4 * y, nc - 1));
  double acc[2][4];
#pragma unroll
  for (int x = 0; x < 2; ++x)
#pragma unroll
    for (int y = 0; y < 4; ++y) acc[x][y] = M[rb[x] + cb[y]];
#pragma unroll
  for (int k = 0; k < kW; ++k) {
    double l[2], u[4];
#pragma unroll
    for (int x = 0; x < 2; ++x) l[x] = M[rb[x] + ld * (k0 + k)];
#pragma unroll
    for (int y = 0; y < 4; ++y) u[y] = M[k0 + k + cb[y]];
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
      for (int y = 0; y < 4; ++y)
        if (Full || (8 * x < nr && 4 * y < ncol)) acc[x][y] = fma(-l[x], u[y], acc[x][y]);
  }
#pragma unroll
  for (int x = 0; x < 2; ++x)
#pragma unroll
    for (int y = 0; y < 4; ++y)
      if (Full || (ra + 8 * x < nc && ca + 4 * y < nc)) M[rb[x] + cb[y]] = acc[x][y];
}

template <int NT>
__global__ void __launch_bounds__(NT, NT == 512 ? 1 : kWarpsPerSm * 32 / NT)
    k_logdet64(long n, LogdetPlan pl, int m_at, const double *__restrict__ theta_g,
               double *__restrict__ slabs, size_t slab_elems, double *__restrict__ logdet,
               int *__restrict__ draw_flags, int *__restrict__ pivot_list, int *__restrict__ next) {
  constexpr int NW = NT / 32;
  extern __shared__ __align__(16) double vals[];  // the slots, and the dense part M at m_at
  __shared__ double prow[2][kW + 1];               // a panel's pivot row (kW: its reciprocal)
  __shared__ double red_m[NW];
  __shared__ int red_e[NW], red_b[NW];
  __shared__ unsigned s_next;                      // the block's next draw
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nc = pl.core_n, ld = pl.ld, cells = ld * nc;
  for (long i = blockIdx.x; i < n;) {
    bool bad = false;
    Product prod;
    // ---- the draw's values
    if (tid == 0) {
      vals[kSlotZero] = 0.0;
      s_next = gridDim.x + (unsigned)atomicAdd(next, 1);
    }
    for (int r = tid; r < pl.m; r += NT) vals[pl.diag_slot[r]] = 1.0;
    const double *th = theta_g + (size_t)i * pl.nnz0;
    for (int q = tid; q < pl.nnz0; q += NT) vals[pl.l0_slot[q]] = -th[q];
    group_sync<NT>();
    // ---- levels
    for (int lev = 0; lev < pl.nlev; ++lev) {
      for (int q = pl.lev_piv[lev] + tid; q < pl.lev_piv[lev + 1]; q += NT) {
        const int sl = pl.piv[q];
        const double pv = vals[sl];
        if (!prod.mul(pv)) bad = true;
        vals[sl] = 1.0 / pv;
      }
      group_sync<NT>();
      for (int q = pl.lev_scale[lev] + tid; q < pl.lev_scale[lev + 1]; q += NT) {
        const unsigned w = pl.scale[q];
        const double l = vals[lo16(w)] * vals[hi16(w)];
        if (!(fabs(l) <= kPivotLimit)) bad = true;
        vals[lo16(w)] = l;
      }
      group_sync<NT>();
      // new entries: warp w takes chunks c_begin + w + NW i, kFlight in flight (the
      // plan's words come from L2)
      const int c_end = pl.lev_chunk[lev + 1];
      for (int c0 = pl.lev_chunk[lev] + warp; c0 < c_end; c0 += NW * kFlight) {
        unsigned e[kFlight], w0[kFlight];
        int toff[kFlight], K[kFlight];
#pragma unroll
        for (int h = 0; h < kFlight; ++h) {
          const int ch = c0 + h * NW;
          const bool ok = ch < c_end;
          e[h] = ok ? __ldg(pl.ent + (size_t)ch * 32 + lane) : kSlotNone;
          const int t0 = ok ? __ldg(pl.chunk_tofs + ch) : 0, t1 = ok ? __ldg(pl.chunk_tofs + ch + 1) : 0;
          K[h] = (t1 - t0) >> 5;
          toff[h] = t0 + lane;
        }
#pragma unroll
        for (int h = 0; h < kFlight; ++h) w0[h] = K[h] > 0 ? __ldg(pl.terms + toff[h]) : 0u;
        double v[kFlight];
        int Kmax = 0;
#pragma unroll
        for (int h = 0; h < kFlight; ++h) {
          if (K[h] > 0) v[h] = fma(-vals[lo16(w0[h])], vals[hi16(w0[h])], vals[hi16(e[h])]);
          Kmax = max(Kmax, K[h]);
        }
#pragma unroll 1
        for (int k = 1; k < Kmax; ++k) {
          unsigned w[kFlight];
#pragma unroll
          for (int h = 0; h < kFlight; ++h) w[h] = (k < K[h]) ? __ldg(pl.terms + toff[h] + 32 * k) : 0u;
#pragma unroll
          for (int h = 0; h < kFlight; ++h)
            if (k < K[h]) v[h] = fma(-vals[lo16(w[h])], vals[hi16(w[h])], v[h]);
        }
#pragma unroll
        for (int h = 0; h < kFlight; ++h)
          if ((unsigned)lo16(e[h]) != kSlotNone) vals[lo16(e[h])] = v[h];
      }
      group_sync<NT>();
    }
    // ---- the dense part M: after the slots, or (slab_elems > 0: no room) in their
    // place by way of the block's slab in global memory (L2)
    double *M = vals + m_at;
    if (slab_elems == 0) {
#pragma unroll 4
      for (int c = tid; c < cells; c += NT) M[c] = vals[pl.core_map[c]];
    } else {
      double *slab = slabs + (size_t)blockIdx.x * slab_elems;
#pragma unroll 4
      for (int c = tid; c < cells; c += NT) slab[c] = vals[pl.core_map[c]];
      group_sync<NT>();  // each thread reads back what it wrote itself
#pragma unroll 4
      for (int c = tid; c < cells; c += NT) M[c] = slab[c];
    }
    group_sync<NT>();
    // ---- LU of M
    for (int k0 = 0; k0 < nc; k0 += kW) {
      const int kw = min(kW, nc - k0), r0 = k0 + kw;
      // panel: one row per thread (nc <= NT), its kw columns in registers
      const int row = k0 + tid;
      const bool mine = row < nc;
      double a[kW];
#pragma unroll
      for (int c = 0; c < kW; ++c) a[c] = (mine && c < kw) ? M[row + ld * (k0 + c)] : 0.0;
#pragma unroll
      for (int k = 0; k < kW; ++k) {
        if (k < kw) {
          double *pr = prow[k & 1];
          if (tid == k) {
            if (!prod.mul(a[k])) bad = true;
            pr[kW] = 1.0 / a[k];
#pragma unroll
            for (int c = k + 1; c < kW; ++c) pr[c] = a[c];
          }
          group_sync<NT>();
          if (mine && tid > k) {
            const double l = a[k] * pr[kW];
            if (!(fabs(l) <= kPivotLimit)) bad = true;
            a[k] = l;
#pragma unroll
            for (int c = k + 1; c < kW; ++c) a[c] = fma(-l, pr[c], a[c]);
          }
        }
      }
      if (r0 >= nc) break;
      if (mine) {
#pragma unroll
        for (int c = 0; c < kW; ++c) M[row + ld * (k0 + c)] = a[c];  // kw = kW here
      }
      group_sync<NT>();
      // U12 = L11^-1 A12: one column per thread
      if (r0 + tid < nc) {
        double *col = M + (size_t)ld * (r0 + tid) + k0;
        double b[kW];
#pragma unroll
        for (int c = 0; c < kW; ++c) b[c] = col[c];
#pragma unroll
        for (int c = 1; c < kW; ++c) {
          double acc = b[c];
#pragma unroll
          for (int q = 0; q < c; ++q) acc = fma(-M[k0 + c + ld * (k0 + q)], b[q], acc);
          b[c] = acc;
          col[c] = acc;
        }
      }
      group_sync<NT>();
      // A22 -= L21 U12: warp tiles of 16 x 16, lane (lr, lc) rows lr + 8a, columns lc + 4b
      const int R = nc - r0, nt = (R + 15) / 16, lr = lane & 7, lc = lane >> 3;
      for (int t = warp; t < nt * nt; t += NW) {
        const int tc = t / nt, tr = t - tc * nt;
        // rows and columns of this tile; an edge tile leaves out whole 8-row and 4-column
        // groups (warp-uniform), and stores only what exists
        const int nr = min(16, R - 16 * tr), ncol = min(16, R - 16 * tc);
        const int ra = r0 + 16 * tr + lr, ca = r0 + 16 * tc + lc;
        if (nr == 16 && ncol == 16)
          tile_update<true>(M, ld, k0, ra, ca, nc, nr, ncol);
        else
          tile_update<false>(M, ld, k0, ra, ca, nc, nr, ncol);
      }
      group_sync<NT>();
    }
    // ---- the product of all pivots, one logarithm
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      prod.mant *= __shfl_xor_sync(kFull, prod.mant, o);
      prod.exp2 += __shfl_xor_sync(kFull, prod.exp2, o);
      prod.norm();
    }
    const int wbad = __any_sync(kFull, bad);
    if (lane == 0) {
      red_m[warp] = prod.mant;
      red_e[warp] = prod.exp2;
      red_b[warp] = wbad;
    }
    group_sync<NT>();
    if (tid == 0) {
      for (int w = 1; w < NW; ++w) {
        prod.mant *= red_m[w];
        prod.exp2 += red_e[w];
        prod.norm();
        bad = bad || red_b[w];
      }
      bad = bad || wbad;
      logdet[i] = fma((double)prod.exp2, 0.69314718055994530942, log(prod.mant));
      if (bad) {
        atomicOr(&draw_flags[i], DRAW_FLAG_PIVOT);
        const int q = atomicAdd(pivot_list, 1);
        if (q < n) pivot_list[1 + q] = (int)i;
      }
    }
    i = (long)s_next;
    group_sync<NT>();
  }
}

template <typename F> void with_kernel(int threads, F f) {
  switch (threads) {
    case 32: f(k_logdet64<32>); break;
    case 64: f(k_logdet64<64>); break;
    case 128: f(k_logdet64<128>); break;
    case 256: f(k_logdet64<256>); break;
    default: f(k_logdet64<512>); break;
  }
}

}  // namespace

int logdet64_max_slots() { return (227 * 1024 - 1024) / (int)sizeof(double); }

Logdet64Launch plan_logdet64_launch(const LogdetPlan &pl, long n, int num_sms, int max_grid) {
  Logdet64Launch L{};
  // one thread per dense row; a draw that fills an SM's shared memory alone takes 512
  // threads (more of the levels' words in flight)
  const size_t cells = (size_t)pl.ld * pl.core_n, one = sizeof(double) * std::max<size_t>(pl.nv, cells);
  L.threads = 32;
  while (L.threads < 512 && L.threads < pl.core_n) L.threads *= 2;
  if (one > 113 * 1024) L.threads = 512;
  // the dense part beside the slots while that leaves the blocks that the registers
  // allow, else in their place
  const size_t both = sizeof(double) * (pl.nv + cells);
  const bool beside = both * (size_t)(kWarpsPerSm * 32 / L.threads + 1) <= 227 * 1024;
  L.smem = beside ? both : one;
  L.m_at = beside ? pl.nv : 0;
  L.slab_elems = beside ? 0 : cells;
  if (pl.core_n > L.threads) return L;
  int per_sm = 0;
  cudaError_t e = cudaSuccess;
  with_kernel(L.threads, [&](auto kernel) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L.smem);
    if (e == cudaSuccess)
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, L.threads, L.smem);
  });
  if (e != cudaSuccess || per_sm < 1) {
    (void)cudaGetLastError();
    return L;
  }
  long grid = (long)num_sms * per_sm;
  if (max_grid > 0) grid = std::min<long>(grid, max_grid);
  L.grid = (int)std::max<long>(1, std::min<long>(grid, n));
  L.ok = 1;
  return L;
}

void launch_logdet64(cudaStream_t s, const Logdet64Launch &L, long n, const LogdetPlan &pl,
                     const double *theta_g, double *slabs, double *logdet, int *draw_flags,
                     int *pivot_list, int *next) {
  with_kernel(L.threads, [&](auto kernel) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L.smem);
    kernel<<<L.grid, L.threads, L.smem, s>>>(n, pl, L.m_at, theta_g, slabs, L.slab_elems, logdet,
                                             draw_flags, pivot_list, next);
  });
}

}  // namespace sgdlm
