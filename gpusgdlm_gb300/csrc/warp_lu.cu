// LU of (I - Gamma_i) for small systems (m <= 32): G = 4, 8, 16 or 32 lanes per draw.
//
// The block LU kernels give a draw a whole CTA and pad its matrix to 32 x 32; at
// m = 6 (the README configuration) that is a CTA of 256 threads for a 6 x 6 matrix.
// Here G lanes own one draw (a warp holds 32 / G of them) and lane r of them one row:
// the row sits in registers (G values), the LU runs with partial pivoting (getrf
// semantics: the row with the largest |entry| of the column becomes the pivot row,
// ties to the lowest row; cublasXgetrfBatched at rSGDLM/src/SGDLM/SGDLM.cu:276-283),
// the pivot row is broadcast by shuffles, rows are never moved (each lane records the
// position of its pivot), and log|det| is the sum of log|pivot|.  No draw needs a redo.
// Forecasts solve L U y = P nu with the same factors (the forward and back
// substitutions as shuffle chains), FP32 draws refined three times with an FP64
// residual of the original rows (kept in shared memory).
//
// Bound: the FP64 pipe (19 cycles per warp instruction and SM, whatever lanes are
// active) for FP64 draws and the logarithms, else the shuffle chains' latency.  So as
// many draws as fit share a warp's instructions, the pivot search compares integer
// keys, and every lane takes its own pivot's logarithm at once.  10 000 draws,
// log|det| / forecast, us, with 32 lanes per draw, rows in local memory and a logarithm
// per step -> now: FP64 m = 3 113 / 178 -> 16 / 33, m = 8 354 / 484 -> 49 / 96, m = 16
// 752 / 994 -> 176 / 310, m = 32 1616 / 2094 -> 807 / 1262; FP32 m = 8 170 / 332 -> 16 /
// 37, m = 16 329 / 516 -> 39 / 103, m = 32 668 / 935 -> 203 / 457.
#include <algorithm>
#include <type_traits>

#include "kernels.hpp"
#include "rng.cuh"

namespace sgdlm {
namespace {

constexpr int kWarpLuThreads = 128;
constexpr int kWarpLuWarps = kWarpLuThreads / 32;
constexpr unsigned kAll = 0xffffffffu;

// f(0), f(1) .. f(N - 1) with constant arguments: the row arrays are indexed by the
// steps, and a loop the compiler leaves rolled would put them into local memory.
template <int N, int I = 0, typename F> __device__ __forceinline__ void for_steps(F f) {
  if constexpr (I < N) {
    f(std::integral_constant<int, I>{});
    for_steps<N, I + 1>(f);
  }
}

template <typename T> __device__ __forceinline__ T wabs(T v) { return v < T(0) ? -v : v; }
// |v| as an ordered integer (a NaN as infinity)
__device__ __forceinline__ int abs_key(float v) { return min(__float_as_int(v) & 0x7FFFFFFF, 0x7F800000); }
__device__ __forceinline__ long long abs_key(double v) {
  return min(__double_as_longlong(v) & 0x7FFFFFFFFFFFFFFFll, 0x7FF0000000000000ll);
}

// One lane's view of a factored draw: the factors' row (multipliers in a[c] for
// c < pos, U's row in a[c] for c >= pos), its pivot position, and the lane (within the
// draw's G) whose pivot position is k, four to a word.
template <typename T, int G> struct Factors {
  T a[G];
  int pos;
  uint32_t rows[(G + 3) / 4];
  __device__ __forceinline__ int row_of(int k) const { return (int)(rows[k >> 2] >> (8 * (k & 3)) & 0xFFu); }
};

// Solves (P^T L U) x = b; b is the lane's right-hand side entry, the result is x_lane
// (column = lane).
template <typename T, int G>
__device__ __forceinline__ T lu_solve(const Factors<T, G> &f, int m, T b) {
  const int lane = threadIdx.x & (G - 1);
  T acc = b;
  for_steps<G>([&](auto step) {
    constexpr int c = decltype(step)::value;
    if (c < m) {
      const T zc = __shfl_sync(kAll, acc, f.row_of(c), G);
      if (f.pos > c) acc -= f.a[c] * zc;
    }
  });
  T x = T(0);
  for_steps<G>([&](auto step) {
    constexpr int c = G - 1 - decltype(step)::value;
    if (c < m) {
      const T q = acc / f.a[c];  // meaningful on the lane whose pivot position is c
      const T xc = __shfl_sync(kAll, q, f.row_of(c), G);
      if (f.pos < c) acc -= f.a[c] * xc;
      if (lane == c) x = xc;
    }
  });
  return x;
}

__device__ __forceinline__ double log_pivot(float v, const double *) { return log(fabs((double)v)); }
__device__ __forceinline__ double log_pivot(double v, const double *tab) { return log_table(fabs(v), tab); }

template <typename T, int G>
__global__ void __launch_bounds__(kWarpLuThreads)
    k_lu_warp(int m, long n, GammaRows rows, const T *__restrict__ theta_g, int nnz,
              double *__restrict__ logdet, int *__restrict__ draw_flags,
              const double *__restrict__ nu, double *__restrict__ y, const double *__restrict__ tab) {
  constexpr int D = 32 / G;  // draws per warp
  __shared__ T tile[kWarpLuWarps][D][G][G + 1];  // the draws' (I - Gamma_i), row-major
  const int lane = threadIdx.x & (G - 1), d = (threadIdx.x & 31) / G, w = threadIdx.x >> 5;
  T(*M)[G + 1] = tile[w][d];
  const int e0 = lane < m ? rows.rowptr[lane] : 0, e1 = lane < m ? rows.rowptr[lane + 1] : 0;
  const long stride = (long)gridDim.x * kWarpLuWarps * D;
  for (long i0 = ((long)blockIdx.x * kWarpLuWarps + w) * D; i0 < n; i0 += stride) {
    const long i = i0 + d;
    const bool valid = i < n;  // (beyond n: the identity, nothing written)
    // ---- row `lane` of (I - Gamma_i), by way of the warp's tile
#pragma unroll
    for (int c = 0; c < G; ++c) M[lane][c] = (lane == c) ? T(1) : T(0);
    if (valid)
      for (int q = e0; q < e1; ++q) M[lane][rows.ent[q].y] = -theta_g[(size_t)i * nnz + q];
    Factors<T, G> f;
#pragma unroll
    for (int c = 0; c < G; ++c) f.a[c] = M[lane][c];
#pragma unroll
    for (int q = 0; q < (G + 3) / 4; ++q) f.rows[q] = 0u;
    // ---- LU with partial pivoting, rows in place
    bool done = lane >= m;
    f.pos = G;
    bool singular = false;
    T pivot = T(1);
    for_steps<G>([&](auto step) {
      constexpr int k = decltype(step)::value;
      if (k < m) {
        // pivot: the active row with the largest |a[k]| (a NaN counts as infinity, and
        // then fails the finiteness check below)
        auto key = abs_key(f.a[k]);
        if (done) key = -1;
        int li = lane;
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) {
          const auto ok = __shfl_xor_sync(kAll, key, o, G);
          const int oi = __shfl_xor_sync(kAll, li, o, G);
          if (ok > key || (ok == key && oi < li)) {
            key = ok;
            li = oi;
          }
        }
        const T pv = __shfl_sync(kAll, f.a[k], li, G);
        if (!(key > 0) || !(wabs(pv) <= T(3.0e38))) singular = true;
        f.rows[k >> 2] |= (uint32_t)li << (8 * (k & 3));
        const bool upd = !done && lane != li;
        if (lane == li) {
          done = true;
          f.pos = k;
          pivot = pv;
        }
        const T l = upd ? f.a[k] / pv : T(0);
        if (upd) f.a[k] = l;
#pragma unroll
        for (int c = k + 1; c < G; ++c) {
          if (c < m) {
            const T u = __shfl_sync(kAll, f.a[c], li, G);
            if (upd) f.a[c] -= l * u;
          }
        }
      }
    });
    // log|det|: every lane its own pivot's logarithm, added in pivot order
    const double lg = log_pivot(pivot, tab);
    double ld = 0.0;
#pragma unroll
    for (int k = 0; k < G; ++k)
      if (k < m) ld += __shfl_sync(kAll, lg, f.row_of(k), G);
    if (valid && lane == 0) {
      logdet[i] = singular ? -INFINITY : ld;
      if (singular) atomicOr(&draw_flags[i], DRAW_FLAG_SINGULAR);
    }
    if (y) {
      const double nur = valid && lane < m ? nu[(size_t)lane * n + i] : 0.0;
      const T x = lu_solve<T, G>(f, m, (T)nur);
      double yr = (double)x;
      // FP32 factors: three refinements with the FP64 residual nu - (I - Gamma) y
      // (y accumulated in FP64)
      constexpr int kRefine = sizeof(T) == 4 ? 3 : 0;
#pragma unroll 1
      for (int it = 0; it < kRefine; ++it) {
        double res = nur;
#pragma unroll
        for (int c = 0; c < G; ++c) {
          const double yc = __shfl_sync(kAll, yr, c, G);
          if (c < m && lane < m) res -= (double)M[lane][c] * yc;
        }
        yr += (double)lu_solve<T, G>(f, m, (T)res);
      }
      if (valid && lane < m) y[(size_t)i * m + lane] = singular ? (double)NAN : yr;
    }
    __syncwarp();
  }
}

}  // namespace

template <typename T>
void launch_lu_warp(cudaStream_t s, int m, long n, int num_sms, GammaRows rows, const T *theta_g,
                    int nnz, double *logdet, int *draw_flags, const double *nu, double *y,
                    const double *tab) {
  auto run = [&](auto kernel, int lanes) {
    const long per_block = (long)kWarpLuWarps * (32 / lanes);
    const long blocks = std::max<long>(1, std::min<long>((n + per_block - 1) / per_block, (long)num_sms * 16));
    kernel<<<(unsigned)blocks, kWarpLuThreads, 0, s>>>(m, n, rows, theta_g, nnz, logdet, draw_flags, nu, y,
                                                       tab);
  };
  if (m <= 4)
    run(k_lu_warp<T, 4>, 4);
  else if (m <= 8)
    run(k_lu_warp<T, 8>, 8);
  else if (m <= 16)
    run(k_lu_warp<T, 16>, 16);
  else
    run(k_lu_warp<T, 32>, 32);
}

template void launch_lu_warp<float>(cudaStream_t, int, long, int, GammaRows, const float *, int, double *,
                                    int *, const double *, double *, const double *);
template void launch_lu_warp<double>(cudaStream_t, int, long, int, GammaRows, const double *, int, double *,
                                     int *, const double *, double *, const double *);

}  // namespace sgdlm
