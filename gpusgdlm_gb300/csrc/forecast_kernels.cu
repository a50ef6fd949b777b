// Forecast solves y_i = (I - Gamma_i)^-1 nu_i by fixed-point (Jacobi) iteration,
// y <- nu + Gamma_i y, on the sparse Gamma_i itself.
//
// The reference factors every forecast draw's dense (I - Gamma_i) and forms its
// inverse (getrf + getri, rSGDLM/src/SGDLM/SGDLM.cu:594-617): (2/3 + 4/3) m^3
// flop per draw.  (I - Gamma_i) has at most max_p entries per row, and in the
// filtering regime the spectral radius of Gamma_i is well below one, so the
// iteration converges geometrically at O(nnz) per sweep -- a few ten thousand
// flop per draw at m = 400 instead of 10^8.  The sweeps run in FP32 (one thread
// per row holds the row's Gamma entries in registers in ELL form, the iterates are
// in shared memory); FP64 residuals r = nu - (I - Gamma_i) y, solved by the same
// iteration, correct their result:
//   FP32 draws: the sweeps from y = nu reach max|dy| <= 2^-20 max|y| within
//     kMaxSweeps, then one correction d; max|d| <= 1e-3 max|y| (the rule the
//     factorising path applies to its refinement step); y + d is written.
//   FP64 draws: y, nu and the residual's Gamma entries are FP64, and corrections
//     are added until one is, in every row, at most 2^-36 of the row's size
//     |nu_r| + sum |gamma_rq y_q| (usually the second).  The sweeps settle every row to
//     2^-20 of its size too, so a correction is right to about 2^-19 of its own and what is
//     left is below the rounding of y itself, also in series far smaller than the largest
//     (measured against max|y| alone, as FP32 draws are, a block of series 10^-8 as large
//     and slower to converge was left with errors of 10^-10 of its size, for 5 to 12 % less
//     time): the result is as good as a solve with FP64 factors.
// Any other draw (slow or no convergence: spectral radius near or above one,
// non-finite values) is appended to `list` and solved by the LU kernels
// (partial pivoting where needed).
//
// The sweeps are bound by the gathers' shared-memory wavefronts (bank conflicts: 32
// scattered 4-byte loads take about 3.5), by the barrier of each sweep and by issue slots;
// so several blocks share an SM, and some sweep while others wait.  Where it is faster
// (two_draws) a block solves NB = 2 FP32 draws at a time, their iterates side by side in
// shared memory: one gather of two floats (two 16-lane phases: about 6 wavefronts for two
// draws), one column index and one barrier per sweep serve both, with 72 registers a thread
// for two blocks on an SM.  10 000 FP32 draws at m = 400 (K = 18): 628 us (908 us one by one
// with the residual's conversions to FP64 at three FP64-rate instructions per entry; they
// are down to one).  FP64 draws, one per block: 1.5 ms, and 94.5 ms with FP64 factors.
#include <algorithm>

#include "kernels.hpp"
#include "max_sets.hpp"

namespace sgdlm {
namespace {

constexpr int kJacMaxThreads = 1024;  // one row per thread: m <= 1024
constexpr int kJacGroupThreads = 512;  // two draws per block: m <= 512 (registers)
constexpr int kJacPairThreads = 448;   // and two such blocks on an SM: m <= 448
constexpr int kMaxSweeps = 128;
// The first solve stops at max|dy| <= 2^-20 max|y|; the FP32 draws' correction,
// whose size is that of y's error, needs only 2^-10 of its own size: y + d is then
// within about 2^-30 of the solution (FP32 sweeps reach a few ulps, not further).
constexpr float kSweepTol = 9.5367431640625e-07f;   // 2^-20
constexpr float kCorrSweepTol = 9.765625e-04f;      // 2^-10
constexpr double kCorrTol = 1e-3;
constexpr int kCorrBits = 20;                         // bits a correction adds
constexpr double kDoneTol = 1.4551915228366852e-11;  // 2^-36: FP64 draws' last correction, per row
constexpr double kUnevenTol = 2.220446049250313e-16;  // 2^-52: the same where not all rows settled
constexpr int kMaxCorrections = 4;                    // FP64 draws

struct JacSmem {
  size_t yd, xa, xb, red, total;
  __host__ __device__ JacSmem(int m, int nb) {
    size_t o = 0;
    auto take = [&](size_t bytes) {
      const size_t at = o;
      o = (o + bytes + 15) & ~(size_t)15;
      return at;
    };
    yd = take((size_t)m * nb * sizeof(double));
    xa = take((size_t)m * nb * sizeof(float));
    xb = take((size_t)m * nb * sizeof(float));
    red = take(kMaxSets * 2 * (size_t)nb * sizeof(unsigned));
    total = o;
  }
};

// The NB (1 or 2) values of row r.
template <int NB> __device__ __forceinline__ void ld_row(const float *x, int r, float (&v)[NB]) {
  if constexpr (NB == 2) {
    const float2 q = reinterpret_cast<const float2 *>(x)[r];
    v[0] = q.x, v[1] = q.y;
  } else {
    v[0] = x[r];
  }
}
template <int NB> __device__ __forceinline__ void st_row(float *x, int r, const float (&v)[NB]) {
  if constexpr (NB == 2)
    reinterpret_cast<float2 *>(x)[r] = make_float2(v[0], v[1]);
  else
    x[r] = v[0];
}
template <int NB> __device__ __forceinline__ void ld_row(const double *x, int r, double (&v)[NB]) {
  if constexpr (NB == 2) {
    const double2 q = reinterpret_cast<const double2 *>(x)[r];
    v[0] = q.x, v[1] = q.y;
  } else {
    v[0] = x[r];
  }
}
template <int NB> __device__ __forceinline__ void st_row(double *x, int r, const double (&v)[NB]) {
  if constexpr (NB == 2)
    reinterpret_cast<double2 *>(x)[r] = make_double2(v[0], v[1]);
  else
    x[r] = v[0];
}

// (double)f of a finite f that is zero or a normal number, in integer instructions: the
// conversion instruction runs at the FP64 rate.
__device__ __forceinline__ double widen(float f) {
  const unsigned b = __float_as_uint(f), a = b & 0x7FFFFFFFu;
  const unsigned hi = (a >> 3) + (a ? (1023u - 127u) << 20 : 0u);
  return __hiloint2double((int)(hi | (b & 0x80000000u)), (int)(b << 29));
}
__device__ __forceinline__ bool is_tiny(float f) {  // not zero, below the normal numbers
  const unsigned a = __float_as_uint(f) & 0x7FFFFFFFu;
  return a - 1u < 0x007FFFFFu;
}

// A non-negative float as an ordered integer key; a NaN counts as infinity.
__device__ __forceinline__ unsigned key_of(float v) {
  return __float_as_uint(v == v ? fabsf(v) : INFINITY);
}
// Block-wide maxima of 2 NB keys (all zero-based): in place.  red: kMaxSets sets of 2 NB
// words, zero at first, used in turn (`set`); one barrier, and none is needed between
// two calls (max_sets.hpp).
template <int NB>
__device__ __forceinline__ void block_max(unsigned (&a)[NB], unsigned (&b)[NB], unsigned *red,
                                          int &set) {
  unsigned *cur = red + set * 2 * NB;
#pragma unroll
  for (int q = 0; q < NB; ++q) {
    const unsigned u = __reduce_max_sync(0xffffffffu, a[q]);
    const unsigned v = __reduce_max_sync(0xffffffffu, b[q]);
    if ((threadIdx.x & 31) == 0) {
      atomicMax(cur + 2 * q, u);
      atomicMax(cur + 2 * q + 1, v);
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < NB; ++q) {
    a[q] = cur[2 * q];
    b[q] = cur[2 * q + 1];
  }
  if (threadIdx.x < 2 * NB) red[set_to_clear(set) * 2 * NB + threadIdx.x] = 0u;
  set = set_after(set);
}

constexpr unsigned kTopBit = 0x80000000u;

// The thread's row in ELL form held in registers: K slots (entries beyond the row's
// length have value 0 and point at the row itself), the column indices packed two
// to a register, NB draws' values.
template <int K, int NB> struct Row {
  uint32_t col[K / 2];
  float val[NB][K];
  __device__ __forceinline__ int c(int q) const {
    return (int)((col[q >> 1] >> (16 * (q & 1))) & 0xFFFFu);
  }
};

// Sweeps x <- c + Gamma x from x = c over this thread's row r, for the draws in
// `todo` (a mask).  Returns the mask of the draws that converged (everything finite, and
// max|dx| <= tol max|x|); x receives the row's last iterate of each draw, which
// stops there while the others go on.  ROWS: a draw goes on until |dx_r| <= tol size_r in
// every row, size_r = |c_r| + sum |gamma_rq x_q| (`size`), or to the last sweep: a row whose
// terms nearly cancel in a neighbour may stay above that by the neighbour's rounding (one
// draw in 10^4); `even`: the draws whose rows have all come there.  wlen: the longest row of this warp, rounded
// up to even (warp-uniform): slots beyond it are padding in every row of the warp
// (value 0, so skipping them leaves every sum unchanged).  Ends on a barrier; xa and
// xb are free on entry and after it.
template <int K, int NB, bool ROWS>
__device__ __forceinline__ unsigned jacobi(bool mine, int r, int wlen, const Row<K, NB> &R,
                                           const float (&c)[NB], float *xa, float *xb,
                                           unsigned *red, int &set, float tol, unsigned todo,
                                           float (&x)[NB], float (&size)[NB], unsigned &even) {
  unsigned conv = 0;
  even = 0;
#pragma unroll
  for (int b = 0; b < NB; ++b) x[b] = c[b];
  if (mine) st_row<NB>(xa, r, x);
  __syncthreads();
  float *cur = xa, *nxt = xb;
  for (int it = 1; it <= kMaxSweeps && todo; ++it) {
    const bool check = (it & 3) == 0;
    float a0[NB], a1[NB], sz[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) a0[b] = c[b], a1[b] = 0.f, sz[b] = fabsf(c[b]);
#pragma unroll
    for (int q = 0; q < K; q += 2) {
      if (q >= wlen) break;
      float u[NB], v[NB];
      ld_row<NB>(cur, R.c(q), u);
      ld_row<NB>(cur, R.c(q + 1), v);
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        a0[b] = fmaf(R.val[b][q], u[b], a0[b]);
        a1[b] = fmaf(R.val[b][q + 1], v[b], a1[b]);
        if (ROWS && check) {
          sz[b] = fmaf(fabsf(R.val[b][q]), fabsf(u[b]), sz[b]);
          sz[b] = fmaf(fabsf(R.val[b][q + 1]), fabsf(v[b]), sz[b]);
        }
      }
    }
#pragma unroll
    for (int b = 0; b < NB; ++b) a0[b] = a0[b] + a1[b];
    if (mine) st_row<NB>(nxt, r, a0);
    float *t = cur;
    cur = nxt;
    nxt = t;
    unsigned dk[NB], xk[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      const bool live = mine && (todo >> b & 1);
      if (check) {
        if (ROWS) {
          // a row above its bound: the top bit (magnitudes lie below it)
          const float d = a0[b] - x[b];
          dk[b] = live ? key_of(d) | (fabsf(d) <= tol * sz[b] ? 0u : kTopBit) : 0u;
          if (live) size[b] = sz[b];
        } else {
          dk[b] = live ? key_of(a0[b] - x[b]) : 0u;
        }
        xk[b] = live ? key_of(a0[b]) : 0u;
      }
      if (live) x[b] = a0[b];
    }
    if (check) {
      block_max<NB>(dk, xk, red, set);  // also the barrier between sweeps
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        const float xmax = __uint_as_float(xk[b]);
        if (!(todo >> b & 1)) continue;
        if (!(xmax < INFINITY)) {
          todo &= ~(1u << b);
        } else if (ROWS && dk[b] < kTopBit) {
          todo &= ~(1u << b);
          conv |= 1u << b;
          even |= 1u << b;
        } else if ((!ROWS || it == kMaxSweeps) && __uint_as_float(dk[b] & ~kTopBit) <= tol * xmax) {
          todo &= ~(1u << b);
          conv |= 1u << b;
        }
      }
    } else {
      __syncthreads();
    }
  }
  return conv;
}

// FULL: one block of up to kJacMaxThreads (one draw) or kJacGroupThreads (two) per SM;
// otherwise (two draws, m <= kJacPairThreads) registers for two blocks.
template <typename T, int K, int NB, bool FULL>
__global__ void __launch_bounds__(NB > 1 ? (FULL ? kJacGroupThreads : kJacPairThreads) : kJacMaxThreads,
                                  FULL ? 1 : 2)
    k_forecast_jacobi(int m, long n, GammaRows rows, const T *__restrict__ theta_g, int nnz,
                      const double *__restrict__ nu, double *__restrict__ y,
                      double *__restrict__ logdet, int *__restrict__ list,
                      const int *__restrict__ order) {
  static_assert(NB == 1 || NB == 2, "");
  static_assert(kMaxSweeps % 4 == 0, "the last sweep is a checked one");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const JacSmem L(m, NB);
  double *yds = reinterpret_cast<double *>(smem_raw + L.yd);
  float *xa = reinterpret_cast<float *>(smem_raw + L.xa);
  float *xb = reinterpret_cast<float *>(smem_raw + L.xb);
  unsigned *red = reinterpret_cast<unsigned *>(smem_raw + L.red);
  const int tid = threadIdx.x;
  const bool mine = tid < m;
  const int r = mine ? (order ? order[tid] : tid) : 0;  // this thread's row
  Row<K, NB> R;
  const int e0 = mine ? rows.rowptr[r] : 0;
  const int len = mine ? rows.rowptr[r + 1] - e0 : 0;
  const int wlen = (__reduce_max_sync(0xffffffffu, (unsigned)len) + 1) & ~1;
#pragma unroll
  for (int q = 0; q < K; q += 2) {
    const uint32_t c0 = q < len ? (uint32_t)rows.ent[e0 + q].y : (uint32_t)r;
    const uint32_t c1 = q + 1 < len ? (uint32_t)rows.ent[e0 + q + 1].y : (uint32_t)r;
    R.col[q >> 1] = c0 | (c1 << 16);
  }
  if (tid < kMaxSets * 2 * NB) red[tid] = 0u;
  int set = 0;
  __syncthreads();
  for (long i0 = (long)blockIdx.x * NB; i0 < n; i0 += (long)gridDim.x * NB) {
    const int nd = (int)min((long)NB, n - i0);
    unsigned ok = (1u << nd) - 1u;  // the draws that are solved here (uniform)
    // the draws' Gamma entries (row r's runs of their Gamma copies) and nu
    double nud[NB], out[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      const T *th = theta_g + (size_t)(i0 + b) * nnz + e0;
#pragma unroll
      for (int q = 0; q < K; ++q) R.val[b][q] = (b < nd && q < len) ? (float)th[q] : 0.f;
      nud[b] = (mine && b < nd) ? nu[(size_t)r * n + i0 + b] : 0.0;
    }
    float c[NB], x[NB], yo[NB], size[NB] = {};
    unsigned even;
    unsigned ka[NB], kb[NB];
    if constexpr (sizeof(T) == 4) {
#pragma unroll
      for (int b = 0; b < NB; ++b) c[b] = (float)nud[b];
      ok = jacobi<K, NB, false>(mine, r, wlen, R, c, xa, xb, red, set, kSweepTol, ok, yo, size, even);
      if (ok) {
        // residual in FP64 and its correction by the same iteration.  The iterates are
        // widened once per row, the Gamma entries without the conversion instruction
        // (those of a draw that is still solved here are finite)
        double v[NB], yw[NB];
        bool tiny = false;
#pragma unroll
        for (int b = 0; b < NB; ++b) {
          yw[b] = (double)yo[b];
          v[b] = nud[b] - yw[b];
#pragma unroll
          for (int q = 0; q < K; ++q) tiny |= is_tiny(R.val[b][q]);
        }
        if (mine) st_row<NB>(yds, r, yw);
        __syncthreads();
        if (!__any_sync(0xffffffffu, tiny)) {
#pragma unroll
          for (int q = 0; q < K; ++q) {
            if (q >= wlen) break;
            double u[NB];
            ld_row<NB>(yds, R.c(q), u);
#pragma unroll
            for (int b = 0; b < NB; ++b) v[b] += widen(R.val[b][q]) * u[b];
          }
        } else {
#pragma unroll
          for (int q = 0; q < K; ++q) {
            if (q >= wlen) break;
            double u[NB];
            ld_row<NB>(yds, R.c(q), u);
#pragma unroll
            for (int b = 0; b < NB; ++b) v[b] += (double)R.val[b][q] * u[b];
          }
        }
#pragma unroll
        for (int b = 0; b < NB; ++b) c[b] = (float)v[b];
        const unsigned conv =
            jacobi<K, NB, false>(mine, r, wlen, R, c, xa, xb, red, set, kCorrSweepTol, ok, x, size, even);
#pragma unroll
        for (int b = 0; b < NB; ++b) {
          ka[b] = mine ? key_of(x[b]) : 0u;
          kb[b] = mine ? key_of(yo[b]) : 0u;
          out[b] = (double)yo[b] + (double)x[b];
        }
        block_max<NB>(ka, kb, red, set);
#pragma unroll
        for (int b = 0; b < NB; ++b) {
          const float dmax = __uint_as_float(ka[b]), ymax = __uint_as_float(kb[b]);
          if (!((conv >> b & 1) && ymax < INFINITY && dmax < INFINITY &&
                (double)dmax <= kCorrTol * (double)ymax))
            ok &= ~(1u << b);
        }
      }
    } else {
      // FP64 draws.  The system is scaled by a power of two to max|nu| in [1, 2), and
      // a correction's right-hand side by the bits gained so far, so that the FP32
      // sweeps meet values of normal range whatever the data's (powers of two: exact)
      double inv[NB];
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        ka[b] = (unsigned)__double2hiint(nud[b]) & 0x7FFFFFFFu;
        kb[b] = 0u;
      }
      block_max<NB>(ka, kb, red, set);
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        const int ex = (int)(ka[b] >> 20);  // biased exponent of the largest |nu|
        if (ex == 0x7FF) ok &= ~(1u << b);
        const int e = max(-1000, min(1000, ex - 1023));
        const bool sc = ex > 0 && ex < 0x7FF;
        inv[b] = sc ? __hiloint2double((1023 + e) << 20, 0) : 1.0;
        if (sc) nud[b] *= __hiloint2double((1023 - e) << 20, 0);
        c[b] = (float)nud[b];
      }
      ok = jacobi<K, NB, true>(mine, r, wlen, R, c, xa, xb, red, set, kSweepTol, ok, yo, size, even);
      unsigned todo = ok;
      float csize[NB] = {};  // (a correction's)
#pragma unroll
      for (int b = 0; b < NB; ++b) out[b] = (double)yo[b];
      double up = 1.0, down = 1.0;
#pragma unroll 1
      for (int it = 1; it <= kMaxCorrections && todo; ++it) {
        up *= (double)(1 << kCorrBits);
        down *= 1.0 / (double)(1 << kCorrBits);
        if (mine) st_row<NB>(yds, r, out);
        __syncthreads();
        double v[NB];
#pragma unroll
        for (int b = 0; b < NB; ++b) v[b] = nud[b] - out[b];
#pragma unroll 2
        for (int q = 0; q < len; ++q) {
          double u[NB];
          ld_row<NB>(yds, rows.ent[e0 + q].y, u);
#pragma unroll
          for (int b = 0; b < NB; ++b)
            if (b < nd) v[b] = fma((double)theta_g[(size_t)(i0 + b) * nnz + e0 + q], u[b], v[b]);
        }
#pragma unroll
        for (int b = 0; b < NB; ++b) c[b] = (float)(v[b] * up);
        const unsigned conv =
            jacobi<K, NB, true>(mine, r, wlen, R, c, xa, xb, red, set, kSweepTol, todo, x, csize, even);
        ok &= ~(todo & ~conv);
        todo &= conv;
        // the top bit of ka: a row whose correction is not yet small against its own size;
        // ka is then the largest such row's
#pragma unroll
        for (int b = 0; b < NB; ++b) {
          if (todo >> b & 1) out[b] += (double)x[b] * down;
          const float done = (float)((even >> b & 1 ? kDoneTol : kUnevenTol) * up);
          ka[b] = mine ? key_of(x[b]) | (fabsf(x[b]) <= done * size[b] ? 0u : kTopBit) : 0u;
          kb[b] = mine ? key_of((float)out[b]) : 0u;
        }
        block_max<NB>(ka, kb, red, set);
#pragma unroll
        for (int b = 0; b < NB; ++b) {
          const double dmax = (double)__uint_as_float(ka[b] & ~kTopBit) * down,
                       ymax = (double)__uint_as_float(kb[b]);
          if (!(todo >> b & 1)) continue;
          if (!(ymax < INFINITY && dmax <= kCorrTol * ymax)) {
            ok &= ~(1u << b);
            todo &= ~(1u << b);
          } else if (ka[b] < kTopBit) {
            todo &= ~(1u << b);
          }
        }
      }
      ok &= ~todo;  // corrections that do not shrink
#pragma unroll
      for (int b = 0; b < NB; ++b) out[b] *= inv[b];
    }
    if (ok) {
      // thread t writes row t: a warp's stores are one contiguous run, also when y is
      // page-locked host memory
      if (mine) st_row<NB>(yds, r, out);
      __syncthreads();
      if (mine) {
        ld_row<NB>(yds, tid, out);
#pragma unroll
        for (int b = 0; b < NB; ++b)
          if (ok >> b & 1) y[(size_t)(i0 + b) * m + tid] = out[b];
      }
    }
    if (tid < nd) {
      if (ok >> tid & 1) {
        logdet[i0 + tid] = NAN;  // no factorisation: no log|det| for this forecast draw
      } else {
        const int q = atomicAdd(list, 1);
        if (q < n) list[1 + q] = (int)(i0 + tid);
      }
    }
    __syncthreads();
  }
}

// ELL widths: the smallest of these that holds the longest row
constexpr int kJacWidths[] = {8, 12, 16, 18, 20, 24, 32};
// Two draws per block: FP32 draws, K entries per row,
//   K <= 8 (m to 448), K <= 18 (m from 385 to 448): the form for two blocks on an SM;
//   K >= 24 (m to 512): one block with 128 registers per thread;
// elsewhere one draw per block, of which the 64 registers per thread leave room for more
// blocks.  Time of two draws per block to that of one, 10 000 draws (3 000, 40 000 alike):
//   K = 8: m = 33 0.97, 64 1.09, 100 0.98, 133 0.98, 200 0.98, 300 0.91, 448 0.93, 500 1.16;
//   12: m = 64 1.16, 100 1.05, 180 1.12, 256 1.04, 300 1.09, 400 0.98, 448 0.97;
//   16: 100 1.05, 200 0.99, 300 1.06, 400 0.99, 448 1.00; 18: 250 1.08, 300 1.13, 350 1.04,
//   400 1.00, 448 1.01, 500 1.10; 20: 200 1.13, 300 1.16, 400 1.05, 448 1.09;
//   24: 200 0.97, 300 1.11, 400 0.97, 448 0.95, 500 0.98; 32: 200 0.83, 300 1.02, 400 0.87,
//   500 0.75.  FP64 draws: 1.00 to 1.27 (m = 33 .. 500, K = 8 .. 24), so one.
template <typename T> bool two_draws(int K, int threads) {
  if (sizeof(T) == 8 || threads > kJacGroupThreads) return false;
  return K >= 24 || (threads <= kJacPairThreads && (K <= 8 || (K <= 18 && threads > 384)));
}

// Calls f with the kernel of type T, width K and draws per block (group: two).
template <typename T, typename F> void with_jacobi_kernel(int K, bool group, F f) {
#define SGDLM_JACOBI(KK)                                          \
  case KK:                                                        \
    if constexpr (sizeof(T) == 4 && (KK <= 18 || KK >= 24)) {      \
      if (group) {                                                \
        f(k_forecast_jacobi<T, KK, 2, (KK >= 24)>, 2);            \
        break;                                                    \
      }                                                           \
    }                                                             \
    f(k_forecast_jacobi<T, KK, 1, true>, 1);                      \
    break
  switch (K) {
    SGDLM_JACOBI(8);
    SGDLM_JACOBI(12);
    SGDLM_JACOBI(16);
    SGDLM_JACOBI(18);
    SGDLM_JACOBI(20);
    SGDLM_JACOBI(24);
    SGDLM_JACOBI(32);
  }
#undef SGDLM_JACOBI
}

}  // namespace

template <typename T> JacobiPlan plan_jacobi(int m, int max_row, int num_sms) {
  JacobiPlan jp{};
  if (m < 1 || m > kJacMaxThreads || max_row > 32) return jp;
  jp.nnz = 32;
  for (int k : kJacWidths)
    if (max_row <= k) {
      jp.nnz = k;
      break;
    }
  jp.threads = (m + 31) / 32 * 32;
  // [0] one draw per block, [1] two
  for (int g = 0; g < 2; ++g) {
    if (g == 1 && !two_draws<T>(jp.nnz, jp.threads)) break;
    int per_sm = 0;
    cudaError_t e = cudaSuccess;
    with_jacobi_kernel<T>(jp.nnz, g == 1, [&](auto kernel, int nb) {
      jp.draws[g] = nb;
      jp.smem[g] = JacSmem(m, nb).total;
      if (jp.smem[g] > 48 * 1024)
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)jp.smem[g]);
      if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, jp.threads, jp.smem[g]);
    });
    if (e != cudaSuccess || per_sm < 1) {
      (void)cudaGetLastError();
      jp.draws[g] = 0;
      continue;
    }
    jp.grid[g] = num_sms * per_sm;
  }
  jp.ok = jp.draws[0] > 0;
  return jp;
}
template JacobiPlan plan_jacobi<float>(int, int, int);
template JacobiPlan plan_jacobi<double>(int, int, int);

template <typename T>
void launch_forecast_jacobi(cudaStream_t s, const JacobiPlan &jp, int m, long n, GammaRows rows,
                            const T *theta_g, int nnz, const double *nu, double *y,
                            double *logdet, int *list) {
  // two draws per block (where the plan has them) from two rounds of the resident blocks
  // on; fewer draws spread over more SMs one by one (m = 400, K = 18, 304 blocks: 304 draws
  // 51 us one by one, 61 us in twos; 608 74, 76; 912 96, 113; 1 216 116, 117; 2 432 205, 203)
  const int g = jp.draws[1] > 0 && n >= 2L * jp.grid[1] * jp.draws[1] ? 1 : 0;
  const long blocks = (n + jp.draws[g] - 1) / jp.draws[g];
  const unsigned grid = (unsigned)std::max<long>(std::min<long>(jp.grid[g], blocks), 1);
  with_jacobi_kernel<T>(jp.nnz, g == 1, [&](auto kernel, int) {
    if (jp.smem[g] > 48 * 1024)
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)jp.smem[g]);
    kernel<<<grid, (unsigned)jp.threads, jp.smem[g], s>>>(m, n, rows, theta_g, nnz, nu, y, logdet, list,
                                                          jp.order);
  });
}
template void launch_forecast_jacobi<float>(cudaStream_t, const JacobiPlan &, int, long, GammaRows,
                                            const float *, int, const double *, double *, double *,
                                            int *);
template void launch_forecast_jacobi<double>(cudaStream_t, const JacobiPlan &, int, long, GammaRows,
                                             const double *, int, const double *, double *, double *,
                                             int *);

}  // namespace sgdlm
