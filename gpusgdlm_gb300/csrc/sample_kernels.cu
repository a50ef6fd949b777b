// Draw generation: (lambda, theta) from the per-series normal-gamma posterior or
// prior, and the multi-step evolution of forecast draws.
//
// The reference samples with four cuRAND calls into HBM caches, a Marsaglia-Tsang
// kernel with atomic slot compaction, a one-thread-per-series Cholesky and a
// pointer-array gemmBatched of batch m*n for theta = U' z
// (rSGDLM/src/SGDLM/SGDLM.cu:623-677).  Here one thread owns one (draw, series)
// pair: its normals come out of Philox in registers, U_j sits in shared memory
// (every thread of the block shares series j, so reads are broadcasts), and the
// block's theta rows are staged in shared memory so the series-major store is one
// contiguous coalesced run.  From the same staged rows the block writes its draws'
// Gamma entries to the draw-major Gamma copy (GammaDraws), which the LU and
// iterative-solve kernels read as one run per draw.
#include <type_traits>

#include "kernels.hpp"
#include "rng.cuh"

namespace sgdlm {
namespace {

constexpr int kSampleThreads = 128;

// The series' Gamma coefficients: k of the c-th entry of its row (gks[c], the k
// with a simultaneous parent, sp[j*P + k] < m*m, in increasing k), their count and
// the row's first position in the CSR order.  One whole warp: lane l tests k = l,
// l + 32 (P <= 64) and places its k by a ballot of the lanes before it.
__device__ __forceinline__ void gamma_row_of(const unsigned *__restrict__ sp, const int *rowptr,
                                             int j, int P, unsigned mm, int *gks, int *gcnt,
                                             int *gq0) {
  const int lane = threadIdx.x & 31;
  int base = 0;
  for (int k0 = 0; k0 < P; k0 += 32) {
    const int k = k0 + lane;
    const bool g = k < P && sp[(size_t)j * P + k] < mm;
    const unsigned mask = __ballot_sync(0xffffffffu, g);
    if (g) gks[base + __popc(mask & ((1u << lane) - 1u))] = k;
    base += __popc(mask);
  }
  if (lane == 0) {
    *gcnt = base;
    *gq0 = rowptr[j];
  }
}

// The block's draws i0 .. i0 + cnt - 1 of series j, staged row by row (P values
// per draw), to their Gamma runs of the draw-major copy (GammaDraws: draw i's run
// at v[i*nnz + q0 ..]).  Consecutive threads take consecutive entries, so a warp
// writes the runs of several draws at once.
template <typename T>
__device__ __forceinline__ void write_gamma_runs(const GammaDraws<T> &gd, int P, long i0, int cnt,
                                                 const T *stage, const int *gks, int gcnt,
                                                 int gq0) {
  if (gcnt == 0) return;
  // entry x = t gcnt + c of the block; from one of a thread's entries to its next without
  // a division (one per entry was a ninth of k_sample's instructions)
  const int dt = (int)blockDim.x / gcnt, dc = (int)blockDim.x - dt * gcnt;
  int t = (int)threadIdx.x / gcnt, c = (int)threadIdx.x - t * gcnt;
  T *v = gd.v + (size_t)i0 * gd.nnz + gq0;
  while (t < cnt) {
    v[(size_t)t * gd.nnz + c] = stage[t * P + gks[c]];
    t += dt;
    c += dc;
    if (c >= gcnt) {
      c -= gcnt;
      ++t;
    }
  }
}

// W values of 16 bytes (aligned).
template <typename T> struct V16 {
  static constexpr int W = (int)(16 / sizeof(T));
  __device__ static __forceinline__ void ld(const T *p, T *o) {
    const uint4 v = *reinterpret_cast<const uint4 *>(p);
    const T *t = reinterpret_cast<const T *>(&v);
#pragma unroll
    for (int b = 0; b < W; ++b) o[b] = t[b];
  }
  __device__ static __forceinline__ void st(T *p, const T *o) {
    uint4 v;
    T *t = reinterpret_cast<T *>(&v);
#pragma unroll
    for (int b = 0; b < W; ++b) t[b] = o[b];
    *reinterpret_cast<uint4 *>(p) = v;
  }
};

// sum_{l <= k} U[l + P k] z[l] in increasing l; VEC: P is a multiple of V16<T>::W, so that
// every column of U starts on 16 bytes (the padding behind l = k is read, not used).
template <typename T, bool VEC>
__device__ __forceinline__ T column_dot(const T *Us, int P, int k, const T *z) {
  constexpr int W = V16<T>::W;
  T acc = T(0);
  if constexpr (VEC) {
#pragma unroll
    for (int l = 0; l <= k; l += W) {
      T u[W];
      V16<T>::ld(Us + l + P * k, u);
#pragma unroll
      for (int b = 0; b < W; ++b)
        if (l + b <= k) acc += u[b] * z[l + b];
    }
  } else {
#pragma unroll
    for (int l = 0; l <= k; ++l) acc += Us[l + P * k] * z[l];
  }
  return acc;
}

// Both kernels: VEC (P a multiple of four FP32 or two FP64 values) reads U's columns and
// the staged rows 16 bytes at a time.  A row of P = 20 FP32 values read and written value by
// value meets four-way bank conflicts (20 l mod 32 takes eight values), as 16-byte accesses
// none; an odd P has none either way.
template <typename T, int PMAX, bool VEC>
__global__ void __launch_bounds__(kSampleThreads)
    k_sample(int m, int P, long n, const double *__restrict__ m_t,
             const double *__restrict__ n_t, const double *__restrict__ s_t,
             const T *__restrict__ U, RngKey key, T *__restrict__ lambda,
             T *__restrict__ theta, GammaDraws<T> gd, int *__restrict__ draw_flags,
             const unsigned *__restrict__ p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *Us = reinterpret_cast<T *>(smem_raw);  // P*P, U[row + P*col]
  T *ms = Us + P * P;                       // P
  T *stage = ms + P;                        // blockDim.x * P
  __shared__ GammaShape<T> shape;           // the series' gamma shape
  __shared__ T ser[2];                      // its rate, s_j
  __shared__ int gks[64], gcnt, gq0;        // its Gamma coefficients (gamma_row_of)
  const int j = blockIdx.y;
  // the series' active coefficients: U_j is zero outside its leading pj x pj
  // block (the Cholesky factor's cut), so theta_k = m_k exactly for k >= pj and
  // the normals z_l, l >= pj, are never used; they are not generated (counter-based
  // streams: the others do not move)
  const int pj = p ? min((int)p[j], P) : P;
  for (int e = threadIdx.x; e < P * P; e += blockDim.x) Us[e] = U[(size_t)j * P * P + e];
  for (int e = threadIdx.x; e < P; e += blockDim.x) ms[e] = (T)m_t[(size_t)j * P + e];
  if (gd.v && (threadIdx.x >> 5) == 1)  // warp 1 (thread 0 sets up ser)
    gamma_row_of(gd.sp, gd.rowptr, j, P, (unsigned)m * (unsigned)m, gks, &gcnt, &gq0);
  if (threadIdx.x == 0) {
    // FP64 once per series (FP64 is a narrow pipe on this GPU)
    const double nj = n_t[j], sj = s_t[j];
    shape = gamma_shape<T>((T)(0.5 * nj), false);
    ser[0] = (T)(0.5 * nj * sj);
    ser[1] = (T)sj;
  }
  __syncthreads();
  const long i0 = (long)blockIdx.x * blockDim.x;
  const long i = i0 + threadIdx.x;
  if (i < n) {
    const uint32_t ep = key_epoch(key);
    const T rate = ser[0];
    bool fail = false;
    const T lam = gamma_mt<T>(shape, (uint32_t)i, (uint32_t)j, TAG_GAMMA, ep, key.k0,
                              key.k1, key.tab, &fail) / rate;
    T z[PMAX];
#pragma unroll
    for (int q = 0; q < PMAX / 4; ++q) {
      if (4 * q < pj) {
        const U4 r = philox((uint32_t)i, (uint32_t)j, tag_sub(TAG_THETA, q), ep, key.k0, key.k1);
        box_muller<T>(r.x, r.y, z[4 * q], z[4 * q + 1], key.tab);
        if (4 * q + 2 < pj)
          box_muller<T>(r.z, r.w, z[4 * q + 2], z[4 * q + 3], key.tab);
        else
          z[4 * q + 2] = z[4 * q + 3] = T(0);
      } else {
        z[4 * q] = z[4 * q + 1] = z[4 * q + 2] = z[4 * q + 3] = T(0);
      }
    }
    // theta = m + (U' z) / sqrt(s lambda)   (makeVB_MVN, kernel_functions.cuh:72-83);
    // one reciprocal instead of P divisions (within 1-2 ulp of the quotients)
    const T rden = T(1) / dev_sqrt(ser[1] * lam);
    T *row = stage + (size_t)threadIdx.x * P;
    constexpr int W = VEC ? V16<T>::W : 1;
#pragma unroll
    for (int k = 0; k < PMAX; k += W) {
      if (k < P) {
        T o[W];
        if constexpr (VEC)
          V16<T>::ld(ms + k, o);
        else
          o[0] = ms[k];
#pragma unroll
        for (int b = 0; b < W; ++b) {
          T acc = T(0);
          if (k + b < pj) acc = column_dot<T, VEC>(Us, P, k + b, z);
          o[b] = o[b] + acc * rden;
        }
        if constexpr (VEC)
          V16<T>::st(row + k, o);
        else
          row[k] = o[0];
      }
    }
    lambda[(size_t)j * n + i] = lam;
    if (fail) atomicOr(&draw_flags[i], DRAW_FLAG_GAMMA_CAP);
  }
  __syncthreads();
  if (gd.v) write_gamma_runs<T>(gd, P, i0, (int)min((long)blockDim.x, n - i0), stage, gks, gcnt, gq0);
  const long cnt = (long)min((long)blockDim.x, n - i0) * P;
  T *dst = theta + ((size_t)j * n + i0) * P;
  if (((size_t)j * n + i0) * P * sizeof(T) % 16 == 0 && cnt * sizeof(T) % 16 == 0 &&
      (reinterpret_cast<uintptr_t>(stage) & 15) == 0) {
    // 16-byte copies (the staged run, its length and its destination are aligned)
    constexpr int W = (int)(16 / sizeof(T));
    for (long e = (long)threadIdx.x * W; e < cnt; e += (long)blockDim.x * W)
      *reinterpret_cast<uint4 *>(dst + e) = *reinterpret_cast<const uint4 *>(stage + e);
  } else {
    for (long e = threadIdx.x; e < cnt; e += blockDim.x) dst[e] = stage[e];
  }
}

// eta ~ Beta(beta r/2, (1-beta) r/2) / beta via two gammas (make_gamma_1 and
// make_beta, kernel_functions.cuh:644-798); lambda *= eta (batchedMultiply
// :458-466); omega ~ N(0, I) scaled by 1/sqrt(c lambda) and cut at p
// (scale_omegas :986-1001); theta += U_W' omega (SGDLM.cu:755-758).
// Bound by the instructions of a (draw, series) pair, most of them the random numbers'.
// The series' inactive coefficients (k >= p_j: U_W is zero outside its leading block, their
// omega is cut) take no normals, quotients or products; the rows of theta are on their way
// (cp.async) while the gammas are drawn.  m = 400, P = 20 (11.9 active on average), 10 000
// draws, FP32: 752 us with all of it over P coefficients, 500 us so.
template <typename T, int PMAX, bool VEC>
__global__ void __launch_bounds__(kSampleThreads)
    k_evolve(int m, int P, long n, const unsigned *__restrict__ p,
             const double *__restrict__ r_t, const double *__restrict__ c_t,
             const double *__restrict__ beta, const T *__restrict__ UW, RngKey key,
             bool compat_unscaled, bool compat_no_boost, T *__restrict__ lambda,
             T *__restrict__ theta, GammaDraws<T> gd, int *__restrict__ draw_flags,
             const T *__restrict__ G) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *Us = reinterpret_cast<T *>(smem_raw);
  T *Gs = Us + P * P;  // G_j when an evolution matrix is given
  T *stage = Gs + (G ? P * P : 0);
  __shared__ int gks[64], gcnt, gq0;  // the series' Gamma coefficients (gamma_row_of)
  __shared__ GammaShape<T> shapes[2];  // of the Beta draw's two gammas
  const int j = blockIdx.y;
  // the reference's unscaled omegas are not cut at p_j: all P take part then
  const int na = compat_unscaled ? P : min(P, (int)p[j]);
  if (threadIdx.x < 64 && threadIdx.x % 32 == 0) {  // one thread of warps 0 and 1 each
    const double bj = beta[j], rj = r_t[j];
    const bool second = threadIdx.x == 32;
    shapes[second] = gamma_shape<T>((T)(second ? 0.5 * (1.0 - bj) * rj : 0.5 * bj * rj), compat_no_boost);
  }
  if (gd.v && (threadIdx.x >> 5) == 2)
    gamma_row_of(gd.sp, gd.rowptr, j, P, (unsigned)m * (unsigned)m, gks, &gcnt, &gq0);
  const long i0 = (long)blockIdx.x * blockDim.x;
  const long cnt = (long)min((long)blockDim.x, n - i0) * P;
  T *src = theta + ((size_t)j * n + i0) * P;
  for (int e = threadIdx.x; e < P * P; e += blockDim.x) Us[e] = UW[(size_t)j * P * P + e];
  if (G)
    for (int e = threadIdx.x; e < P * P; e += blockDim.x) Gs[e] = G[(size_t)j * P * P + e];
  const bool run16 = ((size_t)j * n + i0) * P * sizeof(T) % 16 == 0 && cnt * sizeof(T) % 16 == 0 &&
                     ((reinterpret_cast<uintptr_t>(stage) | reinterpret_cast<uintptr_t>(theta)) & 15) == 0;
  if (run16) {
    constexpr int W16 = V16<T>::W;
    for (long e = (long)threadIdx.x * W16; e < cnt; e += (long)blockDim.x * W16)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                       (unsigned)__cvta_generic_to_shared(stage + e)),
                   "l"(src + e)
                   : "memory");
  } else {
    for (long e = threadIdx.x; e < cnt; e += blockDim.x) stage[e] = src[e];
  }
  __syncthreads();
  const long i = i0 + threadIdx.x;
  T w[PMAX];
  bool fail = false;
  if (i < n) {
    const uint32_t ep = key_epoch(key);
    const T lam0 = lambda[(size_t)j * n + i];
    const double bj = beta[j];
    T eta = T(1);
    if (bj != 1.0) {
      const T ga = gamma_mt<T>(shapes[0], (uint32_t)i, (uint32_t)j, TAG_BETA_A, ep, key.k0, key.k1,
                               key.tab, &fail);
      const T gb = gamma_mt<T>(shapes[1], (uint32_t)i, (uint32_t)j, TAG_BETA_B, ep, key.k0, key.k1,
                               key.tab, &fail);
      eta = (ga / (ga + gb)) / (T)bj;
    }
    const T lam = lam0 * eta;
    lambda[(size_t)j * n + i] = lam;
#pragma unroll
    for (int q = 0; q < PMAX / 4; ++q) {
      if (4 * q < na) {
        const U4 r = philox((uint32_t)i, (uint32_t)j, tag_sub(TAG_OMEGA, q), ep, key.k0, key.k1);
        box_muller<T>(r.x, r.y, w[4 * q], w[4 * q + 1], key.tab);
        if (4 * q + 2 < na)
          box_muller<T>(r.z, r.w, w[4 * q + 2], w[4 * q + 3], key.tab);
        else
          w[4 * q + 2] = w[4 * q + 3] = T(0);
      } else {
        w[4 * q] = w[4 * q + 1] = w[4 * q + 2] = w[4 * q + 3] = T(0);
      }
    }
    // The reference's scale_omegas launch only ever reaches draw 0 of series 0
    // (its z index is always 0), leaving every other omega unscaled; compat mode
    // reproduces that, the default applies the scaling to every draw.
    const bool do_scale = !compat_unscaled || (i == 0 && j == 0);
    if (do_scale) {
      const T den = dev_sqrt((T)c_t[j] * lam);
      const unsigned pj = p[j];
#pragma unroll
      for (int k = 0; k < PMAX; ++k) w[k] = ((unsigned)k < pj) ? w[k] / den : T(0);
    }
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  __syncthreads();  // the staged rows
  if (i < n) {
    T *row = stage + (size_t)threadIdx.x * P;
    if (G) {
      // theta = G theta over the full max_p x max_p product (SGDLM.cu:729-740)
      T g[PMAX];
#pragma unroll
      for (int k = 0; k < PMAX; ++k) {
        T acc = T(0);
        if (k < P)
          for (int l = 0; l < P; ++l) acc += Gs[k + P * l] * row[l];
        g[k] = acc;
      }
#pragma unroll
      for (int k = 0; k < PMAX; ++k)
        if (k < P) row[k] = g[k];
    }
    // an inactive coefficient's sum: U_W's zeros times omega, NaN where omega is not finite
    T zeros = T(0);
#pragma unroll
    for (int l = 0; l < PMAX; ++l) zeros += T(0) * w[l];
    constexpr int W = VEC ? V16<T>::W : 1;
#pragma unroll
    for (int k = 0; k < PMAX; k += W) {
      if (k < P) {
        T o[W];
        if constexpr (VEC)
          V16<T>::ld(row + k, o);
        else
          o[0] = row[k];
#pragma unroll
        for (int b = 0; b < W; ++b) {
          T acc = zeros;
          if (k + b < na) acc = column_dot<T, VEC>(Us, P, k + b, w);
          o[b] = acc + o[b];
        }
        if constexpr (VEC)
          V16<T>::st(row + k, o);
        else
          row[k] = o[0];
      }
    }
    if (fail) atomicOr(&draw_flags[i], DRAW_FLAG_GAMMA_CAP);
  }
  __syncthreads();
  if (gd.v) write_gamma_runs<T>(gd, P, i0, (int)min((long)blockDim.x, n - i0), stage, gks, gcnt, gq0);
  if (run16) {
    constexpr int W16 = V16<T>::W;
    for (long e = (long)threadIdx.x * W16; e < cnt; e += (long)blockDim.x * W16)
      *reinterpret_cast<uint4 *>(src + e) = *reinterpret_cast<const uint4 *>(stage + e);
  } else {
    for (long e = threadIdx.x; e < cnt; e += blockDim.x) src[e] = stage[e];
  }
}

// The draws' Gamma entries from theta, one per thread; scattered reads, as only draws whose
// parental sets changed, or address other rows than their series', come here.
template <typename T>
__global__ void __launch_bounds__(128)
    k_gather_gamma(int P, long n, const int2 *__restrict__ ent, int nnz, const T *__restrict__ theta,
                   T *__restrict__ theta_g) {
  const int q = blockIdx.x * 128 + threadIdx.x;
  if (q >= nnz) return;
  const int e = ent[q].x, j = e / P, k = e - j * P;
  for (long i = blockIdx.y; i < n; i += gridDim.y)
    theta_g[(size_t)i * nnz + q] = theta[((size_t)j * n + i) * P + k];
}

template <typename T> size_t sample_smem(int P) {
  return ((size_t)P * P + P + (size_t)kSampleThreads * P) * sizeof(T);
}

// The instantiation for P coefficients: registers for 8, 16, 24, 32 or 64 of them, and
// 16-byte accesses where P allows them (above 32 the unrolled products are instructions
// enough once).
template <typename T, typename F> void by_width(int P, F f) {
  const auto pick = [&](auto pm) {
    if (P % V16<T>::W == 0)
      f(pm, std::true_type{});
    else
      f(pm, std::false_type{});
  };
  if (P <= 8)
    pick(std::integral_constant<int, 8>{});
  else if (P <= 16)
    pick(std::integral_constant<int, 16>{});
  else if (P <= 24)
    pick(std::integral_constant<int, 24>{});
  else if (P <= 32)
    pick(std::integral_constant<int, 32>{});
  else
    f(std::integral_constant<int, 64>{}, std::false_type{});
}

}  // namespace

template <typename T>
void launch_sample(cudaStream_t s, int m, int P, long n, const double *m_t,
                   const double *n_t, const double *s_t, const T *U, RngKey key,
                   T *lambda, T *theta, GammaDraws<T> gd, int *draw_flags, const unsigned *p) {
  dim3 grid((unsigned)((n + kSampleThreads - 1) / kSampleThreads), (unsigned)m);
  const size_t smem = sample_smem<T>(P);
  by_width<T>(P, [&](auto pm, auto vec) {
    auto *f = k_sample<T, pm.value, vec.value>;
    if (smem > 48 * 1024) cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    f<<<grid, kSampleThreads, smem, s>>>(m, P, n, m_t, n_t, s_t, U, key, lambda, theta, gd, draw_flags, p);
  });
}

template <typename T>
void launch_evolve(cudaStream_t s, int m, int P, long n, const unsigned *p,
                   const double *r_t, const double *c_t, const double *beta,
                   const T *UW, RngKey key, bool compat_unscaled_omega,
                   bool compat_beta_no_boost, T *lambda, T *theta, GammaDraws<T> gd,
                   int *draw_flags, const T *G) {
  dim3 grid((unsigned)((n + kSampleThreads - 1) / kSampleThreads), (unsigned)m);
  const size_t smem =
      ((size_t)P * P * (G ? 2 : 1) + (size_t)kSampleThreads * P) * sizeof(T);
  by_width<T>(P, [&](auto pm, auto vec) {
    auto *f = k_evolve<T, pm.value, vec.value>;
    if (smem > 48 * 1024) cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    f<<<grid, kSampleThreads, smem, s>>>(m, P, n, p, r_t, c_t, beta, UW, key, compat_unscaled_omega,
                                         compat_beta_no_boost, lambda, theta, gd, draw_flags, G);
  });
}

template <typename T>
void launch_gather_gamma(cudaStream_t s, int P, long n, const int2 *ent, int nnz, const T *theta,
                         T *theta_g) {
  if (nnz == 0) return;
  const dim3 grid((unsigned)((nnz + 127) / 128), (unsigned)(n < 4096 ? n : 4096));
  k_gather_gamma<T><<<grid, 128, 0, s>>>(P, n, ent, nnz, theta, theta_g);
}
template void launch_gather_gamma<float>(cudaStream_t, int, long, const int2 *, int, const float *,
                                         float *);
template void launch_gather_gamma<double>(cudaStream_t, int, long, const int2 *, int, const double *,
                                          double *);

template void launch_sample<float>(cudaStream_t, int, int, long, const double *,
                                   const double *, const double *, const float *, RngKey,
                                   float *, float *, GammaDraws<float>, int *, const unsigned *);
template void launch_sample<double>(cudaStream_t, int, int, long, const double *,
                                    const double *, const double *, const double *,
                                    RngKey, double *, double *, GammaDraws<double>, int *,
                                    const unsigned *);
template void launch_evolve<float>(cudaStream_t, int, int, long, const unsigned *,
                                   const double *, const double *, const double *,
                                   const float *, RngKey, bool, bool, float *, float *,
                                   GammaDraws<float>, int *, const float *);
template void launch_evolve<double>(cudaStream_t, int, int, long, const unsigned *,
                                    const double *, const double *, const double *,
                                    const double *, RngKey, bool, bool, double *,
                                    double *, GammaDraws<double>, int *, const double *);

}  // namespace sgdlm
