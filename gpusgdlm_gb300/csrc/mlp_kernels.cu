// The learned importance proposal's network: a per-series MLP
//   features (F) -> 128 -> GELU -> 128 -> GELU -> outputs (O)
// with BF16 weights and FP32 accumulation, its backward pass, a masked
// mean-squared-error loss and Adam -- hand-written kernels, no library GEMM.
//
// Parameters live as FP32 master copies (what Adam updates) and BF16 copies
// (what the forward and the backward's data gradients multiply by), in one flat
// layout: W1 (H x F, row-major), b1 (H), W2 (H x H), b2 (H), W3 (O x H), b3 (O).
// Activations are row-major (batch x width).
//
// The reference has no counterpart: its proposal is the decoupled naive
// posterior (rSGDLM/src/SGDLM/SGDLM.cu:623-677).
#include <algorithm>

#include <cuda_bf16.h>

#include "kernels.hpp"
#include "proposal.hpp"

namespace sgdlm {
namespace {

// C[i, j] = sum_k A[i, k] B(k, j), A row-major (M x K), B BF16: the N x K row-major matrix
// (BT) or the K x N one; C row-major with leading dimension ldc.  Optional epilogue:
// + bias[j], store the pre-activation to Z, apply GELU; or times GELU'(Zg) (the backward's
// dZ = dA * GELU'(Z)).
//
// FP32 sums in increasing k, one thread per output, as long as the network is this narrow
// (K, N <= 128: a layer of 4 096 rows is 67 MFMA, 2 us of the FP32 pipe, and 1 us of
// memory).  Bound by shared-memory loads and by the latency of the K chunks' loads: 32 x 64
// outputs per block of 128 threads, 4 x 4 each (two 16-byte loads per 16 FMAs), so that a
// layer of 4 096 rows is 256 blocks and one of 200 series still 14; the next chunk's values
// come into registers while the current one is multiplied, two buffers, one barrier per
// chunk.  4 096 x 128 x 128: 15.7 us with 2 x 2 outputs per thread and 32 x 32 tiles,
// 10.1 us (11.2 us with GELU') so; 200 rows: 12.4 us, 9.1 us.
constexpr int kTileM = 32, kTileN = 64, kTileK = 32, kMatThreads = 128;
template <bool BT>
__global__ void __launch_bounds__(kMatThreads)
    k_matmul(int M, int N, int K, const float *__restrict__ A, const __nv_bfloat16 *__restrict__ B,
             float *__restrict__ C, int ldc, const float *__restrict__ bias, float *__restrict__ Z,
             int gelu, const float *__restrict__ Zg) {
  __shared__ __align__(16) float As[2][kTileM][kTileK + 4];  // [i][k]
  __shared__ __align__(16) float Bs[2][kTileK][kTileN + 4];  // [k][j]
  constexpr int NA = kTileM * kTileK / kMatThreads, NB = kTileK * kTileN / kMatThreads;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int i0 = blockIdx.y * kTileM, j0 = blockIdx.x * kTileN;
  float ra[NA], rb[NB];
  // the thread's e-th value of A's and B's chunk: A by rows; B by rows of j, or (BT) eight
  // k by four j per 32 values (distinct banks in Bs)
  auto at_a = [&](int e, int &r, int &c) {
    r = (e * kMatThreads + tid) / kTileK;
    c = tid % kTileK;
  };
  auto at_b = [&](int e, int &k, int &j) {
    if (BT) {
      const int g = e * (kMatThreads / 32) + tid / 32;
      k = g % (kTileK / 8) * 8 + tid % 8;
      j = g / (kTileK / 8) * 4 + tid % 32 / 8;
    } else {
      k = (e * kMatThreads + tid) / kTileN;
      j = tid % kTileN;
    }
  };
  auto fetch = [&](int k0) {
#pragma unroll
    for (int e = 0; e < NA; ++e) {
      int r, c;
      at_a(e, r, c);
      const int i = i0 + r, k = k0 + c;
      ra[e] = (i < M && k < K) ? A[(long)i * K + k] : 0.f;
    }
#pragma unroll
    for (int e = 0; e < NB; ++e) {
      int k, j;
      at_b(e, k, j);
      k += k0, j += j0;
      rb[e] = (k < K && j < N) ? __bfloat162float(B[BT ? (long)j * K + k : (long)k * N + j]) : 0.f;
    }
  };
  float acc[4][4] = {};
  fetch(0);
  // this thread's outputs: rows i .. i + 3, columns j .. j + 3, 16 bytes at a time where
  // the rows of C, Z and Zg allow it; Zg is on its way during the products
  const int i = i0 + 4 * ty, j = j0 + 4 * tx;
  const bool vec = j + 3 < N && ldc % 4 == 0 &&
                   ((reinterpret_cast<uintptr_t>(C) | reinterpret_cast<uintptr_t>(Z) |
                     reinterpret_cast<uintptr_t>(Zg)) & 15) == 0;
  float zg[4][4] = {};
  if (Zg) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (i + u >= M) break;
      const float *src = Zg + (long)(i + u) * ldc + j;
      if (vec) {
        const float4 v = *reinterpret_cast<const float4 *>(src);
        zg[u][0] = v.x, zg[u][1] = v.y, zg[u][2] = v.z, zg[u][3] = v.w;
      } else {
#pragma unroll
        for (int v = 0; v < 4; ++v)
          if (j + v < N) zg[u][v] = src[v];
      }
    }
  }
  int buf = 0;
  for (int k0 = 0; k0 < K; k0 += kTileK, buf ^= 1) {
    // (the buffer was read two chunks ago, before the last barrier)
#pragma unroll
    for (int e = 0; e < NA; ++e) {
      int r, c;
      at_a(e, r, c);
      As[buf][r][c] = ra[e];
    }
#pragma unroll
    for (int e = 0; e < NB; ++e) {
      int k, j;
      at_b(e, k, j);
      Bs[buf][k][j] = rb[e];
    }
    __syncthreads();
    if (k0 + kTileK < K) fetch(k0 + kTileK);
#pragma unroll
    for (int k = 0; k < kTileK; k += 4) {
      float av[4][4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float4 a = *reinterpret_cast<const float4 *>(&As[buf][4 * ty + u][k]);
        av[u][0] = a.x, av[u][1] = a.y, av[u][2] = a.z, av[u][3] = a.w;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float4 b = *reinterpret_cast<const float4 *>(&Bs[buf][k + q][4 * tx]);
        const float bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int v = 0; v < 4; ++v) acc[u][v] = fmaf(av[u][q], bv[v], acc[u][v]);
      }
    }
  }
  auto put = [&](float *dst, const float (&x)[4]) {
    if (vec) {
      *reinterpret_cast<float4 *>(dst) = make_float4(x[0], x[1], x[2], x[3]);
    } else {
#pragma unroll
      for (int v = 0; v < 4; ++v)
        if (j + v < N) dst[v] = x[v];
    }
  };
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    if (i + u >= M) break;
    if (bias) {
#pragma unroll
      for (int v = 0; v < 4; ++v)
        if (j + v < N) acc[u][v] += bias[j + v];
    }
    if (Z) put(Z + (long)(i + u) * ldc + j, acc[u]);
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      if (gelu) acc[u][v] = gelu_f(acc[u][v]);
      if (Zg) acc[u][v] *= gelu_grad_f(zg[u][v]);
    }
    put(C + (long)(i + u) * ldc + j, acc[u]);
  }
}

// Weight and bias gradients dW = dZ' A, db = colsum dZ of the three layers in one
// launch: block (tile, chunk) sums a chunk of the batch's rows for a 64 x 64 tile of
// one layer's dW (256 threads, 4 x 4 outputs each, FP32) into its place of
// part[chunk * total ..], laid out as the gradient; k_grad_sum adds the chunks.  The
// batch is the reduction dimension, so without chunks a layer's dW is at most 16
// blocks that walk through all rows one after the other (4096 rows: 272 us a layer,
// and 227 us for a bias's column sums; all of them in chunks of 64 rows: 19 us, the
// sum of the chunks 8 us).
constexpr int kGradTile = 64, kGradRows = 16;
struct GradLayer {
  const float *dZ, *A;  // B x M, B x N row-major
  int M, N;
  long w, b;            // where dW (M x N) and db (M) lie in the gradient
  int tiles_n, tile0;   // column tiles; the layer's first tile
};
struct GradLayers {
  GradLayer l[3];
  int tiles;
};
__global__ void __launch_bounds__(256)
    k_grad(GradLayers g, int B, int rows, long total, float *__restrict__ part) {
  __shared__ float Zs[kGradRows][kGradTile + 4], As[kGradRows][kGradTile + 4];
  const int tile = blockIdx.x;
  const GradLayer q = g.l[tile >= g.l[2].tile0 ? 2 : (tile >= g.l[1].tile0 ? 1 : 0)];
  const int t = tile - q.tile0, i0 = t / q.tiles_n * kGradTile, j0 = t % q.tiles_n * kGradTile;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int b0 = blockIdx.y * rows, b1 = min(B, b0 + rows);
  float acc[4][4] = {}, bias[4] = {};
  for (int k0 = b0; k0 < b1; k0 += kGradRows) {
    for (int e = threadIdx.x; e < kGradRows * kGradTile; e += 256) {
      const int r = e / kGradTile, c = e % kGradTile, k = k0 + r;
      Zs[r][c] = (k < b1 && i0 + c < q.M) ? q.dZ[(long)k * q.M + i0 + c] : 0.f;
      As[r][c] = (k < b1 && j0 + c < q.N) ? q.A[(long)k * q.N + j0 + c] : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kGradRows; ++r) {
      const float4 z = *reinterpret_cast<const float4 *>(&Zs[r][4 * ty]);
      const float4 a = *reinterpret_cast<const float4 *>(&As[r][4 * tx]);
      const float zv[4] = {z.x, z.y, z.z, z.w}, av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        bias[u] += zv[u];
#pragma unroll
        for (int v = 0; v < 4; ++v) acc[u][v] = fmaf(zv[u], av[v], acc[u][v]);
      }
    }
    __syncthreads();
  }
  float *out = part + (long)blockIdx.y * total;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int i = i0 + 4 * ty + u;
    if (i >= q.M) continue;
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const int j = j0 + 4 * tx + v;
      if (j < q.N) out[q.w + (long)i * q.N + j] = acc[u][v];
    }
    if (j0 == 0 && tx == 0) out[q.b + i] = bias[u];
  }
}
__global__ void k_grad_sum(long total, int chunks, const float *__restrict__ part,
                           float *__restrict__ grad) {
  const long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (e >= total) return;
  float s = 0.f;
#pragma unroll 8
  for (int c = 0; c < chunks; ++c) s += part[(long)c * total + e];
  grad[e] = s;
}

// Masked mean squared error over B x O outputs: loss = sum mask (o - y)^2 / cnt,
// dO = 2 mask (o - y) / cnt, cnt = sum mask (at least 1).  Two launches over the same
// blocks: each block's sums into part (2 doubles per block), then every block adds
// them up and writes its share of dO (131 000 outputs: 278 us in one block, now 15 us).
constexpr int kMseThreads = 256, kMseBlocks = 256;
__device__ __forceinline__ void mse_block_sum(double &l, double &c) {
  __shared__ double s_l[kMseThreads / 32], s_c[kMseThreads / 32];
  for (int o = 16; o > 0; o >>= 1) {
    l += __shfl_xor_sync(0xffffffffu, l, o);
    c += __shfl_xor_sync(0xffffffffu, c, o);
  }
  if ((threadIdx.x & 31) == 0) {
    s_l[threadIdx.x >> 5] = l;
    s_c[threadIdx.x >> 5] = c;
  }
  __syncthreads();
  l = c = 0.0;
  for (int w = 0; w < kMseThreads / 32; ++w) {
    l += s_l[w];
    c += s_c[w];
  }
}
__global__ void __launch_bounds__(kMseThreads)
    k_mse_sums(long n, const float *__restrict__ O, const float *__restrict__ Y,
               const float *__restrict__ mask, double *__restrict__ part) {
  double l = 0.0, c = 0.0;
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < n; e += (long)gridDim.x * blockDim.x) {
    const double d = (double)O[e] - (double)Y[e];
    l += (double)mask[e] * d * d;
    c += (double)mask[e];
  }
  mse_block_sum(l, c);
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = l;
    part[2 * blockIdx.x + 1] = c;
  }
}
__global__ void __launch_bounds__(kMseThreads)
    k_mse_grad(long n, const float *__restrict__ O, const float *__restrict__ Y,
               const float *__restrict__ mask, const double *__restrict__ part,
               float *__restrict__ dO, double *__restrict__ loss) {
  const bool have = threadIdx.x < gridDim.x;  // gridDim.x <= kMseBlocks = kMseThreads
  double l = have ? part[2 * threadIdx.x] : 0.0, c = have ? part[2 * threadIdx.x + 1] : 0.0;
  mse_block_sum(l, c);
  const double cnt = c > 1.0 ? c : 1.0;
  if (blockIdx.x == 0 && threadIdx.x == 0 && loss) *loss = l / cnt;
  const float g = (float)(2.0 / cnt);
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < n; e += (long)gridDim.x * blockDim.x)
    dO[e] = g * mask[e] * (O[e] - Y[e]);
}

// Adam (Kingma & Ba 2015) on the flat FP32 parameters, bias-corrected with the
// step count t, then the BF16 copy.
__global__ void k_adam(long n, float *__restrict__ w, __nv_bfloat16 *__restrict__ w16,
                       const float *__restrict__ g, float *__restrict__ m1, float *__restrict__ m2,
                       float lr, float b1, float b2, float eps, float c1, float c2) {
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < n; e += (long)gridDim.x * blockDim.x) {
    const float ge = g[e];
    const float a = b1 * m1[e] + (1.f - b1) * ge;
    const float b = b2 * m2[e] + (1.f - b2) * ge * ge;
    m1[e] = a;
    m2[e] = b;
    const float x = w[e] - lr * (a / c1) / (sqrtf(b / c2) + eps);
    w[e] = x;
    w16[e] = __float2bfloat16_rn(x);
  }
}

__global__ void k_to_bf16(long n, const float *__restrict__ w, __nv_bfloat16 *__restrict__ w16) {
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < n; e += (long)gridDim.x * blockDim.x)
    w16[e] = __float2bfloat16_rn(w[e]);
}

// B is N x K row-major if b_transposed, else K x N
void matmul(cudaStream_t s, int M, int N, int K, const float *A, const __nv_bfloat16 *B,
            bool b_transposed, float *C, int ldc, const float *bias, float *Z, bool gelu,
            const float *Zg = nullptr) {
  const dim3 grid((N + kTileN - 1) / kTileN, (M + kTileM - 1) / kTileM);
  auto *f = b_transposed ? k_matmul<true> : k_matmul<false>;
  f<<<grid, kMatThreads, 0, s>>>(M, N, K, A, B, C, ldc, bias, Z, gelu ? 1 : 0, Zg);
}

int grid_for(long n) {
  long g = (n + 255) / 256;
  return (int)(g < 1024 ? (g < 1 ? 1 : g) : 1024);
}

}  // namespace

MlpLayout mlp_layout(int F, int O) {
  MlpLayout L{};
  L.F = F;
  L.H = kMlpHidden;
  L.O = O;
  L.w1 = 0;
  L.b1 = L.w1 + (long)L.H * F;
  L.w2 = L.b1 + L.H;
  L.b2 = L.w2 + (long)L.H * L.H;
  L.w3 = L.b2 + L.H;
  L.b3 = L.w3 + (long)O * L.H;
  L.total = L.b3 + O;
  return L;
}

void mlp_forward(cudaStream_t s, const MlpLayout &L, int B, const float *X, const float *w,
                 const __nv_bfloat16 *w16, MlpActs a) {
  // Z1 = X W1' + b1, A1 = GELU(Z1): W1 is H x F row-major
  matmul(s, B, L.H, L.F, X, w16 + L.w1, true, a.A1, L.H, w + L.b1, a.Z1, true);
  matmul(s, B, L.H, L.H, a.A1, w16 + L.w2, true, a.A2, L.H, w + L.b2, a.Z2, true);
  matmul(s, B, L.O, L.H, a.A2, w16 + L.w3, true, a.Out, L.O, w + L.b3, nullptr, false);
}

namespace {
// Chunks of the batch in the gradient's sums: 64 rows each, at most 64 chunks.
int grad_rows(int B) { return std::max(64, (B + 63) / 64); }
int grad_chunks(int B) { return (B + grad_rows(B) - 1) / grad_rows(B); }
}  // namespace

size_t mlp_workspace(const MlpLayout &L, int B) {
  return 4 * (size_t)kMseBlocks + (size_t)grad_chunks(B) * L.total;
}

void mlp_loss_backward(cudaStream_t s, const MlpLayout &L, int B, const float *X, const float *Y,
                       const float *mask, const __nv_bfloat16 *w16, MlpActs a, float *work,
                       float *grad, double *loss) {
  const long nO = (long)B * L.O;
  const int mse_blocks = (int)std::min<long>(kMseBlocks, (nO + kMseThreads - 1) / kMseThreads);
  double *sums = reinterpret_cast<double *>(work);
  float *part = work + 4 * kMseBlocks;
  k_mse_sums<<<mse_blocks, kMseThreads, 0, s>>>(nO, a.Out, Y, mask, sums);
  k_mse_grad<<<mse_blocks, kMseThreads, 0, s>>>(nO, a.Out, Y, mask, sums, a.dOut, loss);
  // dZ2 = (dOut W3) GELU'(Z2), dZ1 = (dZ2 W2) GELU'(Z1)
  matmul(s, B, L.H, L.O, a.dOut, w16 + L.w3, false, a.dA, L.H, nullptr, nullptr, false, a.Z2);
  matmul(s, B, L.H, L.H, a.dA, w16 + L.w2, false, a.dA2, L.H, nullptr, nullptr, false, a.Z1);
  // dW3 = dOut' A2, dW2 = dZ2' A1, dW1 = dZ1' X and the bias gradients
  GradLayers g{};
  auto layer = [&](int q, const float *dZ, const float *A, int M, int N, long w, long b) {
    const int tn = (N + kGradTile - 1) / kGradTile;
    g.l[q] = GradLayer{dZ, A, M, N, w, b, tn, g.tiles};
    g.tiles += tn * ((M + kGradTile - 1) / kGradTile);
  };
  layer(0, a.dOut, a.A2, L.O, L.H, L.w3, L.b3);
  layer(1, a.dA, a.A1, L.H, L.H, L.w2, L.b2);
  layer(2, a.dA2, X, L.H, L.F, L.w1, L.b1);
  const int chunks = grad_chunks(B);
  k_grad<<<dim3(g.tiles, chunks), 256, 0, s>>>(g, B, grad_rows(B), L.total, part);
  k_grad_sum<<<(unsigned)((L.total + 127) / 128), 128, 0, s>>>(L.total, chunks, part, grad);
}

void mlp_adam(cudaStream_t s, const MlpLayout &L, float *w, __nv_bfloat16 *w16, const float *grad,
              float *m1, float *m2, float lr, long step) {
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
  k_adam<<<grid_for(L.total), 256, 0, s>>>(L.total, w, w16, grad, m1, m2, lr, b1, b2, eps, c1, c2);
}

void mlp_refresh_bf16(cudaStream_t s, const MlpLayout &L, const float *w, __nv_bfloat16 *w16) {
  k_to_bf16<<<grid_for(L.total), 256, 0, s>>>(L.total, w, w16);
}

}  // namespace sgdlm
