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

constexpr int kTile = 32;

template <typename T> __device__ __forceinline__ float to_f(T v);
template <> __device__ __forceinline__ float to_f<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) {
  return __bfloat162float(v);
}

// C[i, j] (+)= sum_k A(i, k) B(k, j), A(i, k) = A[i*sai + k*sak],
// B(k, j) = B[k*sbk + j*sbj], C row-major with leading dimension ldc; 32 x 32
// output tiles, 16 x 16 threads with 2 x 2 outputs each, K in chunks of 32
// staged in shared memory, FP32 accumulation.  Optional epilogue: + bias[j],
// store the pre-activation to Z, apply GELU; or times GELU'(Zg) (the backward's
// dZ = dA * GELU'(Z)).
template <typename TB>
__global__ void __launch_bounds__(256)
    k_matmul(int M, int N, int K, const float *__restrict__ A, long sai, long sak,
             const TB *__restrict__ B, long sbk, long sbj, float *__restrict__ C, int ldc,
             const float *__restrict__ bias, float *__restrict__ Z, int gelu,
             const float *__restrict__ Zg) {
  __shared__ float As[kTile][kTile + 1];
  __shared__ float Bs[kTile][kTile + 1];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int i0 = blockIdx.y * kTile, j0 = blockIdx.x * kTile;
  float acc[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
  for (int k0 = 0; k0 < K; k0 += kTile) {
    for (int e = threadIdx.x; e < kTile * kTile; e += blockDim.x) {
      const int r = e / kTile, c = e % kTile;
      const int i = i0 + r, k = k0 + c;
      As[r][c] = (i < M && k < K) ? A[(long)i * sai + (long)k * sak] : 0.f;
      const int kk = k0 + r, j = j0 + c;
      Bs[r][c] = (kk < K && j < N) ? to_f(B[(long)kk * sbk + (long)j * sbj]) : 0.f;
    }
    __syncthreads();
#pragma unroll 8
    for (int k = 0; k < kTile; ++k) {
      const float a0 = As[ty][k], a1 = As[ty + 16][k];
      const float b0 = Bs[k][tx], b1 = Bs[k][tx + 16];
      acc[0][0] = fmaf(a0, b0, acc[0][0]);
      acc[0][1] = fmaf(a0, b1, acc[0][1]);
      acc[1][0] = fmaf(a1, b0, acc[1][0]);
      acc[1][1] = fmaf(a1, b1, acc[1][1]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int v = 0; v < 2; ++v) {
      const int i = i0 + ty + 16 * u, j = j0 + tx + 16 * v;
      if (i >= M || j >= N) continue;
      float x = acc[u][v];
      if (bias) x += bias[j];
      if (Z) Z[(long)i * ldc + j] = x;
      if (gelu) x = gelu_f(x);
      if (Zg) x *= gelu_grad_f(Zg[(long)i * ldc + j]);
      C[(long)i * ldc + j] = x;
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

template <typename TB>
void matmul(cudaStream_t s, int M, int N, int K, const float *A, long sai, long sak, const TB *B,
            long sbk, long sbj, float *C, int ldc, const float *bias, float *Z, bool gelu,
            const float *Zg = nullptr) {
  const dim3 grid((N + kTile - 1) / kTile, (M + kTile - 1) / kTile);
  k_matmul<TB><<<grid, 256, 0, s>>>(M, N, K, A, sai, sak, B, sbk, sbj, C, ldc, bias, Z,
                                    gelu ? 1 : 0, Zg);
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
  // Z1 = X W1' + b1, A1 = GELU(Z1): W1 is H x F row-major, B(k, j) = W1[j*F + k]
  matmul<__nv_bfloat16>(s, B, L.H, L.F, X, L.F, 1, w16 + L.w1, 1, L.F, a.A1, L.H, w + L.b1, a.Z1,
                        true);
  matmul<__nv_bfloat16>(s, B, L.H, L.H, a.A1, L.H, 1, w16 + L.w2, 1, L.H, a.A2, L.H, w + L.b2,
                        a.Z2, true);
  matmul<__nv_bfloat16>(s, B, L.O, L.H, a.A2, L.H, 1, w16 + L.w3, 1, L.H, a.Out, L.O, w + L.b3,
                        nullptr, false);
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
  matmul<__nv_bfloat16>(s, B, L.H, L.O, a.dOut, L.O, 1, w16 + L.w3, L.H, 1, a.dA, L.H, nullptr,
                        nullptr, false, a.Z2);
  matmul<__nv_bfloat16>(s, B, L.H, L.H, a.dA, L.H, 1, w16 + L.w2, L.H, 1, a.dA2, L.H, nullptr,
                        nullptr, false, a.Z1);
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
