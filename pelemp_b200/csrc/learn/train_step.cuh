// train_step.cuh -- one training step of the surrogate as two kernels.
//
// k_train_rows takes 64 batch rows per CTA through the whole network and
// back with everything in shared memory: batch gather, normalisation and
// residual targets, the four layers, the loss, the four backward products and
// the weight gradients of its rows, which stay in registers while the CTA
// takes further tiles and leave it once, as one partial gradient per CTA.
// k_train_update sums the partials (in a fixed order) and applies Adam.
// The network is 10-64-64-64-5: a batch of 8192 rows is 470 MFLOP of FP32
// and its activations are 64 wide, so a step is bound by passes over memory
// and by launches when each product, activation and column sum is a kernel
// of its own: 25 launches and 350 us a step, the split-K weight gradients
// 45 us each (32 CTAs, FP32 atomics) and the column sums 11 us each (64
// CTAs).  Now 29 us for the rows and 4 us for the update (256 threads a CTA
// with 4 x 4 outputs each: 36 us; weights staged a word at a time and before
// the tuples are asked for: 31 us).  Of the 55k cycles of a tile, 4k are its
// loads, 7k each 64 x 64 product with its activation or its derivative, 3.4k
// each 64 x 64 weight gradient; 42 % of the issue slots, the waits are on
// shared memory.  Every product's sums run in the order of the reduction index, as
// an FP32 multiply-add chain; only the gradients' sum over rows is split (64
// rows, then the CTAs' partials).
#pragma once

#include <cuda_bf16.h>

#include "learn_common.cuh"

namespace pmp {

// flat parameter vector (weights row major [out][in])
constexpr int kP_W1 = 0;               // 64 x 16 (inputs padded to 16)
constexpr int kP_B1 = kP_W1 + 64 * 16;
constexpr int kP_W2 = kP_B1 + 64;      // 64 x 64
constexpr int kP_B2 = kP_W2 + 64 * 64;
constexpr int kP_W3 = kP_B2 + 64;      // 64 x 64
constexpr int kP_B3 = kP_W3 + 64 * 64;
constexpr int kP_W4 = kP_B3 + 64;      // 8 x 64 (outputs padded to 8)
constexpr int kP_B4 = kP_W4 + 8 * 64;
constexpr int kP_N = kP_B4 + 8;

__host__ __device__ inline unsigned long long mix64(unsigned long long z)
{
  z += 0x9e3779b97f4a7c15ULL;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
  return z ^ (z >> 31);
}

__device__ __forceinline__ float bf16r(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

__device__ __forceinline__ float silu_exact(float x) { return x / (1.f + expf(-x)); }

// silu(x) as the inference kernel rounds it (mlp_mma.cuh): h = bf16(x/2),
// bf16(fma(h, bf16(tanh h), h))
__device__ __forceinline__ float silu_bf16(float x)
{
  const float h = bf16r(0.5f * x);
  return bf16r(fmaf(h, bf16r(tanhf(h)), h));
}

constexpr int kTrainRows = 64;      // batch rows per tile
constexpr int kTrainThreads = 512;  // 2 x 4 outputs each; weight gradients 4 x 4 over half of the rows each
constexpr int kTP = 68;             // pitch of 64-wide tiles: 16-byte rows, 4 banks apart
constexpr int kTX = 20;             // pitch of the 16-wide input tile
constexpr int kTY = 12;             // pitch of the output gradients

// The rows of a batch: drawn from the tuples (random: by seed and step, else
// in order from `base`), or given (X: 16 columns, Y: 8 columns a row).
struct TrainBatch {
  const float* tuples;
  long long ntuples, base;
  unsigned long long seed;
  long long step;
  int random;
  const float *X, *Y;
  long long rows;
};

struct TrainSmem {
  float W1[64 * kTX], W2[64 * kTP], W3[64 * kTP], W4[8 * kTP];
  float b1[64], b2[64], b3[64], b4[8];
  float X[kTrainRows * kTX];
  float Y[kTrainRows * 8];
  float dY[kTrainRows * kTY];
  float H1[kTrainRows * kTP], A1[kTrainRows * kTP];
  float H2[kTrainRows * kTP], A2[kTrainRows * kTP];
  float H3[kTrainRows * kTP], A3[kTrainRows * kTP];
  float dH[kTrainRows * kTP];
  float bell[kTrainRows], bg[kTrainRows];
  float red[8 * 64];
  double val[kLearnOut];
};

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float at4(const float4& v, int i) { return i == 0 ? v.x : (i == 1 ? v.y : (i == 2 ? v.z : v.w)); }

__device__ __forceinline__ void st4(float* p, const float4& v) { *reinterpret_cast<float4*>(p) = v; }

// batch row r's tuple (want, and there is one)
__device__ __forceinline__ void load_row(const TrainBatch& T, long long r, float4 (&t)[4], bool want)
{
  if (!want || !T.tuples || r >= T.rows) {
    return;
  }
  const long long i = T.random ? (long long)(mix64(T.seed ^ mix64((unsigned long long)T.step * 1315423911ULL + r)) %
                                             (unsigned long long)T.ntuples)
                               : T.base + r;
  const float4* o = reinterpret_cast<const float4*>(T.tuples + i * 16);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    t[q] = __ldg(o + q);
  }
}

// rows [r][n] = sum_k A[r][k] W[n][k] of a hidden layer, bias and SiLU: this
// thread's rows 2 ty + i and columns tx + 16 j (the W rows of 16 neighbouring
// lanes are then 4 banks apart)
template <int K, int PA>
__device__ __forceinline__ void layer_fwd(const float* A, const float* W, const float* b, float* H, float* Act, int tx,
                                          int ty, int quant)
{
  float acc[2][4] = {};
#pragma unroll 4
  for (int k = 0; k < K; k += 4) {
    float4 a[2], w[4];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      a[i] = ld4(A + (2 * ty + i) * PA + k);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      w[j] = ld4(W + (tx + 16 * j) * PA + k);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc[i][j] = fmaf(at4(a[i], q), at4(w[j], q), acc[i][j]);
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = tx + 16 * j;
      const float h = acc[i][j] + b[n];
      const int o = (2 * ty + i) * kTP + n;
      H[o] = h;
      Act[o] = quant ? silu_bf16(h) : silu_exact(h);
    }
  }
}

// acc[n][k] += sum over rows [r0, r0 + 32) of dH[r][n] A[r][k]: rows n = 4 ty + i,
// columns 4 tx + j
__device__ __forceinline__ void layer_dw(const float* dH, const float* A, float (&acc)[4][4], int tx, int ty, int r0)
{
#pragma unroll 4
  for (int r = r0; r < r0 + kTrainRows / 2; ++r) {
    const float4 d = ld4(dH + r * kTP + 4 * ty);
    const float4 a = ld4(A + r * kTP + 4 * tx);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[i][j] = fmaf(at4(d, i), at4(a, j), acc[i][j]);
      }
    }
  }
}

// dH of the layer below: (sum_n D[r][n] W[n][k]) silu'(H[r][k]), N outputs;
// overwrites dH (= D for the hidden layers) between two barriers
template <int N, int PD>
__device__ __forceinline__ void layer_bwd(const float* D, const float* W, const float* H, float* dH, int tx, int ty)
{
  float acc[2][4] = {};
#pragma unroll 2
  for (int n = 0; n < N; n += 4) {
    float4 d[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      d[i] = ld4(D + (2 * ty + i) * PD + n);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float4 w = ld4(W + (n + q) * kTP + 4 * tx);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc[i][j] = fmaf(at4(d[i], q), at4(w, j), acc[i][j]);
        }
      }
    }
  }
  __syncthreads();  // every reader of dH is done
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int o = (2 * ty + i) * kTP + 4 * tx;
    const float4 h4 = ld4(H + o);
    float v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float h = at4(h4, j);
      const float s = 1.f / (1.f + expf(-h));
      v[j] = acc[i][j] * s * (1.f + h * (1.f - s));
    }
    *reinterpret_cast<float4*>(dH + o) = make_float4(v[0], v[1], v[2], v[3]);
  }
  __syncthreads();
}

// sum of 8 of the tile's rows of column n (part p of 8)
__device__ __forceinline__ float col_part(const float* D, int pitch, int n, int p)
{
  float s = 0.f;
#pragma unroll 4
  for (int r = 8 * p; r < 8 * p + 8; ++r) {
    s += D[r * pitch + n];
  }
  return s;
}

// BACK: partial gradients part[blockIdx.x][kP_N] and, with `loss`, the sum of
// squared errors.  Otherwise the forward pass alone: val[k] += the squared
// error of output k in the targets' units.
template <bool BACK>
__global__ void __launch_bounds__(kTrainThreads) k_train_rows(const __grid_constant__ TrainBatch T,
                                                              const __grid_constant__ LearnNorm nrm, const float* w,
                                                              int quant, float* part, double* loss, double* val)
{
  extern __shared__ __align__(16) unsigned char train_smem[];
  TrainSmem& S = *reinterpret_cast<TrainSmem*>(train_smem);
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  // weight gradients: the CTA's halves take half of the rows each
  const int ht = tid & 255, wy = ht >> 4, hr0 = (tid >> 8) * (kTrainRows / 2);
  // the first tile's tuples and the weights, 16 bytes a load, are asked for
  // together
  const long long tiles = (T.rows + kTrainRows - 1) / kTrainRows;
  float4 t4[4] = {};
  load_row(T, (long long)blockIdx.x * kTrainRows + tid, t4, tid < kTrainRows);
  {
    static_assert(kTrainThreads == 512, "W2 and W3 twice, W1 half, W4 a quarter");
    const float4* g = reinterpret_cast<const float4*>(w);
    float4 a[6];
    a[0] = __ldg(g + kP_W2 / 4 + tid);
    a[1] = __ldg(g + kP_W2 / 4 + 512 + tid);
    a[2] = __ldg(g + kP_W3 / 4 + tid);
    a[3] = __ldg(g + kP_W3 / 4 + 512 + tid);
    a[4] = tid < 256 ? __ldg(g + kP_W1 / 4 + tid) : make_float4(0.f, 0.f, 0.f, 0.f);
    a[5] = tid < 128 ? __ldg(g + kP_W4 / 4 + tid) : make_float4(0.f, 0.f, 0.f, 0.f);
    const int o = (tid >> 4) * kTP + 4 * (tid & 15);
    st4(S.W2 + o, a[0]);
    st4(S.W2 + o + 32 * kTP, a[1]);
    st4(S.W3 + o, a[2]);
    st4(S.W3 + o + 32 * kTP, a[3]);
    if (tid < 256) {
      st4(S.W1 + (tid >> 2) * kTX + 4 * (tid & 3), a[4]);
    }
    if (tid < 128) {
      st4(S.W4 + o, a[5]);
    }
  }
  if (tid < 64) {
    S.b1[tid] = w[kP_B1 + tid];
    S.b2[tid] = w[kP_B2 + tid];
    S.b3[tid] = w[kP_B3 + tid];
  }
  if (tid < 8) {
    S.b4[tid] = w[kP_B4 + tid];
  }
  if (tid < kLearnOut) {
    S.val[tid] = 0.;
  }
  float g2[4][4] = {}, g3[4][4] = {}, g1[4] = {}, g4[2] = {};
  float gb1 = 0.f, gb2 = 0.f, gb3 = 0.f, gb4 = 0.f;
  double sq = 0.;
  for (long long tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const long long r0 = tile * kTrainRows;
    __syncthreads();  // the previous tile's readers are done
    if (T.tuples) {
      if (tid < kTrainRows) {
        float x[16] = {};
        float ell = 0.f, g = 0.f;
        if (r0 + tid < T.rows) {
          float t[16];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            t[4 * q] = t4[q].x;
            t[4 * q + 1] = t4[q].y;
            t[4 * q + 2] = t4[q].z;
            t[4 * q + 3] = t4[q].w;
          }
#pragma unroll
          for (int k = 0; k < kLearnIn; ++k) {
            x[k] = (t[k] - nrm.x_mean[k]) * nrm.x_inv_std[k];
          }
          const BaseVars bv = base_vars(t, nrm);
          ell = bv.ell;
          g = bv.g;
#pragma unroll
          for (int k = 0; k < kLearnOut; ++k) {
            S.Y[tid * 8 + k] = t[kLearnIn + k];
          }
        }
        load_row(T, r0 + (long long)gridDim.x * kTrainRows + tid, t4, true);  // of the CTA's next tile
        S.bell[tid] = ell;
        S.bg[tid] = g;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          S.X[tid * kTX + k] = x[k];
        }
      }
      __syncthreads();
      // residual targets: one (row, output) a thread, the output the same over
      // a warp (the baseline's coefficients are read from the constant bank)
      {
        static_assert(kTrainThreads == kTrainRows * 8, "one (row, output) a thread");
        const int k = tid / kTrainRows, r = tid % kTrainRows;
        float y = 0.f;
        if (k < kLearnOut && r0 + r < T.rows) {
          float xn[kLearnIn];
#pragma unroll
          for (int q = 0; q < kLearnIn; ++q) {
            xn[q] = S.X[r * kTX + q];
          }
          BaseVars bv;
          bv.ell = S.bell[r];
          bv.g = S.bg[r];
          y = (S.Y[r * 8 + k] - learn_base(nrm, k, xn, bv) - nrm.y_mean[k]) / nrm.y_std[k];
        }
        S.Y[r * 8 + k] = y;
      }
    } else {
      for (int i = tid; i < kTrainRows * 16; i += kTrainThreads) {
        const bool in = r0 + (i >> 4) < T.rows;
        S.X[(i >> 4) * kTX + (i & 15)] = in ? T.X[r0 * 16 + i] : 0.f;
        if (i < kTrainRows * 8) {
          S.Y[i] = r0 + (i >> 3) < T.rows ? T.Y[r0 * 8 + i] : 0.f;
        }
      }
    }
    __syncthreads();
    layer_fwd<16, kTX>(S.X, S.W1, S.b1, S.H1, S.A1, tx, ty, quant);
    __syncthreads();
    layer_fwd<64, kTP>(S.A1, S.W2, S.b2, S.H2, S.A2, tx, ty, quant);
    __syncthreads();
    layer_fwd<64, kTP>(S.A2, S.W3, S.b3, S.H3, S.A3, tx, ty, quant);
    __syncthreads();
    // output layer and the loss: one (row, output) a thread
    float l = 0.f;
    {
      const int r = tid >> 3, k = tid & 7;
      float acc = 0.f;
#pragma unroll 4
      for (int c = 0; c < 64; c += 4) {
        const float4 a = ld4(S.A3 + r * kTP + c), v = ld4(S.W4 + k * kTP + c);
        acc = fmaf(a.x, v.x, acc);
        acc = fmaf(a.y, v.y, acc);
        acc = fmaf(a.z, v.z, acc);
        acc = fmaf(a.w, v.w, acc);
      }
      float dy = 0.f;
      if (k < kLearnOut && r0 + r < T.rows) {
        const float yp = acc + S.b4[k];
        const float d = yp - S.Y[r * 8 + k];
        if (BACK) {
          dy = 2.f * d / (float)(T.rows * kLearnOut);
          l += d * d;
        } else {
          const double a = yp * nrm.y_std[k] + nrm.y_mean[k];
          const double t = S.Y[r * 8 + k] * nrm.y_std[k] + nrm.y_mean[k];
          sq += (a - t) * (a - t);
        }
      }
      if (BACK) {
        S.dY[r * kTY + k] = dy;
      }
    }
    if (!BACK) {
      continue;
    }
    if (loss) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        l += __shfl_down_sync(0xffffffffu, l, o);
      }
      if ((tid & 31) == 0) {
        atomicAdd(loss, (double)l);
      }
    }
    __syncthreads();
    // layer 4: 8 x 64, output ht / 32, columns 2 (ht % 32)
    {
      const int n = ht >> 5, c = 2 * (ht & 31);
#pragma unroll 4
      for (int r = hr0; r < hr0 + kTrainRows / 2; ++r) {
        const float d = S.dY[r * kTY + n];
        const float2 a = *reinterpret_cast<const float2*>(S.A3 + r * kTP + c);
        g4[0] = fmaf(d, a.x, g4[0]);
        g4[1] = fmaf(d, a.y, g4[1]);
      }
      if (tid < 64) {
        gb4 += col_part(S.dY, kTY, tid & 7, tid >> 3);
      }
    }
    layer_bwd<8, kTY>(S.dY, S.W4, S.H3, S.dH, tx, ty);
    layer_dw(S.dH, S.A2, g3, tx, wy, hr0);
    gb3 += col_part(S.dH, kTP, tid & 63, tid >> 6);
    layer_bwd<64, kTP>(S.dH, S.W3, S.H2, S.dH, tx, ty);
    layer_dw(S.dH, S.A1, g2, tx, wy, hr0);
    gb2 += col_part(S.dH, kTP, tid & 63, tid >> 6);
    layer_bwd<64, kTP>(S.dH, S.W2, S.H1, S.dH, tx, ty);
    // layer 1: 64 x 16, output ht / 4, columns 4 (ht % 4)
    {
      const int n = ht >> 2, c = 4 * (ht & 3);
#pragma unroll 4
      for (int r = hr0; r < hr0 + kTrainRows / 2; ++r) {
        const float d = S.dH[r * kTP + n];
        const float4 x = ld4(S.X + r * kTX + c);
        g1[0] = fmaf(d, x.x, g1[0]);
        g1[1] = fmaf(d, x.y, g1[1]);
        g1[2] = fmaf(d, x.z, g1[2]);
        g1[3] = fmaf(d, x.w, g1[3]);
      }
    }
    gb1 += col_part(S.dH, kTP, tid & 63, tid >> 6);
  }
  if (!BACK) {
    // the lanes of an output: 4 in a warp
    sq += __shfl_xor_sync(0xffffffffu, sq, 8);
    sq += __shfl_xor_sync(0xffffffffu, sq, 16);
    if ((tid & 31) < kLearnOut) {
      atomicAdd(&S.val[tid & 31], sq);
    }
    __syncthreads();
    if (tid < kLearnOut) {
      atomicAdd(&val[tid], S.val[tid]);
    }
    return;
  }
  // the second half's sums to the first through the activations' tiles
  float* X = S.H1;
  __syncthreads();
  if (tid >= 256) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        X[(4 * i + j) * 256 + ht] = g2[i][j];
        X[(16 + 4 * i + j) * 256 + ht] = g3[i][j];
      }
      X[(32 + i) * 256 + ht] = g1[i];
    }
    X[36 * 256 + ht] = g4[0];
    X[37 * 256 + ht] = g4[1];
  }
  __syncthreads();
  float* P = part + (size_t)blockIdx.x * kP_N;
  if (tid < 256) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        g2[i][j] += X[(4 * i + j) * 256 + ht];
        g3[i][j] += X[(16 + 4 * i + j) * 256 + ht];
      }
      g1[i] += X[(32 + i) * 256 + ht];
      const int o = (4 * wy + i) * 64 + 4 * tx;
      *reinterpret_cast<float4*>(P + kP_W2 + o) = make_float4(g2[i][0], g2[i][1], g2[i][2], g2[i][3]);
      *reinterpret_cast<float4*>(P + kP_W3 + o) = make_float4(g3[i][0], g3[i][1], g3[i][2], g3[i][3]);
    }
    g4[0] += X[36 * 256 + ht];
    g4[1] += X[37 * 256 + ht];
    *reinterpret_cast<float4*>(P + kP_W1 + 4 * ht) = make_float4(g1[0], g1[1], g1[2], g1[3]);
    *reinterpret_cast<float2*>(P + kP_W4 + 2 * ht) = make_float2(g4[0], g4[1]);
  }
  const float gb[4] = {gb1, gb2, gb3, gb4};
  const int at[4] = {kP_B1, kP_B2, kP_B3, kP_B4};
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int cols = q < 3 ? 64 : 8;  // the output layer's parts lie in the first 64 threads
    __syncthreads();
    S.red[tid] = gb[q];
    __syncthreads();
    if (tid < cols) {
      float v = 0.f;
#pragma unroll
      for (int p = 0; p < 8; ++p) {
        v += S.red[p * cols + tid];
      }
      P[at[q] + tid] = v;
    }
  }
}

__device__ __forceinline__ bool is_bias(int i)
{
  return (i >= kP_B1 && i < kP_W2) || (i >= kP_B2 && i < kP_W3) || (i >= kP_B3 && i < kP_W4) || i >= kP_B4;
}

struct AdamStep {
  float lr, b1, b2, eps, bc1, bc2;
};

// The gradient as the sum of `parts` partials, eight lanes a parameter, and
// Adam (step: null for the gradient alone); wq = the bf16-rounded weights
// used by the forward pass (biases exact).
__global__ void __launch_bounds__(256) k_train_update(const float* part, int parts, float* p, float* wq, float* g, float* m,
                                                      float* v, int apply, AdamStep A, int quant)
{
  const int i = blockIdx.x * 32 + (threadIdx.x & 31);  // a warp reads 32 neighbouring parameters
  const int q = threadIdx.x >> 5;
  __shared__ float red[8][32];
  float s = 0.f;
  if (i < kP_N) {
#pragma unroll 4
    for (int c = q; c < parts; c += 8) {
      s += part[(size_t)c * kP_N + i];
    }
  }
  red[q][threadIdx.x & 31] = s;
  __syncthreads();
  if (q != 0 || i >= kP_N) {
    return;
  }
  float gi = 0.f;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    gi += red[c][threadIdx.x & 31];
  }
  g[i] = gi;
  if (!apply) {
    return;
  }
  const float mi = A.b1 * m[i] + (1.f - A.b1) * gi;
  const float vi = A.b2 * v[i] + (1.f - A.b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  const float pi = p[i] - A.lr * (mi / A.bc1) / (sqrtf(vi / A.bc2) + A.eps);
  p[i] = pi;
  wq[i] = (quant && !is_bias(i)) ? bf16r(pi) : pi;
}

__global__ void k_quantize(const float* p, float* wq, int n, int quant)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    wq[i] = (quant && !is_bias(i)) ? bf16r(p[i]) : p[i];
  }
}

}  // namespace pmp
