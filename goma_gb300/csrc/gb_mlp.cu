// A small fully-connected network (FP32) trained on the GPU by hand-written
// kernels: forward, backward and Adam.  It predicts the next Newton initial
// guess of a parameter continuation from (node coordinates, parameter); the
// reference's own predictor (ac_conti.c ALC_ZEROTH / ALC_FIRST,
// src/ac_conti.c:759-784) stays the fallback and the converged Newton
// solve always decides.
//
// Layout: layer l maps width_in -> width_out with W_l [out][in] row-major and
// b_l [out]; hidden layers use tanh, the last is linear.  All parameters
// live in one flat FP32 buffer (and gradients / Adam moments in three more),
// so the host can read, write and checksum them in one copy.
//
// The products run on the FP32 pipe in FP32 FMA.  A sum over k is split in a
// fixed way (two groups of k in the tiled kernel, lanes in the narrow ones,
// parts of the batch for the gradients) and added in a fixed order: results do
// not depend on timing, and the predictor's accuracy is that of FP32 arithmetic.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <vector>

#include "../../include/gb_newton.h"
#include "gb_context.h"
#include "gb_launch.cuh"

namespace gb {

constexpr int TM = 64, TN = 64, TK = 32;
constexpr int kMaxSplit = 32;  // batch splits of the weight-gradient product
constexpr int kNarrow = 8;     // widths up to this take the narrow kernels

// ---- tiled product C[M][N] = sum_k A(m, k) B(k, n)
//
// Operand tiles (64 rows, 32 k) go through registers to shared memory as
// S[k][row], rows in 16-byte pieces moved by 4 * (k / 4 % 8): the transposing
// stores of k-contiguous operands and all loads then hit distinct banks.  256
// threads in two groups, each with half of a tile's k and 8 x 4 outputs a
// thread, in packed FMA (fma.rn.f32x2, 15 % faster than single ones): 16 FMA
// instructions per 3 shared loads.  At the end the groups add their sums and
// each keeps half of the rows.  The next tile's global loads are in flight
// while a tile is multiplied.
//
// Bound by the FP32 pipe, 128 FMA a clock and SM: 4096 x 256 x 256 takes 7.2
// us at that rate.  64 x 64 tiles make 256 blocks of it, at most two on an SM
// (84 %), and the second group keeps the pipe fed with so few blocks: 14.5
// us, 16.5 us with one group, 21.5 us (forward 25 us) with 4 x 4 outputs, twice
// the shared loads and no prefetch.  8 x 8 outputs in four groups: 17.5 us.
// 34,306 rows: 100 us, 58 % of the pipe.

// A thread's two pieces of 16 bytes of the tiles of one operand.  KC:
// P[row][k], ld = row stride; else P[k][row], ld = k stride.  Whole aligned
// tiles take the short path: the checks of the others were 40 % of the
// instructions.
template <bool KC>
struct TileLoad {
  const float *p;  // the first piece
  int64_t second;  // the other from it
  int64_t ld;
  int r, k, rows, kend;
  bool whole;
  __device__ __forceinline__ TileLoad(const float *P, int ld_, int r0, int rows_, int k0, int kend_,
                                      bool vec)
      : ld(ld_), rows(rows_), kend(kend_), whole(vec && r0 + TM <= rows_) {
    const int t = threadIdx.x;
    r = KC ? r0 + t / (TK / 4) : r0 + (t % 16) * 4;
    k = KC ? k0 + (t % (TK / 4)) * 4 : k0 + t / 16;
    p = KC ? P + (int64_t)r * ld + k : P + (int64_t)k * ld + r;
    second = KC ? 32 * ld : TK / 2 * ld;
  }
  // the tile at k0, then on to the next
  __device__ __forceinline__ void next(int k0, float4 (&v)[2]) {
    if (whole && k0 + TK <= kend) {
      v[0] = *reinterpret_cast<const float4 *>(p);
      v[1] = *reinterpret_cast<const float4 *>(p + second);
    } else {
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const float *x = p + u * second;
        const int left = KC ? (r + 32 * u < rows ? kend - k : 0)
                            : (k + TK / 2 * u < kend ? rows - r : 0);
        v[u].x = left > 0 ? x[0] : 0.f;
        v[u].y = left > 1 ? x[1] : 0.f;
        v[u].z = left > 2 ? x[2] : 0.f;
        v[u].w = left > 3 ? x[3] : 0.f;
      }
    }
    k += TK;
    p += KC ? TK : TK * ld;
  }
};

// the move of the pieces of row k
__device__ __forceinline__ int tile_swz(int k) { return ((k >> 2) & 7) * 4; }

template <bool KC>
__device__ __forceinline__ void tile_store(float (*S)[TM], const float4 (&v)[2]) {
  const int t = threadIdx.x;
#pragma unroll
  for (int u = 0; u < 2; u++) {
    if (KC) {
      const int k = (t % 8) * 4, r = (t / 8 + 32 * u) ^ tile_swz(k);
      S[k][r] = v[u].x;
      S[k + 1][r] = v[u].y;
      S[k + 2][r] = v[u].z;
      S[k + 3][r] = v[u].w;
    } else {
      const int k = t / 16 + 16 * u, r = ((t % 16) * 4) ^ tile_swz(k);
      *reinterpret_cast<float4 *>(&S[k][r]) = v[u];
    }
  }
}

// two FP32 FMA, each rounded like fmaf, and two adds
__device__ __forceinline__ void fma2(unsigned long long &d, unsigned long long a,
                                     unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long dup2(float x) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float2 split2(unsigned long long x) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(x));
  return r;
}

// MLP_FORWARD  C = A W^T + E[n], with act: tanh of it   (A [M][K], W [N][K])
// MLP_BACK     C = (A W) (1 - E[m][n]^2)                (A [M][K], W [K][N])
// MLP_GRAD     split z of the sum over the batch k in chunks of kchunk, A
//              [K][M] and B [K][N], to C + z (M N + M), followed by the split's
//              sums of A over k (the bias gradient); grad_sum_kernel adds the
//              splits in a fixed order, so the result is deterministic
enum { MLP_FORWARD, MLP_BACK, MLP_GRAD };

template <int OP>
__global__ void __launch_bounds__(256, 2)
    mlp_gemm_kernel(int M, int N, int K, const float *A, const float *B, const float *E,
                    float *__restrict__ C, int act, int kchunk, bool vec_a, bool vec_b,
                    bool vec_c) {
  dependent_begin();
  constexpr bool AK = OP != MLP_GRAD, BK = OP == MLP_FORWARD;
  union Smem {
    float t[2][2][TK][TM];         // buffer, operand
    unsigned long long x[8][256];  // the groups' exchange
    float s[256];
  };
  __shared__ __align__(16) Smem S;
  const int tid = threadIdx.x, lane = tid & 31, wp = (tid >> 5) & 3, g = tid >> 7;
  const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
  const int mi = (wp >> 1) * 32 + (lane >> 3) * 8, ni = (wp & 1) * 32 + (lane & 7) * 4;
  const int kb = OP == MLP_GRAD ? blockIdx.z * kchunk : 0;
  const int ke = OP == MLP_GRAD ? min(K, kb + kchunk) : K;
  const int lda = AK ? K : M, ldb = BK ? K : N;
  if (OP == MLP_GRAD) C += (int64_t)blockIdx.z * ((int64_t)M * N + M);
  unsigned long long acc[4][4] = {};  // row pair i, column j
  float cs = 0.f;
  float4 va[2], vb[2];
  TileLoad<AK> la(A, lda, m0, M, kb, ke, vec_a);
  TileLoad<BK> lb(B, ldb, n0, N, kb, ke, vec_b);
  la.next(kb, va);
  lb.next(kb, vb);
  int buf = 0;
  for (int k0 = kb; k0 < ke; k0 += TK, buf ^= 1) {
    float(*As)[TM] = S.t[buf][0], (*Bs)[TN] = S.t[buf][1];
    tile_store<AK>(As, va);
    tile_store<BK>(Bs, vb);
    __syncthreads();
    if (k0 + TK < ke) {
      la.next(k0 + TK, va);
      lb.next(k0 + TK, vb);
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {  // four k with the same moves
      const int k4 = g * 16 + q * 4, sw = tile_swz(k4);
      const float *pa0 = &As[k4][mi ^ sw], *pa1 = &As[k4][(mi + 4) ^ sw];
      const float *pb = &Bs[k4][ni ^ sw];
#pragma unroll
      for (int kk = 0; kk < 4; kk++) {
        const ulonglong2 a0 = *reinterpret_cast<const ulonglong2 *>(pa0 + kk * TM);
        const ulonglong2 a1 = *reinterpret_cast<const ulonglong2 *>(pa1 + kk * TM);
        const float4 b = *reinterpret_cast<const float4 *>(pb + kk * TN);
        const unsigned long long a[4] = {a0.x, a0.y, a1.x, a1.y};
        const unsigned long long d[4] = {dup2(b.x), dup2(b.y), dup2(b.z), dup2(b.w)};
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
          for (int j = 0; j < 4; j++) fma2(acc[i][j], a[i], d[j]);
      }
    }
    if (OP == MLP_GRAD && blockIdx.x == 0) {  // sums of A: a column, eight k
      const int k8 = (tid >> 6) * 8;
      float ts = 0.f;
#pragma unroll
      for (int k = 0; k < 8; k++) ts += As[k8 + k][(tid & 63) ^ tile_swz(k8 + k)];
      cs += ts;
    }
    // the buffer after next is written only after the next barrier
  }
  // group 0 keeps the first four rows of the groups' sums, group 1 the others
  unsigned long long r[2][4];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) S.x[i * 4 + j][tid] = g ? acc[i][j] : acc[i + 2][j];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 4; j++)
      r[i][j] = add2(g ? acc[i + 2][j] : acc[i][j], S.x[i * 4 + j][tid ^ 128]);
  const int gm0 = m0 + mi + 4 * g, gn = n0 + ni;
  float v[4][4];
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const float2 x = split2(r[i][j]);
      v[2 * i][j] = x.x;
      v[2 * i + 1][j] = x.y;
    }
  if (OP == MLP_FORWARD) {
    float e[4];
#pragma unroll
    for (int j = 0; j < 4; j++) e[j] = gn + j < N ? E[gn + j] : 0.f;
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int j = 0; j < 4; j++) {
        v[i][j] += e[j];
        if (act) v[i][j] = tanhf(v[i][j]);
      }
  }
  // whole tiles in pieces of 16 bytes
  if (vec_c && m0 + TM <= M && n0 + TN <= N) {
    if (OP == MLP_BACK) {
      float4 h[4];
#pragma unroll
      for (int i = 0; i < 4; i++)
        h[i] = *reinterpret_cast<const float4 *>(E + (int64_t)(gm0 + i) * N + gn);
#pragma unroll
      for (int i = 0; i < 4; i++) {
        v[i][0] *= 1.f - h[i].x * h[i].x;
        v[i][1] *= 1.f - h[i].y * h[i].y;
        v[i][2] *= 1.f - h[i].z * h[i].z;
        v[i][3] *= 1.f - h[i].w * h[i].w;
      }
    }
#pragma unroll
    for (int i = 0; i < 4; i++)
      *reinterpret_cast<float4 *>(C + (int64_t)(gm0 + i) * N + gn) =
          make_float4(v[i][0], v[i][1], v[i][2], v[i][3]);
  } else {
    for (int i = 0; i < 4; i++)
      for (int j = 0; j < 4; j++) {
        if (gm0 + i >= M || gn + j >= N) continue;
        const int64_t o = (int64_t)(gm0 + i) * N + gn + j;
        C[o] = OP == MLP_BACK ? v[i][j] * (1.f - E[o] * E[o]) : v[i][j];
      }
  }
  if (OP == MLP_GRAD && blockIdx.x == 0) {
    __syncthreads();
    S.s[tid] = cs;
    __syncthreads();
    if (tid < TM && m0 + tid < M)
      C[(int64_t)M * N + m0 + tid] =
          (S.s[tid] + S.s[64 + tid]) + (S.s[128 + tid] + S.s[192 + tid]);
  }
}

// ---- layers with at most kNarrow outputs or inputs, where a 64 x 64 tile
// would be nearly empty

// C[M][N] = A[M][K] W[N][K]^T + bias (tanh): a warp per row, lanes over k
// (4096 x 1 x 256: 4 us, 10 us as a tile)
__global__ void __launch_bounds__(256)
    mlp_forward_narrow_kernel(int M, int N, int K, const float *A, const float *W,
                              const float *bias, float *__restrict__ C, int act) {
  dependent_begin();
  const int m = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (m >= M) return;
  float s[kNarrow] = {};
  const float *a = A + (int64_t)m * K;
  for (int k = lane; k < K; k += 32) {
    const float x = a[k];
#pragma unroll
    for (int j = 0; j < kNarrow; j++)
      if (j < N) s[j] = fmaf(x, W[(int64_t)j * K + k], s[j]);
  }
#pragma unroll
  for (int j = 0; j < kNarrow; j++)
    if (j < N) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s[j] += __shfl_xor_sync(0xffffffffu, s[j], o);
      float v = s[j] + bias[j];
      if (act) v = tanhf(v);
      if (lane == 0) C[(int64_t)m * N + j] = v;
    }
}

// C[M][K] = (D[M][N] W[N][K]) (1 - H^2), N <= kNarrow: a thread keeps its
// column of W over its rows
__global__ void __launch_bounds__(256)
    mlp_back_narrow_kernel(int M, int N, int K, const float *D, const float *W, const float *H,
                           float *__restrict__ C) {
  dependent_begin();
  for (int k = blockIdx.x * 256 + threadIdx.x; k < K; k += gridDim.x * 256) {
    float w[kNarrow];
#pragma unroll
    for (int j = 0; j < kNarrow; j++) w[j] = j < N ? W[(int64_t)j * K + k] : 0.f;
#pragma unroll 4
    for (int m = blockIdx.y; m < M; m += gridDim.y) {
      const float h = H[(int64_t)m * K + k];
      float s = 0.f;
#pragma unroll
      for (int j = 0; j < kNarrow; j++)
        if (j < N) s = fmaf(D[(int64_t)m * N + j], w[j], s);
      C[(int64_t)m * K + k] = s * (1.f - h * h);
    }
  }
}

// Split blockIdx.y of dW[N][K] = D^T X and of the sums of D where D or X
// (wide_is_d) has at most kNarrow columns: a thread per column of the wide
// one, four groups of rows a block, 32 rows of the narrow one at a time in
// shared memory (4096 rows, 256 x 8: 5 us, 21 us as tiles and column sums).
__global__ void __launch_bounds__(256)
    mlp_grad_narrow_kernel(int M, int N, int K, const float *D, const float *X,
                           float *__restrict__ G, int mchunk, int wide_is_d) {
  dependent_begin();
  constexpr int R = 32;
  __shared__ __align__(16) float q[4][R][kNarrow];
  __shared__ float red[4][kNarrow + 1][64];
  const int c = threadIdx.x & 63, grp = threadIdx.x >> 6, i = blockIdx.x * 64 + c;
  const int nw = wide_is_d ? N : K, nn = wide_is_d ? K : N;
  const float *P = wide_is_d ? D : X, *Q = wide_is_d ? X : D;
  const int per = (mchunk + 3) / 4, b0 = blockIdx.y * mchunk;
  const int mb = b0 + grp * per, me = min(min(M, b0 + mchunk), mb + per);
  G += (int64_t)blockIdx.y * ((int64_t)N * K + N);
  float s[kNarrow] = {}, sd = 0.f;
  for (int r0 = 0; r0 < per; r0 += R) {
    __syncthreads();
    for (int t = c; t < R * kNarrow; t += 64) {
      const int m = mb + r0 + t / kNarrow, j = t % kNarrow;
      q[grp][t / kNarrow][j] = m < me && j < nn ? Q[(int64_t)m * nn + j] : 0.f;
    }
    __syncthreads();
    if (i >= nw) continue;
    const float *p = P + (int64_t)(mb + r0) * nw + i;
    auto add = [&](int r, float x) {
      const float4 u = *reinterpret_cast<const float4 *>(&q[grp][r][0]);
      const float4 v = *reinterpret_cast<const float4 *>(&q[grp][r][4]);
      const float y[kNarrow] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < kNarrow; j++) s[j] = fmaf(x, y[j], s[j]);
      sd += wide_is_d ? x : q[grp][r][c & (kNarrow - 1)];
    };
    if (mb + r0 + R <= me) {  // 16 loads in flight; under a condition one
      for (int r = 0; r < R; r += 16) {
        float x[16];
#pragma unroll
        for (int t = 0; t < 16; t++) x[t] = p[(int64_t)(r + t) * nw];
#pragma unroll
        for (int t = 0; t < 16; t++) add(r + t, x[t]);
      }
    } else {
      for (int r = 0; mb + r0 + r < me; r++) add(r, p[(int64_t)r * nw]);
    }
  }
#pragma unroll
  for (int j = 0; j < kNarrow; j++) red[grp][j][c] = s[j];
  red[grp][kNarrow][c] = sd;
  __syncthreads();
  if (grp != 0 || i >= nw) return;
#pragma unroll
  for (int j = 0; j < kNarrow; j++) {
    if (j >= nn) break;
    const float v = (red[0][j][c] + red[1][j][c]) + (red[2][j][c] + red[3][j][c]);
    G[wide_is_d ? (int64_t)i * K + j : (int64_t)j * K + i] = v;
  }
  if (i < N)
    G[(int64_t)N * K + i] = (red[0][kNarrow][c] + red[1][kNarrow][c]) +
                            (red[2][kNarrow][c] + red[3][kNarrow][c]);
}

// aligned for the 16-byte loads of tile_load
static bool vec4(const float *p, int ld) { return (ld & 3) == 0 && ((uintptr_t)p & 15) == 0; }

// act(X W^T + b) of one layer
static void launch_layer(const float *X, int B, int K, int N, const float *W, const float *b,
                         float *Y, int act, cudaStream_t st) {
  if (N <= kNarrow) {
    launch_dependent(mlp_forward_narrow_kernel, (B + 7) / 8, 256, 0, st, B, N, K, X, W, b, Y, act);
    return;
  }
  dim3 grid((N + TN - 1) / TN, (B + TM - 1) / TM);
  launch_dependent(mlp_gemm_kernel<MLP_FORWARD>, grid, 256, 0, st, B, N, K, X, W, b, Y, act, 0,
                   vec4(X, K), vec4(W, K), vec4(Y, N));
}

// g[i] = sum over the splits z (in order) of P[z][i]
__global__ void grad_sum_kernel(int nsplit, int n, const float *P, float *__restrict__ g) {
  dependent_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float s = 0.f;
#pragma unroll 8
  for (int z = 0; z < nsplit; z++) s += P[(int64_t)z * n + i];
  g[i] = s;
}

// dY = 2 mask (Y - T) / msum ; per-block partial of sum mask (Y-T)^2
__global__ void loss_grad_kernel(int n, const float *Y, const float *__restrict__ T,
                                 const float *__restrict__ mask, float inv_msum,
                                 float *__restrict__ dY, float *__restrict__ part) {
  dependent_begin();
  __shared__ float sh[256];
  float s = 0.f;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float d = (Y[i] - T[i]) * mask[i];
    dY[i] = 2.f * d * inv_msum;
    s += d * d;
  }
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = sh[0];
}

__global__ void adam_kernel(int n, float *__restrict__ w, const float *g,
                            float *__restrict__ m, float *__restrict__ v, float lr, float b1,
                            float b2, float eps, float c1, float c2) {
  dependent_begin();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    w[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  }
}

// All layers' gradients from their splits and, with adam, the parameters'
// step: one launch for the whole network instead of a sum a layer and Adam (a
// training step of 8-256-256-256-1: 18 -> 14 launches, 14 -> 5 us of sums and
// step).
constexpr int kMaxFused = 16;  // layers
struct LayerTab {
  int n = 0, off[kMaxFused] = {}, len[kMaxFused] = {};  // in the parameters
};
struct AdamArgs {
  float lr, b1, b2, eps, c1, c2;
};
__global__ void __launch_bounds__(256)
    grad_step_kernel(int n, LayerTab L, int nsplit, const float *P, float *g, bool adam,
                     float *__restrict__ w, float *__restrict__ m, float *__restrict__ v,
                     AdamArgs a) {
  dependent_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int off = 0, len = 0;
#pragma unroll
  for (int l = 0; l < kMaxFused; l++)
    if (l < L.n && i >= L.off[l]) {
      off = L.off[l];
      len = L.len[l];
    }
  const float *p = P + (int64_t)off * nsplit + (i - off);
  float s = 0.f;
#pragma unroll 8
  for (int z = 0; z < nsplit; z++) s += p[(int64_t)z * len];
  g[i] = s;
  if (!adam) return;
  const float mi = a.b1 * m[i] + (1.f - a.b1) * s;
  const float vi = a.b2 * v[i] + (1.f - a.b2) * s * s;
  m[i] = mi;
  v[i] = vi;
  w[i] -= a.lr * (mi / a.c1) / (sqrtf(vi / a.c2) + a.eps);
}

// rows idx[b] of X[n][ni], T[n][no] and K[n][no] -> Xb, Tb, Kb
__global__ void gather_rows_kernel(int B, int ni, int no, const int *__restrict__ idx,
                                   const float *__restrict__ X, const float *__restrict__ T,
                                   const float *__restrict__ K, float *__restrict__ Xb,
                                   float *__restrict__ Tb, float *__restrict__ Kb) {
  dependent_begin();
  const int64_t w = ni + 2 * no;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < B * w;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t b = t / w, r = idx[b];
    const int j = (int)(t - b * w);
    if (j < ni)
      Xb[b * ni + j] = X[r * ni + j];
    else if (j < ni + no)
      Tb[b * no + j - ni] = T[r * no + j - ni];
    else
      Kb[b * no + j - ni - no] = K[r * no + j - ni - no];
  }
}

struct Mlp {
  std::vector<int> width;  // n_in, hidden..., n_out
  int nparam = 0;
  std::vector<int> woff, boff;
  float *d_w = nullptr, *d_g = nullptr, *d_m = nullptr, *d_v = nullptr;
  int cap = 0;                       // batch capacity of the activations
  std::vector<float *> act;          // per layer output [cap][width]
  float *d_dA = nullptr, *d_dB = nullptr;  // backward scratch [cap][maxw]
  float *d_part = nullptr, *h_part = nullptr;
  float *d_xb = nullptr, *d_tb = nullptr, *d_mb = nullptr;
  float *d_split = nullptr;          // gradient partial sums [kMaxSplit][maxw * (maxw + 1)]
  int *d_idx = nullptr;
  int adam_t = 0;
  int dev = 0;                       // the device the network lives on
  cudaStream_t st = nullptr;
  // orders a caller's stream after the network's own stream and back
  cudaEvent_t ev_own = nullptr, ev_caller = nullptr;
  ~Mlp() {
    cudaFree(d_w);
    cudaFree(d_g);
    cudaFree(d_m);
    cudaFree(d_v);
    for (float *a : act) cudaFree(a);
    cudaFree(d_dA);
    cudaFree(d_dB);
    cudaFree(d_part);
    cudaFree(d_xb);
    cudaFree(d_tb);
    cudaFree(d_mb);
    cudaFree(d_idx);
    cudaFree(d_split);
    if (h_part) cudaFreeHost(h_part);
    if (ev_own) cudaEventDestroy(ev_own);
    if (ev_caller) cudaEventDestroy(ev_caller);
    if (st) cudaStreamDestroy(st);
  }
  int maxw() const {
    int m = 0;
    for (int w : width) m = w > m ? w : m;
    return m;
  }
  int layers() const { return (int)width.size() - 1; }
  // the splits of all layers at once: small networks
  bool fused() const { return layers() <= kMaxFused && nparam <= (2 << 20); }
  int ensure(int B) {
    if (B <= cap) return 0;
    for (float *a : act) cudaFree(a);
    act.assign(layers(), nullptr);
    cudaFree(d_dA);
    cudaFree(d_dB);
    cudaFree(d_xb);
    cudaFree(d_tb);
    cudaFree(d_mb);
    cudaFree(d_idx);
    for (int l = 0; l < layers(); l++)
      if (cudaMalloc(&act[l], sizeof(float) * (size_t)B * width[l + 1]) != cudaSuccess)
        return fail("MLP activations");
    const size_t mw = (size_t)B * maxw();
    if (cudaMalloc(&d_dA, sizeof(float) * mw) != cudaSuccess ||
        cudaMalloc(&d_dB, sizeof(float) * mw) != cudaSuccess ||
        cudaMalloc(&d_xb, sizeof(float) * (size_t)B * width[0]) != cudaSuccess ||
        cudaMalloc(&d_tb, sizeof(float) * (size_t)B * width.back()) != cudaSuccess ||
        cudaMalloc(&d_mb, sizeof(float) * (size_t)B * width.back()) != cudaSuccess ||
        cudaMalloc(&d_idx, sizeof(int) * (size_t)B) != cudaSuccess)
      return fail("MLP scratch");
    if (!d_split &&
        cudaMalloc(&d_split, sizeof(float) * kMaxSplit *
                                 (fused() ? (size_t)nparam : (size_t)maxw() * (maxw() + 1))) !=
            cudaSuccess)
      return fail("MLP scratch");
    cap = B;
    return 0;
  }
  void forward(const float *X, int B) {
    const float *in = X;
    for (int l = 0; l < layers(); l++) {
      launch_layer(in, B, width[l], width[l + 1], d_w + woff[l], d_w + boff[l], act[l],
                   l + 1 < layers() ? 1 : 0, st);
      in = act[l];
    }
  }
  // gradient of sum mask (Y - T)^2 / sum(mask) into d_g; with loss != NULL
  // also waits for and returns the loss (host)
  // and with adam takes the step
  int backward(const float *X, const float *T, const float *Mk, int B, float msum, float *loss,
               const AdamArgs *adam = nullptr) {
    const int nl = layers(), no = width.back();
    const int nb = 64;
    launch_dependent(loss_grad_kernel, nb, 256, 0, st, B * no, act[nl - 1], T, Mk, 1.f / msum,
                     d_dA, d_part);
    float *dcur = d_dA, *dnext = d_dB;
    const int nsplit = std::max(1, std::min(kMaxSplit, B / 128));
    const int mchunk = ((B + nsplit - 1) / nsplit + TK - 1) / TK * TK;
    LayerTab tab;
    for (int l = nl - 1; l >= 0; l--) {
      const int K = width[l], N = width[l + 1];
      const float *Hin = l == 0 ? X : act[l - 1];
      // dW_l = dZ^T Hin  [N][K] and db_l = colsum dZ, which follows it in
      // d_g; the batch split over up to kMaxSplit CTA layers so that the grid
      // covers the GPU
      float *part = nsplit == 1 ? d_g + woff[l]
                                : d_split + (fused() ? (size_t)woff[l] * nsplit : 0);
      if (K <= kNarrow || N <= kNarrow) {
        const int wide_is_d = K <= kNarrow;
        dim3 g1(((wide_is_d ? N : K) + 63) / 64, nsplit);
        launch_dependent(mlp_grad_narrow_kernel, g1, 256, 0, st, B, N, K, dcur, Hin, part, mchunk,
                         wide_is_d);
      } else {
        dim3 g1((K + TN - 1) / TN, (N + TM - 1) / TM, nsplit);
        launch_dependent(mlp_gemm_kernel<MLP_GRAD>, g1, 256, 0, st, N, K, B, dcur, Hin, nullptr,
                         part, 0, mchunk, vec4(dcur, N), vec4(Hin, K),
                         vec4(part, K) && (nsplit == 1 || (N & 3) == 0));
      }
      if (nsplit > 1 && !fused())
        launch_dependent(grad_sum_kernel, (N * K + N + 255) / 256, 256, 0, st, nsplit, N * K + N,
                         d_split, d_g + woff[l]);
      if (l == 0) break;
      // dZ_{l-1} = (dZ W_l) (1 - H^2)  [B][K]
      const float *W = d_w + woff[l];
      if (N <= kNarrow) {
        dim3 g2((K + 255) / 256, std::min(B, 1216));
        launch_dependent(mlp_back_narrow_kernel, g2, 256, 0, st, B, N, K, dcur, W, act[l - 1],
                         dnext);
      } else {
        dim3 g2((K + TN - 1) / TN, (B + TM - 1) / TM);
        launch_dependent(mlp_gemm_kernel<MLP_BACK>, g2, 256, 0, st, B, K, N, dcur, W, act[l - 1],
                         dnext, 0, 0, vec4(dcur, N), vec4(W, K),
                         vec4(dnext, K) && vec4(act[l - 1], K));
      }
      float *t = dcur;
      dcur = dnext;
      dnext = t;
    }
    if (fused() && (nsplit > 1 || adam)) {
      tab.n = nl;
      for (int l = 0; l < nl; l++) {
        tab.off[l] = woff[l];
        tab.len[l] = width[l + 1] * (width[l] + 1);
      }
      launch_dependent(grad_step_kernel, (nparam + 255) / 256, 256, 0, st, nparam, tab, nsplit,
                       nsplit == 1 ? d_g : d_split, d_g, adam != nullptr, d_w, d_m, d_v,
                       adam ? *adam : AdamArgs{});
    } else if (adam) {
      launch_adam(*adam);
    }
    if (!loss) return 0;  // no loss wanted: nothing to wait for
    cudaMemcpyAsync(h_part, d_part, sizeof(float) * nb, cudaMemcpyDeviceToHost, st);
    cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return cuda_fail(e, "MLP backward");
    double s = 0.0;
    for (int b = 0; b < nb; b++) s += h_part[b];
    if (loss) *loss = (float)(s / msum);
    return 0;
  }
  AdamArgs adam_args(float lr, float b1, float b2, float eps) {
    adam_t++;
    return {lr, b1, b2, eps, 1.f - powf(b1, (float)adam_t), 1.f - powf(b2, (float)adam_t)};
  }
  void launch_adam(const AdamArgs &a) {
    launch_dependent(adam_kernel, 304, 256, 0, st, nparam, d_w, d_g, d_m, d_v, a.lr, a.b1, a.b2,
                     a.eps, a.c1, a.c2);
  }
};

}  // namespace gb

struct gb_mlp {
  gb::Mlp m;
};

extern "C" {

int gb_mlp_create(int n_in, int width, int hidden_layers, int n_out, unsigned long long seed,
                  gb_mlp **out) {
  if (!out || n_in <= 0 || width <= 0 || hidden_layers < 1 || n_out <= 0)
    return gb::fail("invalid MLP shape");
  *out = nullptr;
  gb_mlp *h = new (std::nothrow) gb_mlp;
  if (!h) return gb::fail("out of host memory");
  gb::Mlp &M = h->m;
  M.width.push_back(n_in);
  for (int l = 0; l < hidden_layers; l++) M.width.push_back(width);
  M.width.push_back(n_out);
  int off = 0;
  for (int l = 0; l < M.layers(); l++) {
    M.woff.push_back(off);
    off += M.width[l] * M.width[l + 1];
    M.boff.push_back(off);
    off += M.width[l + 1];
  }
  M.nparam = off;
  // Glorot-uniform weights from a fixed integer hash (splitmix64), zero biases
  std::vector<float> w(off, 0.f);
  uint64_t z = seed * 0x9E3779B97F4A7C15ull + 1;
  auto next = [&]() {
    z += 0x9E3779B97F4A7C15ull;
    uint64_t r = z;
    r = (r ^ (r >> 30)) * 0xBF58476D1CE4E5B9ull;
    r = (r ^ (r >> 27)) * 0x94D049BB133111EBull;
    r ^= r >> 31;
    return (double)(r >> 11) * (1.0 / 9007199254740992.0);
  };
  for (int l = 0; l < M.layers(); l++) {
    const int fi = M.width[l], fo = M.width[l + 1];
    const double a = std::sqrt(6.0 / (fi + fo));
    for (int i = 0; i < fi * fo; i++) w[M.woff[l] + i] = (float)((2.0 * next() - 1.0) * a);
  }
  cudaError_t e = cudaGetDevice(&M.dev);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&M.st, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&M.ev_own, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&M.ev_caller, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaMalloc(&M.d_w, sizeof(float) * off);
  if (e == cudaSuccess) e = cudaMalloc(&M.d_g, sizeof(float) * off);
  if (e == cudaSuccess) e = cudaMalloc(&M.d_m, sizeof(float) * off);
  if (e == cudaSuccess) e = cudaMalloc(&M.d_v, sizeof(float) * off);
  if (e == cudaSuccess) e = cudaMalloc(&M.d_part, sizeof(float) * 64);
  if (e == cudaSuccess) e = cudaMallocHost(&M.h_part, sizeof(float) * 64);
  if (e == cudaSuccess) e = cudaMemcpy(M.d_w, w.data(), sizeof(float) * off, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemset(M.d_m, 0, sizeof(float) * off);
  if (e == cudaSuccess) e = cudaMemset(M.d_v, 0, sizeof(float) * off);
  if (e == cudaSuccess) e = cudaMemset(M.d_g, 0, sizeof(float) * off);
  if (e != cudaSuccess) {
    delete h;
    return gb::cuda_fail(e, "MLP create");
  }
  *out = h;
  return 0;
}

void gb_mlp_destroy(gb_mlp *m) { delete m; }

int gb_mlp_num_params(const gb_mlp *m) { return m ? m->m.nparam : -1; }

int gb_mlp_get_params(const gb_mlp *m, float *host) {
  if (!m || !host) return gb::fail("NULL argument");
  cudaError_t e = cudaMemcpy(host, m->m.d_w, sizeof(float) * m->m.nparam, cudaMemcpyDeviceToHost);
  return e == cudaSuccess ? 0 : gb::cuda_fail(e, "MLP params");
}

int gb_mlp_set_params(gb_mlp *m, const float *host) {
  if (!m || !host) return gb::fail("NULL argument");
  cudaError_t e = cudaMemcpy(m->m.d_w, host, sizeof(float) * m->m.nparam, cudaMemcpyHostToDevice);
  m->m.adam_t = 0;
  cudaMemset(m->m.d_m, 0, sizeof(float) * m->m.nparam);
  cudaMemset(m->m.d_v, 0, sizeof(float) * m->m.nparam);
  return e == cudaSuccess ? 0 : gb::cuda_fail(e, "MLP params");
}

int gb_mlp_get_grads(const gb_mlp *m, float *host) {
  if (!m || !host) return gb::fail("NULL argument");
  cudaError_t e = cudaMemcpy(host, m->m.d_g, sizeof(float) * m->m.nparam, cudaMemcpyDeviceToHost);
  return e == cudaSuccess ? 0 : gb::cuda_fail(e, "MLP grads");
}

int gb_mlp_forward_device(gb_mlp *m, const float *d_x, int B, float *d_y) {
  if (!m || !d_x || !d_y || B <= 0) return gb::fail("invalid argument");
  gb::Mlp &M = m->m;
  if (M.ensure(B)) return -1;
  M.forward(d_x, B);
  cudaError_t e = cudaMemcpyAsync(d_y, M.act.back(), sizeof(float) * (size_t)B * M.width.back(),
                                  cudaMemcpyDeviceToDevice, M.st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(M.st);
  return e == cudaSuccess ? 0 : gb::cuda_fail(e, "MLP forward");
}

int gb_mlp_loss_grad_device(gb_mlp *m, const float *d_x, const float *d_t, const float *d_mask,
                            int B, float *loss) {
  if (!m || !d_x || !d_t || !d_mask || B <= 0) return gb::fail("invalid argument");
  gb::Mlp &M = m->m;
  if (M.ensure(B)) return -1;
  // sum of the mask (host side would need a copy; compute on device)
  std::vector<float> hm((size_t)B * M.width.back());
  cudaError_t e = cudaMemcpy(hm.data(), d_mask, sizeof(float) * hm.size(), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return gb::cuda_fail(e, "mask");
  double ms = 0.0;
  for (float v : hm) ms += v;
  if (ms <= 0.0) return gb::fail("empty loss mask");
  M.forward(d_x, B);
  return M.backward(d_x, d_t, d_mask, B, (float)ms, loss);
}

int gb_mlp_adam_step(gb_mlp *m, float lr, float beta1, float beta2, float eps) {
  if (!m) return gb::fail("NULL argument");
  m->m.launch_adam(m->m.adam_args(lr, beta1, beta2, eps));
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : gb::cuda_fail(e, "Adam");
}

int gb_mlp_train_device(gb_mlp *m, const float *d_x, const float *d_t, const float *d_mask,
                        int n_points, int steps, int batch, float lr, unsigned long long seed,
                        float *final_loss) {
  if (!m || !d_x || !d_t || !d_mask || n_points <= 0 || steps <= 0 || batch <= 0)
    return gb::fail("invalid argument");
  gb::Mlp &M = m->m;
  const int B = batch < n_points ? batch : n_points;
  if (M.ensure(B)) return -1;
  const int ni = M.width[0], no = M.width.back();
  std::vector<int> idx(B);
  std::vector<float> hm((size_t)n_points * no);
  cudaError_t e = cudaMemcpy(hm.data(), d_mask, sizeof(float) * hm.size(), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return gb::cuda_fail(e, "mask");
  uint64_t z = seed * 0xD1B54A32D192ED03ull + 7;
  float loss = 0.f;
  for (int s = 0; s < steps; s++) {
    // minibatch: B indices from a fixed integer hash stream
    double ms = 0.0;
    for (int b = 0; b < B; b++) {
      z += 0x9E3779B97F4A7C15ull;
      uint64_t r = z;
      r = (r ^ (r >> 30)) * 0xBF58476D1CE4E5B9ull;
      r = (r ^ (r >> 27)) * 0x94D049BB133111EBull;
      r ^= r >> 31;
      idx[b] = B == n_points ? b : (int)(r % (uint64_t)n_points);
      for (int o = 0; o < no; o++) ms += hm[(size_t)idx[b] * no + o];
    }
    if (ms <= 0.0) continue;
    e = cudaMemcpyAsync(M.d_idx, idx.data(), sizeof(int) * B, cudaMemcpyHostToDevice, M.st);
    if (e != cudaSuccess) return gb::cuda_fail(e, "batch");
    gb::launch_dependent(gb::gather_rows_kernel, 304, 256, 0, M.st, B, ni, no, M.d_idx, d_x, d_t,
                         d_mask, M.d_xb, M.d_tb, M.d_mb);
    M.forward(M.d_xb, B);
    // the loss is read back on the last step only: no per-step host wait
    const gb::AdamArgs step = M.adam_args(lr, 0.9f, 0.999f, 1e-8f);
    if (M.backward(M.d_xb, M.d_tb, M.d_mb, B, (float)ms, s + 1 == steps ? &loss : nullptr, &step))
      return -1;
  }
  e = cudaStreamSynchronize(M.st);
  if (e != cudaSuccess) return gb::cuda_fail(e, "MLP training");
  if (final_loss) *final_loss = loss;
  return 0;
}

}  // extern "C"

// ------------------------------------------------- allocation-free inference
//
// gb_mlp_forward_device keeps its hidden activations in buffers it
// allocates (and grows) on demand.  gb_mlp_forward_noalloc runs the same
// kernels with the activations in the fixed array below instead, for callers
// that cannot allocate device memory at that point.

namespace gb {

// Two ping-pong activation buffers of GB_MLP_NOALLOC_MAX_ACT floats each.
// Every GPU that loads the library holds this array until the process ends.
static __device__ __align__(256) float g_mlp_noalloc_scratch[2 * (size_t)GB_MLP_NOALLOC_MAX_ACT];

constexpr int kNoallocMaxDevices = 64;
static float *g_noalloc_addr[kNoallocMaxDevices];  // device address, per device
static std::mutex g_noalloc_mutex;

// Device address of the scratch array on the current device.  Host code only
// sees a host-side stand-in under the array's name, so the address is
// looked up once per device, with that device current.
static int noalloc_scratch(float **out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
  if (dev < 0 || dev >= kNoallocMaxDevices) return fail("device index beyond the scratch table");
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (!g_noalloc_addr[dev]) {
    void *p = nullptr;
    e = cudaGetSymbolAddress(&p, g_mlp_noalloc_scratch);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(scratch)");
    g_noalloc_addr[dev] = static_cast<float *>(p);
  }
  *out = g_noalloc_addr[dev];
  return 0;
}

}  // namespace gb

extern "C" int gb_mlp_forward_noalloc(gb_mlp *m, const float *d_x, int B, float *d_y,
                                      void *stream) {
  if (!m || !d_x || !d_y) return gb::fail("NULL argument");
  if (B <= 0) return gb::fail("batch size must be positive");
  gb::Mlp &M = m->m;
  {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return gb::cuda_fail(e, "cudaGetDevice");
    if (dev != M.dev) {
      char msg[160];
      snprintf(msg, sizeof msg,
               "current device %d is not the network's device %d; make device %d current", dev,
               M.dev, M.dev);
      return gb::fail(msg);
    }
  }
  int widest = 0;
  for (int l = 1; l + 1 < (int)M.width.size(); l++) widest = M.width[l] > widest ? M.width[l] : widest;
  if ((long long)B * widest > (long long)GB_MLP_NOALLOC_MAX_ACT) {
    char msg[200];
    snprintf(msg, sizeof msg,
             "batch %d x hidden width %d exceeds the static scratch of %d floats per activation "
             "buffer; split the batch",
             B, widest, (int)GB_MLP_NOALLOC_MAX_ACT);
    return gb::fail(msg);
  }
  float *base = nullptr;
  if (gb::noalloc_scratch(&base)) return -1;
  float *buf[2] = {base, base + (size_t)GB_MLP_NOALLOC_MAX_ACT};
  cudaStream_t cs = static_cast<cudaStream_t>(stream);
  // after the network's own queued work (training, parameter updates) ...
  cudaError_t e = cudaEventRecord(M.ev_own, M.st);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(cs, M.ev_own, 0);
  if (e != cudaSuccess) return gb::cuda_fail(e, "MLP forward (no allocation): ordering");
  const float *in = d_x;
  const int L = M.layers();
  for (int l = 0; l < L; l++) {
    const int K = M.width[l], N = M.width[l + 1];
    float *out = l + 1 == L ? d_y : buf[l & 1];
    gb::launch_layer(in, B, K, N, M.d_w + M.woff[l], M.d_w + M.boff[l], out, l + 1 < L ? 1 : 0,
                     cs);
    in = out;
  }
  e = cudaGetLastError();
  // ... and the network's later work after this pass
  if (e == cudaSuccess) e = cudaEventRecord(M.ev_caller, cs);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(M.st, M.ev_caller, 0);
  return e == cudaSuccess ? 0 : gb::cuda_fail(e, "MLP forward (no allocation)");
}
