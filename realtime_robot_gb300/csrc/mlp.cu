// mlp.cu — the keypoint-credibility MLP: inference, gradients and Adam.
//
// 352 -> 128 -> 64 -> 1 (ReLU, ReLU, sigmoid) over SHOT-352 descriptors.
// Parameters live on the device as FP32 master weights plus BF16 copies of
// the three weight matrices; every forward pass multiplies by the BF16
// copies and accumulates in FP32.  Training is minibatch Adam on the mean
// binary cross-entropy of the logit; gradients flow to the master weights
// with the BF16 rounding treated as the identity.
//
// Inference runs on the tensor cores (match_tc.cu); rows at an address that
// is not 16-byte aligned go through a tiled SIMT GEMM (64 x 64 tiles, K steps
// of 16, 4 x 4 outputs per thread, bias and ReLU in the epilogue).  A training
// pass is three launches: k_mlp_rows (everything that is local to a row, from
// the descriptors to dh1), k_mlp_wgrad (the two large weight gradients) and
// k_mlp_reduce.  Reductions are fixed-order, so results repeat run to run.
#include <cuda_bf16.h>
#include <string.h>

#include <vector>

#include "common.cuh"

struct rtr_mlp {
  int device = 0;
  float* theta = nullptr;          // [RTR_MLP_PARAMS] FP32 master weights
  __nv_bfloat16* wbf = nullptr;    // BF16 W1 | W2 | w3
  __nv_bfloat16* w1pad = nullptr;  // BF16 W1 as [128][384], zero past column 352 (tensor-core inference)
  float* m = nullptr;              // Adam first moment
  float* v = nullptr;              // Adam second moment
  int step = 0;                    // Adam steps taken
  uint64_t uid = 0;                // identity for captured recognitions (rtr::next_uid)
};

uint64_t rtr_mlp_uid(const rtr_mlp* m) { return m ? m->uid : 0; }

namespace rtr {

constexpr int MLP_IN = 352, MLP_H1 = 128, MLP_H2 = 64;
constexpr int OFF_W1 = 0, OFF_B1 = OFF_W1 + MLP_H1 * MLP_IN, OFF_W2 = OFF_B1 + MLP_H1,
              OFF_B2 = OFF_W2 + MLP_H2 * MLP_H1, OFF_W3 = OFF_B2 + MLP_H2, OFF_B3 = OFF_W3 + MLP_H2,
              N_PARAMS = OFF_B3 + 1;
static_assert(N_PARAMS == RTR_MLP_PARAMS, "parameter layout");
constexpr int BF_W1 = 0, BF_W2 = MLP_H1 * MLP_IN, BF_W3 = BF_W2 + MLP_H2 * MLP_H1, BF_N = BF_W3 + MLP_H2;

// ---------------------------------------------------------------------------
// tiled SIMT GEMM: C[m][n] = sum_k A(m, k) B(n, k), then the epilogue
//   A(m, k) = A[m * K + k], B(n, k) = B[n * K + k], C = ReLU(. + bias[n])
// ---------------------------------------------------------------------------
constexpr int GT = 64, GK = 16;

__global__ void __launch_bounds__(256) k_gemm(int M, int N, int K, const float* __restrict__ A,
                                              const __nv_bfloat16* __restrict__ B, float* __restrict__ Cm,
                                              const float* __restrict__ bias, const int* __restrict__ dM) {
  __shared__ float As[GK][GT + 4], Bs[GK][GT + 4];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int m0 = blockIdx.y * GT, n0 = blockIdx.x * GT;
  if (dM) M = min(*dM, M);  // rows counted on the device (grid sized for the capacity)
  if (m0 >= M) return;      // uniform per block, before any barrier
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  for (int k0 = 0; k0 < K; k0 += GK) {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int e = tid + 256 * r;  // element of the 64 x 16 tile
      const int kk = e & 15, mm = e >> 4;
      const int gm = m0 + mm, gn = n0 + mm, gk = k0 + kk;
      As[kk][mm] = (gm < M && gk < K) ? A[(long long)gm * K + gk] : 0.f;
      Bs[kk][mm] = (gn < N && gk < K) ? __bfloat162float(B[(long long)gn * K + gk]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < GK; ++kk) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[kk][ty + 16 * i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Bs[kk][tx + 16 * j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int gm = m0 + ty + 16 * i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int gn = n0 + tx + 16 * j;
      if (gn < N) Cm[(long long)gm * N + gn] = fmaxf(acc[i][j] + bias[gn], 0.f);
    }
  }
}

static void gemm(int M, int N, int K, const float* A, const __nv_bfloat16* B, float* C, const float* bias,
                 cudaStream_t st, const int* dM = nullptr) {
  const dim3 grid((N + GT - 1) / GT, (M + GT - 1) / GT);
  k_gemm<<<grid, 256, 0, st>>>(M, N, K, A, B, C, bias, dM);
  RTR_LAUNCHED(1);
}

// ---------------------------------------------------------------------------
// head: score = sigmoid(h2 . w3 + b3) per row
// ---------------------------------------------------------------------------
__global__ void k_head(const float* __restrict__ h2, int n, const __nv_bfloat16* __restrict__ w3bf,
                       const float* __restrict__ theta, float* __restrict__ score, const int* __restrict__ d_n) {
  if (d_n) n = min(*d_n, n);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float* h = h2 + (size_t)i * MLP_H2;
    float z = 0.f;
#pragma unroll 8
    for (int j = 0; j < MLP_H2; ++j) z = fmaf(h[j], __bfloat162float(w3bf[j]), z);
    z += theta[OFF_B3];
    score[i] = 1.f / (1.f + __expf(-z));
  }
}

// ---------------------------------------------------------------------------
// training pass, part 1: everything local to a row.  A block owns MR rows:
//   h1 = relu(X W1^T + b1), h2 = relu(h1 W2^T + b2), z = h2 . w3 + b3,
//   dz = (sigmoid(z) - y) / n, dh2 = dz w3 (h2 > 0), dh1 = (dh2 W2) (h1 > 0)
// with h1, h2 and dh2 in shared memory between the layers; h1, dh2 and dh1 go
// to memory for the weight gradients, and the block's column sums (db1, db2,
// dw3, db3 and the loss) to colpart.
//
// Bound by the FP32 pipe and by the latency of its chain: 0.5 GFLOP of the
// pass at 4096 rows, 128 blocks of 32 rows (64 rows would leave half the SMs
// idle).  The next K chunk of X and W1 is fetched to registers during the
// current one.  As five launches
// this part took 77 us at 4096 rows, 25 us now.
// ---------------------------------------------------------------------------
constexpr int MR = 32, MKT = 32;
constexpr int W1S = MLP_H1;       // stride of the W1 chunk [kk][j]
constexpr int XS = MKT + 4;       // stride of the X chunk [row][kk]
constexpr int H1S = MLP_H1 + 4;   // stride of h1 [row][k]
constexpr int W2S = MLP_H2 + 4;   // stride of W2 [k][j]: float4 reads of 8 consecutive k touch every bank once
constexpr int H2S = MLP_H2 + 4;   // stride of h2 and dh2 [row][j]
constexpr int COLS = MLP_H1 + MLP_H2 + MLP_H2 + 2;  // db1 | db2 | dw3 | db3 | loss
struct MlpRowsSmem {
  float w2[MLP_H1 * W2S];
  float h1[MR * H1S];
  union {
    struct {
      float w1[MKT * W1S];
      float x[MR * XS];
    } in;
    struct {
      float h2[MR * H2S], dh2[MR * H2S];
      float dh1[MR * H1S];
      float dz[MR], loss[MR];
    } out;
  } u;
};

__global__ void __launch_bounds__(256) k_mlp_rows(const float* __restrict__ X, const float* __restrict__ y, int n,
                                                  const __nv_bfloat16* __restrict__ wbf,
                                                  const float* __restrict__ theta, float* __restrict__ gh1,
                                                  float* __restrict__ gdh2, float* __restrict__ gdh1,
                                                  float* __restrict__ colpart) {
  extern __shared__ __align__(16) unsigned char mlp_smem[];
  MlpRowsSmem& S = *reinterpret_cast<MlpRowsSmem*>(mlp_smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r0 = blockIdx.x * MR;
  // W2 [64][128] -> [k][j]; a thread takes one j and 8 consecutive k at a time
  for (int e = tid; e < MLP_H2 * MLP_H1 / 8; e += 256) {
    const int j = e & (MLP_H2 - 1), k8 = (e / MLP_H2) * 8;
    const uint4 v = *reinterpret_cast<const uint4*>(wbf + BF_W2 + j * MLP_H1 + k8);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float2 f = __bfloat1622float2(h[q]);
      S.w2[(k8 + 2 * q) * W2S + j] = f.x;
      S.w2[(k8 + 2 * q + 1) * W2S + j] = f.y;
    }
  }
  // layer 1: thread (warp, lane) owns rows 4 warp .. + 3 and columns 4 lane .. + 3
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  float xr[4];
  uint4 wr[2];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {  // row 4 warp + q, column k0 + lane (MLP_IN is a multiple of MKT)
      const int r = r0 + 4 * warp + q;
      xr[q] = r < n ? X[(size_t)r * MLP_IN + k0 + lane] : 0.f;
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {  // W1 row j = tid & 127, 8 columns from 8 (tid / 128 + 2 q)
      const int j = tid & (MLP_H1 - 1), kc = 8 * ((tid >> 7) + 2 * q);
      wr[q] = *reinterpret_cast<const uint4*>(wbf + BF_W1 + j * MLP_IN + k0 + kc);
    }
  };
  static_assert(MLP_IN % MKT == 0 && MKT == 32, "K chunks");
  fetch(0);
  for (int k0 = 0; k0 < MLP_IN; k0 += MKT) {
    __syncthreads();  // the previous chunk has been read
#pragma unroll
    for (int q = 0; q < 4; ++q) S.u.in.x[(4 * warp + q) * XS + lane] = xr[q];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int j = tid & (MLP_H1 - 1), kc = 8 * ((tid >> 7) + 2 * q);
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&wr[q]);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 f = __bfloat1622float2(h[e]);
        S.u.in.w1[(kc + 2 * e) * W1S + j] = f.x;
        S.u.in.w1[(kc + 2 * e + 1) * W1S + j] = f.y;
      }
    }
    __syncthreads();
    if (k0 + MKT < MLP_IN) fetch(k0 + MKT);
#pragma unroll
    for (int kk = 0; kk < MKT; kk += 4) {
      float4 a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(&S.u.in.x[(4 * warp + i) * XS + kk]);
#pragma unroll
      for (int q = 0; q < 4; ++q) b[q] = *reinterpret_cast<const float4*>(&S.u.in.w1[(kk + q) * W1S + 4 * lane]);
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float av = q == 0 ? a[i].x : (q == 1 ? a[i].y : (q == 2 ? a[i].z : a[i].w));
          acc[i][0] = fmaf(av, b[q].x, acc[i][0]);
          acc[i][1] = fmaf(av, b[q].y, acc[i][1]);
          acc[i][2] = fmaf(av, b[q].z, acc[i][2]);
          acc[i][3] = fmaf(av, b[q].w, acc[i][3]);
        }
    }
  }
  {
    const float4 b1 = make_float4(theta[OFF_B1 + 4 * lane], theta[OFF_B1 + 4 * lane + 1], theta[OFF_B1 + 4 * lane + 2],
                                  theta[OFF_B1 + 4 * lane + 3]);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = 4 * warp + i;
      const float4 h = make_float4(fmaxf(acc[i][0] + b1.x, 0.f), fmaxf(acc[i][1] + b1.y, 0.f),
                                   fmaxf(acc[i][2] + b1.z, 0.f), fmaxf(acc[i][3] + b1.w, 0.f));
      *reinterpret_cast<float4*>(&S.h1[r * H1S + 4 * lane]) = h;
      if (r0 + r < n) *reinterpret_cast<float4*>(gh1 + (size_t)(r0 + r) * MLP_H1 + 4 * lane) = h;
    }
  }
  __syncthreads();  // h1 complete; the chunk buffers are free
  // layer 2 and the head: thread owns rows 2 (tid / 16), + 1 and columns 4 (tid % 16) .. + 3
  {
    const int tx = tid & 15, ty = tid >> 4;
    float c[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll 4
    for (int k = 0; k < MLP_H1; k += 4) {
      float4 a[2], b[4];
#pragma unroll
      for (int i = 0; i < 2; ++i) a[i] = *reinterpret_cast<const float4*>(&S.h1[(2 * ty + i) * H1S + k]);
#pragma unroll
      for (int q = 0; q < 4; ++q) b[q] = *reinterpret_cast<const float4*>(&S.w2[(k + q) * W2S + 4 * tx]);
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float av = q == 0 ? a[i].x : (q == 1 ? a[i].y : (q == 2 ? a[i].z : a[i].w));
          c[i][0] = fmaf(av, b[q].x, c[i][0]);
          c[i][1] = fmaf(av, b[q].y, c[i][1]);
          c[i][2] = fmaf(av, b[q].z, c[i][2]);
          c[i][3] = fmaf(av, b[q].w, c[i][3]);
        }
    }
    float w3[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) w3[q] = __bfloat162float(wbf[BF_W3 + 4 * tx + q]);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = 2 * ty + i;
      float z = 0.f;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        c[i][q] = fmaxf(c[i][q] + theta[OFF_B2 + 4 * tx + q], 0.f);
        z = fmaf(c[i][q], w3[q], z);
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);  // the row's 16 lanes
      z += theta[OFF_B3];
      float d = 0.f, l = 0.f;
      if (r0 + r < n) {
        const float yi = y[r0 + r];
        l = fmaxf(z, 0.f) - yi * z + log1pf(__expf(-fabsf(z)));
        d = (1.f / (1.f + __expf(-z)) - yi) / (float)n;
      }
      if (tx == 0) {
        S.u.out.dz[r] = d;
        S.u.out.loss[r] = l;
      }
      float4 g;
      g.x = c[i][0] > 0.f ? d * w3[0] : 0.f;
      g.y = c[i][1] > 0.f ? d * w3[1] : 0.f;
      g.z = c[i][2] > 0.f ? d * w3[2] : 0.f;
      g.w = c[i][3] > 0.f ? d * w3[3] : 0.f;
      *reinterpret_cast<float4*>(&S.u.out.h2[r * H2S + 4 * tx]) = make_float4(c[i][0], c[i][1], c[i][2], c[i][3]);
      *reinterpret_cast<float4*>(&S.u.out.dh2[r * H2S + 4 * tx]) = g;
      if (r0 + r < n) *reinterpret_cast<float4*>(gdh2 + (size_t)(r0 + r) * MLP_H2 + 4 * tx) = g;
    }
  }
  __syncthreads();
  // dh1: thread owns rows 4 warp .. + 3 and columns lane + 32 c
  {
    float d[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int q = 0; q < 4; ++q) d[i][q] = 0.f;
#pragma unroll 4
    for (int j = 0; j < MLP_H2; j += 4) {
      float4 a[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(&S.u.out.dh2[(4 * warp + i) * H2S + j]);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float4 b = *reinterpret_cast<const float4*>(&S.w2[(lane + 32 * q) * W2S + j]);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          d[i][q] = fmaf(a[i].x, b.x, d[i][q]);
          d[i][q] = fmaf(a[i].y, b.y, d[i][q]);
          d[i][q] = fmaf(a[i].z, b.z, d[i][q]);
          d[i][q] = fmaf(a[i].w, b.w, d[i][q]);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int r = 4 * warp + i, k = lane + 32 * q;
        const float v = S.h1[r * H1S + k] > 0.f ? d[i][q] : 0.f;
        S.u.out.dh1[r * H1S + k] = v;
        if (r0 + r < n) gdh1[(size_t)(r0 + r) * MLP_H1 + k] = v;
      }
  }
  __syncthreads();
  // column sums over the block's rows, in row order (rows past n hold zeros in dh1, dh2, dz and loss)
  float* cp = colpart + (size_t)blockIdx.x * COLS;
  for (int c = tid; c < COLS; c += 256) {
    float a = 0.f;
    if (c < MLP_H1) {
      for (int r = 0; r < MR; ++r) a += S.u.out.dh1[r * H1S + c];
    } else if (c < MLP_H1 + MLP_H2) {
      for (int r = 0; r < MR; ++r) a += S.u.out.dh2[r * H2S + c - MLP_H1];
    } else if (c < MLP_H1 + 2 * MLP_H2) {
      for (int r = 0; r < MR; ++r) a = fmaf(S.u.out.dz[r], S.u.out.h2[r * H2S + c - MLP_H1 - MLP_H2], a);
    } else {
      const float* v = c == COLS - 2 ? S.u.out.dz : S.u.out.loss;
      for (int r = 0; r < MR; ++r) a += v[r];
    }
    cp[c] = a;
  }
}

// ---------------------------------------------------------------------------
// training pass, part 2: dW1[j][k] = sum_i dh1[i][j] X[i][k] and
// dW2[j][k] = sum_i dh2[i][j] h1[i][k].  The outputs are 52 tiles of 32 x 32;
// the rows, the long axis, are cut into slabs (blockIdx.y) and, inside a
// block, between its 8 warps, each with its own staged rows and a 4 x 8
// share of the tile per lane: no block barrier until the warps' tiles are
// added up, in warp order.  Slabs write to part, or, when there is one,
// straight to the gradient.
//
// The rows used to be one serial loop of 2, 1 and 12 blocks (three launches,
// 715 of a 4096-row pass's 810 us, 1 % of the SMs busy); 24.5 us now, and
// 2.6 us of part 3.
// Slabs of 1024 rows or more keep the pass's scratch below what a separate
// buffer for each activation took.
// ---------------------------------------------------------------------------
constexpr int WG_TILES1 = (MLP_H1 / 32) * (MLP_IN / 32), WG_TILES2 = (MLP_H2 / 32) * (MLP_H1 / 32);
constexpr int WG_RC = 16;     // rows a warp stages at a time
constexpr int WG_SLAB = 1024;
constexpr int WG_PART = MLP_H1 * MLP_IN + MLP_H2 * MLP_H1;  // floats of one slab's part: dW1 | dW2
static int wg_slabs(int n) { return n / WG_SLAB > 1 ? n / WG_SLAB : 1; }

__global__ void __launch_bounds__(256) k_mlp_wgrad(const float* __restrict__ X, const float* __restrict__ h1,
                                                   const float* __restrict__ dh1, const float* __restrict__ dh2,
                                                   int n, float* __restrict__ dW1, float* __restrict__ dW2,
                                                   size_t slab_stride) {
  __shared__ __align__(16) float s_a[8][WG_RC][32], s_b[8][WG_RC][32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tile = blockIdx.x;
  const bool first = tile < WG_TILES1;
  const int t = first ? tile : tile - WG_TILES1;
  const int tk = first ? MLP_IN / 32 : MLP_H1 / 32;
  const int j0 = (t / tk) * 32, k0 = (t % tk) * 32;
  const float* A = first ? dh1 : dh2;
  const float* B = first ? X : h1;
  const int lda = first ? MLP_H1 : MLP_H2, ldb = first ? MLP_IN : MLP_H1;
  // this slab's rows, then this warp's: equal shares in steps of WG_RC
  const int slabs = gridDim.y;
  const int srows = ((n + slabs - 1) / slabs + WG_RC - 1) / WG_RC * WG_RC;
  const int sbeg = min(n, (int)blockIdx.y * srows), send = min(n, sbeg + srows);
  const int wrows = ((send - sbeg + 7) / 8 + WG_RC - 1) / WG_RC * WG_RC;
  const int beg = min(send, sbeg + warp * wrows), end = min(send, beg + wrows);
  const int ty = lane >> 2, tx = lane & 3;  // 4 rows of the tile from 4 ty, 8 columns from 8 tx
  float acc[4][8];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
  float ra[WG_RC], rb[WG_RC];
  auto fetch = [&](int i0) {
#pragma unroll
    for (int r = 0; r < WG_RC; ++r) {
      const bool in = i0 + r < end;
      ra[r] = in ? A[(size_t)(i0 + r) * lda + j0 + lane] : 0.f;
      rb[r] = in ? B[(size_t)(i0 + r) * ldb + k0 + lane] : 0.f;
    }
  };
  if (beg < end) fetch(beg);
  for (int i0 = beg; i0 < end; i0 += WG_RC) {
    __syncwarp();
#pragma unroll
    for (int r = 0; r < WG_RC; ++r) {
      s_a[warp][r][lane] = ra[r];
      s_b[warp][r][lane] = rb[r];
    }
    __syncwarp();
    if (i0 + WG_RC < end) fetch(i0 + WG_RC);
#pragma unroll
    for (int r = 0; r < WG_RC; ++r) {
      const float4 a = *reinterpret_cast<const float4*>(&s_a[warp][r][4 * ty]);
      const float4 b0 = *reinterpret_cast<const float4*>(&s_b[warp][r][8 * tx]);
      const float4 b1 = *reinterpret_cast<const float4*>(&s_b[warp][r][8 * tx + 4]);
      const float av[4] = {a.x, a.y, a.z, a.w};
      const float bv[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    }
  }
  // the warps' tiles, added in warp order: warp w's 32 x 32 values in its own
  // staging (1024 floats = s_a[w] and s_b[w])
  __syncwarp();
  float* mine_a = &s_a[warp][0][0];
  float* mine_b = &s_b[warp][0][0];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int e = (4 * ty + i) * 32 + 8 * tx + j;
      (e < 512 ? mine_a : mine_b)[e & 511] = acc[i][j];
    }
  __syncthreads();
  float* out = (first ? dW1 : dW2) + (size_t)blockIdx.y * slab_stride;
  for (int e = tid; e < 1024; e += 256) {
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) v += (e < 512 ? &s_a[w][0][0] : &s_b[w][0][0])[e & 511];
    out[(size_t)(j0 + (e >> 5)) * ldb + k0 + (e & 31)] = v;
  }
}

// Part 3: the slabs' weight gradients summed in slab order, and the blocks'
// column sums (a warp per column, lanes striding over the blocks, then a
// butterfly).  Blocks past the weights take the columns.
__global__ void __launch_bounds__(256) k_mlp_reduce(const float* __restrict__ part, int slabs,
                                                    const float* __restrict__ colpart, int nblk, int n,
                                                    float* __restrict__ g, float* __restrict__ d_loss, int wblocks) {
  if ((int)blockIdx.x < wblocks) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= WG_PART) return;
    float a = 0.f;
#pragma unroll 4
    for (int s = 0; s < slabs; ++s) a += part[(size_t)s * WG_PART + i];
    g[i < MLP_H1 * MLP_IN ? OFF_W1 + i : OFF_W2 + (i - MLP_H1 * MLP_IN)] = a;
    return;
  }
  const int lane = threadIdx.x & 31, c = (blockIdx.x - wblocks) * 8 + (threadIdx.x >> 5);
  if (c >= COLS) return;
  float a = 0.f;
  for (int b = lane; b < nblk; b += 32) a += colpart[(size_t)b * COLS + c];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
  if (lane != 0) return;
  if (c == COLS - 1) {
    *d_loss = a / (float)n;
    return;
  }
  const int dst = c < MLP_H1 ? OFF_B1 + c
                             : (c < MLP_H1 + MLP_H2 ? OFF_B2 + c - MLP_H1
                                                    : (c < COLS - 2 ? OFF_W3 + c - MLP_H1 - MLP_H2 : OFF_B3));
  g[dst] = a;
}

constexpr int W1PAD_K = 384;
__global__ void k_to_bf16(const float* __restrict__ theta, __nv_bfloat16* __restrict__ wbf,
                          __nv_bfloat16* __restrict__ w1pad) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < BF_N; i += gridDim.x * blockDim.x) {
    const int src = i < BF_W2 ? OFF_W1 + i : (i < BF_W3 ? OFF_W2 + (i - BF_W2) : OFF_W3 + (i - BF_W3));
    wbf[i] = __float2bfloat16_rn(theta[src]);
  }
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < MLP_H1 * W1PAD_K; i += gridDim.x * blockDim.x) {
    const int r = i / W1PAD_K, k = i - r * W1PAD_K;
    w1pad[i] = __float2bfloat16_rn(k < MLP_IN ? theta[OFF_W1 + r * MLP_IN + k] : 0.f);
  }
}

__global__ void k_adam(float* __restrict__ theta, const float* __restrict__ g, float* __restrict__ m,
                       float* __restrict__ v, int n, float lr, float b1, float b2, float eps, float c1, float c2) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    theta[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  }
}

__global__ void k_accum(float* __restrict__ acc, const float* __restrict__ x, float w) { *acc += w * *x; }

__global__ void k_gather_rows(const float* __restrict__ X, const float* __restrict__ y, const int* __restrict__ idx,
                              int n, float* __restrict__ Xo, float* __restrict__ yo) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < (long long)n * MLP_IN;
       e += (long long)gridDim.x * blockDim.x) {
    const int r = (int)(e / MLP_IN), c = (int)(e - (long long)r * MLP_IN);
    Xo[e] = X[(size_t)idx[r] * MLP_IN + c];
    if (c == 0) yo[r] = y[idx[r]];
  }
}

// Scratch of one forward/backward over n rows.
struct MlpWork {
  float *h1, *dh2, *dh1, *colpart, *part, *grad;
};

static int mlp_row_blocks(int n) { return (n + MR - 1) / MR; }

static void mlp_plan(ScratchPlan& p, int n) {
  p.add<float>((size_t)n * MLP_H1);
  p.add<float>((size_t)n * MLP_H2);
  p.add<float>((size_t)n * MLP_H1);
  p.add<float>((size_t)mlp_row_blocks(n) * COLS);
  p.add<float>(wg_slabs(n) > 1 ? (size_t)wg_slabs(n) * WG_PART : 0);
  p.add<float>(N_PARAMS);
}

static bool mlp_take(Scratch& s, int n, MlpWork* w) {
  w->h1 = s.take<float>((size_t)n * MLP_H1);
  w->dh2 = s.take<float>((size_t)n * MLP_H2);
  w->dh1 = s.take<float>((size_t)n * MLP_H1);
  w->colpart = s.take<float>((size_t)mlp_row_blocks(n) * COLS);
  w->part = s.take<float>(wg_slabs(n) > 1 ? (size_t)wg_slabs(n) * WG_PART : 0);
  w->grad = s.take<float>(N_PARAMS);
  return w->grad != nullptr;
}

// Mean loss over n labelled rows of X (into *d_loss) and its gradient (into
// g, RTR_MLP_PARAMS floats).
static rtr_status mlp_pass(const rtr_mlp* m, const float* X, const float* y, int n, const MlpWork& w, float* g,
                           float* d_loss, cudaStream_t st) {
  RTR_CUDA(cudaFuncSetAttribute(k_mlp_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(MlpRowsSmem)));
  const int rb = mlp_row_blocks(n), slabs = wg_slabs(n);
  k_mlp_rows<<<rb, 256, sizeof(MlpRowsSmem), st>>>(X, y, n, m->wbf, m->theta, w.h1, w.dh2, w.dh1, w.colpart);
  float* dW1 = slabs > 1 ? w.part : g + OFF_W1;
  float* dW2 = slabs > 1 ? w.part + MLP_H1 * MLP_IN : g + OFF_W2;
  k_mlp_wgrad<<<dim3(WG_TILES1 + WG_TILES2, slabs), 256, 0, st>>>(X, w.h1, w.dh1, w.dh2, n, dW1, dW2, WG_PART);
  const int wblocks = slabs > 1 ? (WG_PART + 255) / 256 : 0;
  k_mlp_reduce<<<wblocks + (COLS + 7) / 8, 256, 0, st>>>(w.part, slabs, w.colpart, rb, n, g, d_loss, wblocks);
  RTR_LAUNCHED(3);
  RTR_CUDA(cudaGetLastError());
  return RTR_OK;
}

static void mlp_refresh_bf16(rtr_mlp* m, cudaStream_t st) {
  k_to_bf16<<<(BF_N + 255) / 256, 256, 0, st>>>(m->theta, m->wbf, m->w1pad);
  RTR_LAUNCHED(1);
}

static void mlp_adam(rtr_mlp* m, const float* grad, float lr, cudaStream_t st) {
  m->step += 1;
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.f - powf(b1, (float)m->step), c2 = 1.f - powf(b2, (float)m->step);
  k_adam<<<(N_PARAMS + 255) / 256, 256, 0, st>>>(m->theta, grad, m->m, m->v, N_PARAMS, lr, b1, b2, 1e-8f, c1, c2);
  RTR_LAUNCHED(1);
  mlp_refresh_bf16(m, st);
}

// He-uniform initialisation on the host (SplitMix64 stream, bound
// sqrt(6 / fan_in)), zero biases.
static void mlp_host_init(uint64_t seed, float* out) {
  uint64_t s = seed;
  auto next = [&s]() {
    uint64_t z = (s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
  };
  auto uni = [&next](float bound) { return (float)((double)(next() >> 11) * 0x1.0p-53 * 2.0 - 1.0) * bound; };
  memset(out, 0, sizeof(float) * N_PARAMS);
  const float bw1 = sqrtf(6.f / MLP_IN), bw2 = sqrtf(6.f / MLP_H1), bw3 = sqrtf(6.f / MLP_H2);
  for (int i = 0; i < MLP_H1 * MLP_IN; ++i) out[OFF_W1 + i] = uni(bw1);
  for (int i = 0; i < MLP_H2 * MLP_H1; ++i) out[OFF_W2 + i] = uni(bw2);
  for (int i = 0; i < MLP_H2; ++i) out[OFF_W3 + i] = uni(bw3);
}

size_t mlp_tc_bytes(int n_cap);
rtr_status mlp_tc_score(rtr_context* ctx, Scratch& s, const float* X, int n_cap, const int* d_n,
                        const __nv_bfloat16* w1pad, const float* b1, const __nv_bfloat16* w2, const float* b2,
                        const __nv_bfloat16* w3, const float* b3, float* score, cudaStream_t st);

// Inference on the tensor cores (match_tc.cu: layer 1 as a tcgen05 GEMM of
// three BF16 parts of X, layers 2 and 3 in its epilogue) when X is 16-byte
// aligned; the SIMT passes otherwise.
static bool mlp_tc_ok(const float* X) { return (reinterpret_cast<uintptr_t>(X) & 15u) == 0; }
static rtr_status mlp_tc(rtr_context* ctx, Scratch& s, const rtr_mlp* m, const float* X, int n_cap, const int* d_n,
                         float* score, cudaStream_t st) {
  const float* th = m->theta;
  return mlp_tc_score(ctx, s, X, n_cap, d_n, m->w1pad, th + OFF_B1, m->wbf + BF_W2, th + OFF_B2, m->wbf + BF_W3,
                      th + OFF_B3, score, st);
}

static rtr_status mlp_simt(Scratch& s, const rtr_mlp* m, const float* X, int n_cap, const int* d_n, float* score,
                           cudaStream_t st) {
  float* h1 = s.take<float>((size_t)n_cap * MLP_H1);
  float* h2 = s.take<float>((size_t)n_cap * MLP_H2);
  if (!h2) return fail(RTR_ERR_CAPACITY, "mlp: scratch");
  const float* th = m->theta;
  gemm(n_cap, MLP_H1, MLP_IN, X, m->wbf + BF_W1, h1, th + OFF_B1, st, d_n);
  gemm(n_cap, MLP_H2, MLP_H1, h1, m->wbf + BF_W2, h2, th + OFF_B2, st, d_n);
  int hb = (n_cap + 255) / 256;
  if (hb > 152 * 8) hb = 152 * 8;
  k_head<<<hb, 256, 0, st>>>(h2, n_cap, m->wbf + BF_W3, th, score, d_n);
  RTR_LAUNCHED(1);
  RTR_CUDA(cudaGetLastError());
  return RTR_OK;
}

rtr_status mlp_score_dev(rtr_context* ctx, Scratch& s, const rtr_mlp* m, const float* X, int n, float* score,
                         cudaStream_t st) {
  if (n <= 0) return RTR_OK;
  if (mlp_tc_ok(X)) return mlp_tc(ctx, s, m, X, n, nullptr, score, st);
  return mlp_simt(s, m, X, n, nullptr, score, st);
}

// Scores of the first *d_n (<= n_cap) rows of X, for callers whose row count
// lives on the device; needs mlp_infer_bytes(n_cap) of scratch.
size_t mlp_infer_bytes(int n_cap) {
  ScratchPlan p;
  p.add<float>((size_t)(n_cap > 0 ? n_cap : 1) * MLP_H1);
  p.add<float>((size_t)(n_cap > 0 ? n_cap : 1) * MLP_H2);
  const size_t tc = mlp_tc_bytes(n_cap);
  return p.bytes > tc ? p.bytes : tc;
}

rtr_status mlp_score_rows(rtr_context* ctx, Scratch& s, const rtr_mlp* m, const float* X, int n_cap, const int* d_n,
                          float* score, cudaStream_t st) {
  if (n_cap <= 0) return RTR_OK;
  if (mlp_tc_ok(X)) return mlp_tc(ctx, s, m, X, n_cap, d_n, score, st);
  return mlp_simt(s, m, X, n_cap, d_n, score, st);
}

size_t mlp_scratch_bytes(int n) {
  ScratchPlan p;
  mlp_plan(p, n > 0 ? n : 1);
  return p.bytes;
}

}  // namespace rtr

using namespace rtr;

extern "C" {

rtr_status rtr_mlp_create(rtr_context* ctx, const float* h_params, uint64_t seed, rtr_mlp** out) {
  RTR_CHECK_ARG(ctx && out, "rtr_mlp_create: bad arguments");
  *out = nullptr;
  RTR_CUDA(cudaSetDevice(ctx->device));
  std::vector<float> init;
  if (!h_params) {
    init.resize(N_PARAMS);
    mlp_host_init(seed, init.data());
    h_params = init.data();
  }
  rtr_mlp* m = new rtr_mlp();
  m->device = ctx->device;
  m->uid = next_uid();
  if (cudaMalloc(&m->theta, sizeof(float) * N_PARAMS) != cudaSuccess ||
      cudaMalloc(&m->wbf, sizeof(__nv_bfloat16) * BF_N) != cudaSuccess ||
      cudaMalloc(&m->w1pad, sizeof(__nv_bfloat16) * MLP_H1 * W1PAD_K) != cudaSuccess ||
      cudaMalloc(&m->m, sizeof(float) * N_PARAMS) != cudaSuccess ||
      cudaMalloc(&m->v, sizeof(float) * N_PARAMS) != cudaSuccess) {
    cudaFree(m->theta);
    cudaFree(m->wbf);
    cudaFree(m->w1pad);
    cudaFree(m->m);
    cudaFree(m->v);
    delete m;
    (void)cudaGetLastError();
    return fail(RTR_ERR_OOM, "rtr_mlp_create: device allocation failed");
  }
  RTR_CUDA(cudaMemcpy(m->theta, h_params, sizeof(float) * N_PARAMS, cudaMemcpyHostToDevice));
  RTR_CUDA(cudaMemset(m->m, 0, sizeof(float) * N_PARAMS));
  RTR_CUDA(cudaMemset(m->v, 0, sizeof(float) * N_PARAMS));
  mlp_refresh_bf16(m, 0);
  RTR_CUDA(cudaDeviceSynchronize());
  *out = m;
  return RTR_OK;
}

rtr_status rtr_mlp_destroy(rtr_mlp* m) {
  if (!m) return RTR_OK;
  cudaSetDevice(m->device);
  cudaFree(m->theta);
  cudaFree(m->wbf);
  cudaFree(m->w1pad);
  cudaFree(m->m);
  cudaFree(m->v);
  delete m;
  return RTR_OK;
}

rtr_status rtr_mlp_get_params(const rtr_mlp* m, float* h_params) {
  RTR_CHECK_ARG(m && h_params, "rtr_mlp_get_params: bad arguments");
  RTR_CUDA(cudaSetDevice(m->device));
  RTR_CUDA(cudaDeviceSynchronize());
  RTR_CUDA(cudaMemcpy(h_params, m->theta, sizeof(float) * N_PARAMS, cudaMemcpyDeviceToHost));
  return RTR_OK;
}

rtr_status rtr_mlp_set_params(rtr_mlp* m, const float* h_params) {
  RTR_CHECK_ARG(m && h_params, "rtr_mlp_set_params: bad arguments");
  RTR_CUDA(cudaSetDevice(m->device));
  RTR_CUDA(cudaDeviceSynchronize());
  RTR_CUDA(cudaMemcpy(m->theta, h_params, sizeof(float) * N_PARAMS, cudaMemcpyHostToDevice));
  RTR_CUDA(cudaMemset(m->m, 0, sizeof(float) * N_PARAMS));
  RTR_CUDA(cudaMemset(m->v, 0, sizeof(float) * N_PARAMS));
  m->step = 0;
  mlp_refresh_bf16(m, 0);
  RTR_CUDA(cudaDeviceSynchronize());
  return RTR_OK;
}

rtr_status rtr_mlp_score(rtr_context* ctx, const rtr_mlp* m, const float* d_x, int n, float* d_score,
                         rtr_stream_t stream) {
  RTR_CHECK_ARG(ctx && m && n >= 0, "rtr_mlp_score: bad arguments");
  if (n == 0) return RTR_OK;
  RTR_CHECK_ARG(d_x && d_score, "rtr_mlp_score: NULL input or output");
  cudaStream_t st = (cudaStream_t)stream;
  RTR_CUDA(cudaSetDevice(ctx->device));
  Scratch s;
  const size_t need = mlp_scratch_bytes(n) > mlp_tc_bytes(n) ? mlp_scratch_bytes(n) : mlp_tc_bytes(n);
  RTR_TRY(ensure_scratch(ctx, need, st, &s));
  ProfScope ps(ctx, st, "mlp_score");
  return mlp_score_dev(ctx, s, m, d_x, n, d_score, st);
}

rtr_status rtr_mlp_loss_grad(rtr_context* ctx, const rtr_mlp* m, const float* d_x, const float* d_y, int n,
                             float* d_grad, float* d_loss, rtr_stream_t stream) {
  RTR_CHECK_ARG(ctx && m && n > 0 && d_x && d_y && d_grad && d_loss, "rtr_mlp_loss_grad: bad arguments");
  cudaStream_t st = (cudaStream_t)stream;
  RTR_CUDA(cudaSetDevice(ctx->device));
  Scratch s;
  RTR_TRY(ensure_scratch(ctx, mlp_scratch_bytes(n), st, &s));
  MlpWork w;
  if (!mlp_take(s, n, &w)) return fail(RTR_ERR_CAPACITY, "mlp: scratch");
  return mlp_pass(m, d_x, d_y, n, w, d_grad, d_loss, st);
}

rtr_status rtr_mlp_train_step(rtr_context* ctx, rtr_mlp* m, const float* d_x, const float* d_y, int n, float lr,
                              float* d_loss, rtr_stream_t stream) {
  RTR_CHECK_ARG(ctx && m && n > 0 && d_x && d_y && d_loss && lr > 0.f, "rtr_mlp_train_step: bad arguments");
  cudaStream_t st = (cudaStream_t)stream;
  RTR_CUDA(cudaSetDevice(ctx->device));
  Scratch s;
  RTR_TRY(ensure_scratch(ctx, mlp_scratch_bytes(n), st, &s));
  MlpWork w;
  if (!mlp_take(s, n, &w)) return fail(RTR_ERR_CAPACITY, "mlp: scratch");
  RTR_TRY(mlp_pass(m, d_x, d_y, n, w, w.grad, d_loss, st));
  mlp_adam(m, w.grad, lr, st);
  RTR_CUDA(cudaGetLastError());
  return RTR_OK;
}

rtr_status rtr_mlp_train(rtr_context* ctx, rtr_mlp* m, const float* d_x, const float* d_y, int n, int batch,
                         int epochs, float lr, uint64_t seed, float* h_epoch_loss) {
  RTR_CHECK_ARG(ctx && m && d_x && d_y && n > 0 && batch > 0 && epochs > 0 && lr > 0.f,
                "rtr_mlp_train: bad arguments");
  RTR_CUDA(cudaSetDevice(ctx->device));
  cudaStream_t st = ctx->host_stream;
  const int b = batch < n ? batch : n;
  ScratchPlan plan;
  mlp_plan(plan, b);
  plan.add<float>((size_t)b * MLP_IN);
  plan.add<float>(b);
  plan.add<int>(n);
  plan.add<float>(epochs * 2 + 2);
  Scratch s;
  RTR_TRY(ensure_scratch(ctx, plan.bytes, st, &s));
  MlpWork w;
  if (!mlp_take(s, b, &w)) return fail(RTR_ERR_CAPACITY, "mlp: scratch");
  float* xb = s.take<float>((size_t)b * MLP_IN);
  float* yb = s.take<float>(b);
  int* perm = s.take<int>(n);
  float* losses = s.take<float>(epochs * 2 + 2);
  if (!losses) return fail(RTR_ERR_CAPACITY, "mlp: scratch");
  // the epoch order: a seeded Fisher-Yates shuffle on the host, one copy per epoch
  std::vector<int> order((size_t)n);
  for (int i = 0; i < n; ++i) order[i] = i;
  uint64_t rs = seed;
  auto next = [&rs]() {
    uint64_t z = (rs += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
  };
  const int nb = (n + b - 1) / b;
  for (int e = 0; e < epochs; ++e) {
    for (int i = n - 1; i > 0; --i) {
      const int j = (int)(next() % (uint64_t)(i + 1));
      const int t = order[i];
      order[i] = order[j];
      order[j] = t;
    }
    RTR_CUDA(cudaMemcpyAsync(perm, order.data(), sizeof(int) * (size_t)n, cudaMemcpyHostToDevice, st));
    RTR_CUDA(cudaMemsetAsync(losses + 2 * e, 0, sizeof(float), st));
    for (int k = 0; k < nb; ++k) {
      const int r0 = k * b, rn = (r0 + b <= n) ? b : n - r0;
      k_gather_rows<<<152 * 4, 256, 0, st>>>(d_x, d_y, perm + r0, rn, xb, yb);
      RTR_LAUNCHED(1);
      RTR_TRY(mlp_pass(m, xb, yb, rn, w, w.grad, losses + 2 * e + 1, st));
      mlp_adam(m, w.grad, lr, st);
      k_accum<<<1, 1, 0, st>>>(losses + 2 * e, losses + 2 * e + 1, (float)rn / (float)n);
      RTR_LAUNCHED(1);
    }
    RTR_CUDA(cudaGetLastError());
  }
  std::vector<float> h((size_t)epochs * 2);
  RTR_CUDA(cudaMemcpyAsync(h.data(), losses, sizeof(float) * h.size(), cudaMemcpyDeviceToHost, st));
  RTR_CUDA(cudaStreamSynchronize(st));
  if (h_epoch_loss)
    for (int e = 0; e < epochs; ++e) h_epoch_loss[e] = h[(size_t)2 * e];
  return RTR_OK;
}

}  // extern "C"
