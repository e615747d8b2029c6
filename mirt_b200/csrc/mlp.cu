// mlp.cu -- the density-compensation regressor: a multilayer perceptron
// 18 -> 64 -> 64 -> 64 -> 1 (ReLU), BF16 weights, FP32 activations and
// accumulation, trained on the device by hand-written forward / backward
// kernels with Adam on FP32 master weights; inference on the tensor cores
// (mlp_infer_mma_kernel).
//
// Parameters, one flat FP32 vector (row-major, out x in):
//   W1[64][18] b1[64] W2[64][64] b2[64] W3[64][64] b3[64] W4[64] b4
// The forward and backward passes use the BF16 rounding (nearest even) of the
// master weights, refreshed after every Adam update.
//
// Gradient: mlp_grad_kernel, persistent over the batch in register tiles on the FP32
// pipes; a reduction kernel sums the partial gradients in a fixed order
// (deterministic) and applies Adam.  FP32 inference (mlp_infer_kernel): a CTA of 256
// threads takes 64 samples with the weights (as FP32) and the activations in shared
// memory (rows padded to 65 floats); thread t owns neuron t mod 64 of samples
// t / 64 + 4k, k < 16, in every layer.
#include "../../include/mirt_b200.h"

#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <string>
#include <new>
#include <vector>

#include "runtime.cuh"

using namespace mirt;

namespace {

#define MCK(call)                                                                     \
  do {                                                                                \
    cudaError_t e_ = (call);                                                          \
    if (e_ != cudaSuccess)                                                            \
      return api_fail(e_ == cudaErrorMemoryAllocation ? MIRT_ERR_ALLOC : MIRT_ERR_CUDA, \
                      std::string(#call) + ": " + cudaGetErrorString(e_));            \
  } while (0)

constexpr int NIN = MIRT_DCF_NFEAT;
constexpr int HID = 64;
constexpr int NS = 64;       // samples per CTA
constexpr int NT = 256;      // threads per CTA
constexpr int KS = NS / 4;   // samples per thread
constexpr int LD = HID + 1;  // padded row
constexpr int LDI = NIN + 1;
constexpr int P_W1 = 0, P_B1 = P_W1 + HID * NIN, P_W2 = P_B1 + HID, P_B2 = P_W2 + HID * HID,
              P_W3 = P_B2 + HID, P_B3 = P_W3 + HID * HID, P_W4 = P_B3 + HID, P_B4 = P_W4 + HID,
              NPARAM = P_B4 + 1;
static_assert(NPARAM == MIRT_MLP_NPARAM, "parameter count");

struct Weights {  // shared-memory FP32 copy of the BF16 weights
  float W1[HID][LDI];
  float b1[HID];
  float W2[HID][LD];
  float b2[HID];
  float W3[HID][LD];
  float b3[HID];
  float W4[HID];
  float b4;
};

struct Acts {
  float X[NS][LDI];
  float H1[NS][LD], H2[NS][LD], H3[NS][LD];
  float out[NS], dout[NS];
};

__device__ void load_weights(Weights &w, const __nv_bfloat16 *__restrict__ p) {
  for (int e = threadIdx.x; e < HID * NIN; e += NT) w.W1[e / NIN][e % NIN] = __bfloat162float(p[P_W1 + e]);
  for (int e = threadIdx.x; e < HID * HID; e += NT) {
    w.W2[e / HID][e % HID] = __bfloat162float(p[P_W2 + e]);
    w.W3[e / HID][e % HID] = __bfloat162float(p[P_W3 + e]);
  }
  for (int e = threadIdx.x; e < HID; e += NT) {
    w.b1[e] = __bfloat162float(p[P_B1 + e]);
    w.b2[e] = __bfloat162float(p[P_B2 + e]);
    w.b3[e] = __bfloat162float(p[P_B3 + e]);
    w.W4[e] = __bfloat162float(p[P_W4 + e]);
  }
  if (threadIdx.x == 0) w.b4 = __bfloat162float(p[P_B4]);
}

// H[s][i] = relu(b[i] + sum_j W[i][j] Hin[s][j]) for the thread's 16 samples
template <int NJ, int LDW, int LDH>
__device__ __forceinline__ void dense_relu(const float (*W)[LDW], const float *b,
                                           const float (*Hin)[LDH], float (*H)[LD]) {
  const int i = threadIdx.x & (HID - 1), s0 = threadIdx.x >> 6;
  float acc[KS];
#pragma unroll
  for (int k = 0; k < KS; k++) acc[k] = b[i];
  for (int j = 0; j < NJ; j++) {
    const float wij = W[i][j];
#pragma unroll
    for (int k = 0; k < KS; k++) acc[k] = fmaf(wij, Hin[s0 + 4 * k][j], acc[k]);
  }
#pragma unroll
  for (int k = 0; k < KS; k++) H[s0 + 4 * k][i] = fmaxf(acc[k], 0.f);
}

// forward through the three hidden layers and the output unit
__device__ void forward(const Weights &w, Acts &a) {
  dense_relu<NIN, LDI, LDI>(w.W1, w.b1, a.X, a.H1);
  __syncthreads();
  dense_relu<HID, LD, LD>(w.W2, w.b2, a.H1, a.H2);
  __syncthreads();
  dense_relu<HID, LD, LD>(w.W3, w.b3, a.H2, a.H3);
  __syncthreads();
  if (threadIdx.x < NS) {
    float acc = w.b4;
    for (int j = 0; j < HID; j++) acc = fmaf(w.W4[j], a.H3[threadIdx.x][j], acc);
    a.out[threadIdx.x] = acc;
  }
  __syncthreads();
}

// counter-based index hash (splitmix64 finaliser)
__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
  z += 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}

struct GradArgs {
  const float *x;        // [n][NIN]
  const float *y;        // [n]
  long long n;
  int batch;
  unsigned long long seed;
  const int *step;       // device step counter of the hashed draw (null: samples 0, 1, ...)
  const __nv_bfloat16 *wb;
  float *part;           // [nunit][NPARAM]
  float *loss_part;      // [nunit]
};

// ---- gradient -------------------------------------------------------------------
// Forward and backward of the mean squared error.  A CTA is two units of 128
// threads; a unit takes 64 samples at a time, and the weight gradients of all its
// samples stay in its registers.  Activations lie in shared memory as
// [neuron][sample], so that
//  * a layer is, per input neuron k, 8 samples of row k (two 16-byte loads) times 4
//    weights of row k (one load): a tile of 8 x 4 outputs a thread;
//  * a weight gradient is, per 4 samples, 8 rows of errors times 4 rows of inputs:
//    12 loads and 128 products, again 8 x 4 outputs a thread;
// both in packed FP32 pairs of samples.  The weights are there in both orders.
// Bound by the FP32 pipes and their operand loads (1.8e9 multiply-adds at 65,536
// samples, 49 us at the pipes' rate; 8 warps an SM): 101 us, against 302 us with one weight and one
// broadcast activation loaded for every product.
constexpr int GU = 128;      // threads of a unit
constexpr int GP = NS + 4;   // row pitch (floats): 8 rows' 16-byte loads hit all banks
constexpr int kGradSMs = 148;

typedef unsigned long long f32x2;  // two packed FP32

__device__ __forceinline__ void fma2(f32x2 &d, f32x2 a, f32x2 b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ f32x2 pack2(float a, float b) {
  f32x2 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}

struct GradUnit {  // shared memory of a unit
  float X[NIN][GP];
  float H1[HID][GP], H2[HID][GP], D[HID][GP];
  float red[4][NS];  // output unit: partial sums of the four warps
  float y[NS];
};
struct GradSmem {
  float W1t[NIN][HID];             // [input][output]
  float W2t[HID][GP], W3t[HID][GP];
  float W2[HID][GP], W3[HID][GP];  // [output][input]
  float b1[HID], b2[HID], b3[HID], W4[HID];
  float b4, pad[3];
  GradUnit u[2];
};

__device__ __forceinline__ void unit_sync(int unit) {
  asm volatile("bar.sync %0, %1;" ::"r"(unit + 1), "r"(GU) : "memory");
}

// acc[c][q] += sum_k W[k][i0 + c] A[k][samples of q]; q: pairs at s0, s0 + 2, s0 + 32, s0 + 34
template <int K>
__device__ __forceinline__ void tile_layer(const float *W, int ldw, const float *A, int i0, int s0,
                                           f32x2 (&acc)[4][4]) {
#pragma unroll 8
  for (int k = 0; k < K; k++) {
    const float4 w = *reinterpret_cast<const float4 *>(W + k * ldw + i0);
    const ulonglong2 a0 = *reinterpret_cast<const ulonglong2 *>(A + k * GP + s0);
    const ulonglong2 a1 = *reinterpret_cast<const ulonglong2 *>(A + k * GP + s0 + 32);
    const float wv[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int c = 0; c < 4; c++) {
      const f32x2 ww = pack2(wv[c], wv[c]);
      fma2(acc[c][0], ww, a0.x);
      fma2(acc[c][1], ww, a0.y);
      fma2(acc[c][2], ww, a1.x);
      fma2(acc[c][3], ww, a1.y);
    }
  }
}

// the tile's 4 x 8 values, row c = neuron i0 + c, v[c][0..3] at s0, v[c][4..7] at s0 + 32
__device__ __forceinline__ void tile_values(const f32x2 (&acc)[4][4], float (&v)[4][8]) {
#pragma unroll
  for (int c = 0; c < 4; c++)
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const float2 f = unpack2(acc[c][q]);
      v[c][2 * q] = f.x;
      v[c][2 * q + 1] = f.y;
    }
}

__device__ __forceinline__ void tile_store(float *H, int i0, int s0, const float (&v)[4][8]) {
#pragma unroll
  for (int c = 0; c < 4; c++) {
    float *r = H + (i0 + c) * GP + s0;
    *reinterpret_cast<float4 *>(r) = make_float4(v[c][0], v[c][1], v[c][2], v[c][3]);
    *reinterpret_cast<float4 *>(r + 32) = make_float4(v[c][4], v[c][5], v[c][6], v[c][7]);
  }
}

// H = relu(b + W A) of the unit's 64 samples; v keeps the thread's tile
template <int K>
__device__ __forceinline__ void tile_relu(const float *W, int ldw, const float *b, const float *A,
                                          int i0, int s0, float (&v)[4][8]) {
  f32x2 acc[4][4];
#pragma unroll
  for (int c = 0; c < 4; c++)
#pragma unroll
    for (int q = 0; q < 4; q++) acc[c][q] = pack2(b[i0 + c], b[i0 + c]);
  tile_layer<K>(W, ldw, A, i0, s0, acc);
  tile_values(acc, v);
#pragma unroll
  for (int c = 0; c < 4; c++)
#pragma unroll
    for (int e = 0; e < 8; e++) v[c][e] = fmaxf(v[c][e], 0.f);
}

// errors of the layer below: v = (H > 0) W^T D, and their sums over the tile's samples
__device__ __forceinline__ void tile_back(const float *W, const float *D, const float *H, int i0,
                                          int s0, float (&v)[4][8], float (&gb)[4]) {
  f32x2 acc[4][4];
#pragma unroll
  for (int c = 0; c < 4; c++)
#pragma unroll
    for (int q = 0; q < 4; q++) acc[c][q] = 0ull;
  tile_layer<HID>(W, GP, D, i0, s0, acc);
  tile_values(acc, v);
#pragma unroll
  for (int c = 0; c < 4; c++) {
    const float *r = H + (i0 + c) * GP + s0;
    const float4 h0 = *reinterpret_cast<const float4 *>(r);
    const float4 h1 = *reinterpret_cast<const float4 *>(r + 32);
    const float h[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
    float sum = 0.f;
#pragma unroll
    for (int e = 0; e < 8; e++) {
      v[c][e] = h[e] > 0.f ? v[c][e] : 0.f;
      sum += v[c][e];
    }
    gb[c] += sum;
  }
}

// g[r][c] += sum_s D[ig + 8r][s] H[jg + 16c][s] over the unit's 64 samples
template <int NC>
__device__ __forceinline__ void tile_outer(const float *D, const float *H, int ig, int jg,
                                           float (&g)[8][NC]) {
  f32x2 acc[8][NC];
#pragma unroll
  for (int r = 0; r < 8; r++)
#pragma unroll
    for (int c = 0; c < NC; c++) acc[r][c] = 0ull;
#pragma unroll 2
  for (int s = 0; s < NS; s += 4) {
    ulonglong2 h[NC];
#pragma unroll
    for (int c = 0; c < NC; c++)
      h[c] = *reinterpret_cast<const ulonglong2 *>(H + (jg + 16 * c) * GP + s);
#pragma unroll
    for (int r = 0; r < 8; r++) {
      const ulonglong2 d = *reinterpret_cast<const ulonglong2 *>(D + (ig + 8 * r) * GP + s);
#pragma unroll
      for (int c = 0; c < NC; c++) {
        fma2(acc[r][c], d.x, h[c].x);
        fma2(acc[r][c], d.y, h[c].y);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < 8; r++)
#pragma unroll
    for (int c = 0; c < NC; c++) {
      const float2 f = unpack2(acc[r][c]);
      g[r][c] += f.x + f.y;
    }
}

// unit u (of 2 gridDim.x) takes samples 64 u .. 64 u + 63, then 128 gridDim.x further
__global__ void __launch_bounds__(2 * GU, 1) mlp_grad_kernel(GradArgs g) {
  extern __shared__ __align__(16) unsigned char smem[];
  GradSmem &S = *reinterpret_cast<GradSmem *>(smem);
  for (int e = threadIdx.x; e < HID * NIN; e += 2 * GU)
    S.W1t[e % NIN][e / NIN] = __bfloat162float(g.wb[P_W1 + e]);
  for (int e = threadIdx.x; e < HID * HID; e += 2 * GU) {
    const float w2 = __bfloat162float(g.wb[P_W2 + e]), w3 = __bfloat162float(g.wb[P_W3 + e]);
    S.W2[e / HID][e % HID] = w2;
    S.W2t[e % HID][e / HID] = w2;
    S.W3[e / HID][e % HID] = w3;
    S.W3t[e % HID][e / HID] = w3;
  }
  if (threadIdx.x < HID) {
    const int e = threadIdx.x;
    S.b1[e] = __bfloat162float(g.wb[P_B1 + e]);
    S.b2[e] = __bfloat162float(g.wb[P_B2 + e]);
    S.b3[e] = __bfloat162float(g.wb[P_B3 + e]);
    S.W4[e] = __bfloat162float(g.wb[P_W4 + e]);
    if (e == 0) S.b4 = __bfloat162float(g.wb[P_B4]);
  }
  __syncthreads();
  const int half = threadIdx.x / GU, t = threadIdx.x % GU;
  const int warp = t >> 5, lane = t & 31;
  const int unit = half * gridDim.x + blockIdx.x;
  const int nset = (g.batch + NS - 1) / NS;
  if (unit >= nset) return;  // no barrier of the whole CTA from here on
  GradUnit &U = S.u[half];
  const int lo = lane & 7, hi = (lane >> 3) + 4 * warp;  // 8 x 16 threads of a unit
  const int s0 = 4 * lo, i0 = 4 * hi;                    // layers: 8 samples, 4 neurons
  const int st = g.step ? *g.step : 0;
  const float inv_b = 1.f / (float)g.batch;
  float gw3[8][4], gw2[8][4], gw1[8][1], gw1b = 0.f;  // entries (lo + 8r, hi + 16c)
  float gb1[4], gb2[4], gb3[4], gw4[4], gb4 = 0.f, loss = 0.f;
#pragma unroll
  for (int r = 0; r < 8; r++) {
    gw1[r][0] = 0.f;
#pragma unroll
    for (int c = 0; c < 4; c++) gw3[r][c] = gw2[r][c] = 0.f;
  }
#pragma unroll
  for (int c = 0; c < 4; c++) gb1[c] = gb2[c] = gb3[c] = gw4[c] = 0.f;

  // this set's inputs, loaded ahead: thread t takes elements t + 128 k of [sample][input]
  constexpr int NX = NS * NIN / GU;
  static_assert(NX * GU == NS * NIN, "inputs of a set");
  float xv[NX], yv = 0.f;
  auto fetch = [&](int set) {
    const int b0 = set * NS, cnt = min(NS, g.batch - b0);
    auto row = [&](int s) -> long long {
      const long long r = b0 + s;
      return g.step ? (long long)(mix64(g.seed ^ ((unsigned long long)st << 32) ^
                                        (unsigned long long)r) % (unsigned long long)g.n)
                    : r;
    };
#pragma unroll
    for (int k = 0; k < NX; k++) {
      const int e = t + k * GU, s = e / NIN, j = e - s * NIN;
      xv[k] = s < cnt ? g.x[row(s) * NIN + j] : 0.f;
    }
    if (t < cnt) yv = g.y[row(t)];
  };
  fetch(unit);
#pragma unroll 1
  for (int set = unit; set < nset; set += 2 * gridDim.x) {
    const int cnt = min(NS, g.batch - set * NS);
#pragma unroll
    for (int k = 0; k < NX; k++) {
      const int e = t + k * GU, s = e / NIN, j = e - s * NIN;
      U.X[j][s] = xv[k];
    }
    if (t < NS) U.y[t] = yv;
    unit_sync(half);
    float v[4][8];
    tile_relu<NIN>(&S.W1t[0][0], HID, S.b1, &U.X[0][0], i0, s0, v);
    tile_store(&U.H1[0][0], i0, s0, v);
    unit_sync(half);
    tile_relu<HID>(&S.W2t[0][0], GP, S.b2, &U.H1[0][0], i0, s0, v);
    tile_store(&U.H2[0][0], i0, s0, v);
    unit_sync(half);
    tile_relu<HID>(&S.W3t[0][0], GP, S.b3, &U.H2[0][0], i0, s0, v);
    // output unit: the tile's 4 neurons, the warp's 16, then the four warps'
    {
      float o[8];
#pragma unroll
      for (int e = 0; e < 8; e++) {
        o[e] = 0.f;
#pragma unroll
        for (int c = 0; c < 4; c++) o[e] = fmaf(S.W4[i0 + c], v[c][e], o[e]);
        o[e] += __shfl_xor_sync(0xffffffffu, o[e], 8);
        o[e] += __shfl_xor_sync(0xffffffffu, o[e], 16);
      }
      if (lane < 8) {
        *reinterpret_cast<float4 *>(&U.red[warp][s0]) = make_float4(o[0], o[1], o[2], o[3]);
        *reinterpret_cast<float4 *>(&U.red[warp][s0 + 32]) = make_float4(o[4], o[5], o[6], o[7]);
      }
    }
    unit_sync(half);
    {
      float dout[8];
#pragma unroll
      for (int e = 0; e < 8; e++) {
        const int s = s0 + (e & 3) + (e >> 2) * 32;
        const float o = S.b4 + ((U.red[0][s] + U.red[1][s]) + (U.red[2][s] + U.red[3][s]));
        const float r = s < cnt ? o - U.y[s] : 0.f;
        dout[e] = 2.f * r * inv_b;
        if (hi == 0) {
          loss = fmaf(r, r, loss);
          gb4 += dout[e];
        }
      }
#pragma unroll
      for (int c = 0; c < 4; c++) {
        const float w4 = S.W4[i0 + c];
        float a = 0.f, b = 0.f;
#pragma unroll
        for (int e = 0; e < 8; e++) {
          a = fmaf(dout[e], v[c][e], a);
          v[c][e] = v[c][e] > 0.f ? w4 * dout[e] : 0.f;
          b += v[c][e];
        }
        gw4[c] += a;
        gb3[c] += b;
      }
    }
    tile_store(&U.D[0][0], i0, s0, v);
    unit_sync(half);
    if (set + 2 * gridDim.x < nset) fetch(set + 2 * gridDim.x);
    tile_outer(&U.D[0][0], &U.H2[0][0], lo, hi, gw3);
    tile_back(&S.W3[0][0], &U.D[0][0], &U.H2[0][0], i0, s0, v, gb2);
    unit_sync(half);
    tile_store(&U.H2[0][0], i0, s0, v);  // the errors of layer 2 in place of its outputs
    unit_sync(half);
    tile_outer(&U.H2[0][0], &U.H1[0][0], lo, hi, gw2);
    tile_back(&S.W2[0][0], &U.H2[0][0], &U.H1[0][0], i0, s0, v, gb1);
    tile_store(&U.D[0][0], i0, s0, v);
    unit_sync(half);
    // first layer: inputs 0..15 as above, the last two one entry a thread
    tile_outer(&U.D[0][0], &U.X[0][0], lo, hi, gw1);
    {
      const float *d = U.D[t % HID], *x = U.X[16 + t / HID];
      float a = 0.f;
#pragma unroll 4
      for (int s = 0; s < NS; s += 4) {
        const float4 dv = *reinterpret_cast<const float4 *>(d + s);
        const float4 xv = *reinterpret_cast<const float4 *>(x + s);
        a = fmaf(dv.x, xv.x, fmaf(dv.y, xv.y, fmaf(dv.z, xv.z, fmaf(dv.w, xv.w, a))));
      }
      gw1b += a;
    }
    unit_sync(half);
  }
  static_assert(NIN == 18 && GU == 2 * HID, "first layer's gradient tile");
  float *part = g.part + (size_t)unit * NPARAM;
#pragma unroll
  for (int r = 0; r < 8; r++) {
    const int i = lo + 8 * r;
#pragma unroll
    for (int c = 0; c < 4; c++) {
      part[P_W3 + i * HID + hi + 16 * c] = gw3[r][c];
      part[P_W2 + i * HID + hi + 16 * c] = gw2[r][c];
    }
    part[P_W1 + i * NIN + hi] = gw1[r][0];
  }
  part[P_W1 + (t % HID) * NIN + 16 + t / HID] = gw1b;
#pragma unroll
  for (int h = 4; h > 0; h >>= 1) {
#pragma unroll
    for (int c = 0; c < 4; c++) {
      gb1[c] += __shfl_xor_sync(0xffffffffu, gb1[c], h);
      gb2[c] += __shfl_xor_sync(0xffffffffu, gb2[c], h);
      gb3[c] += __shfl_xor_sync(0xffffffffu, gb3[c], h);
      gw4[c] += __shfl_xor_sync(0xffffffffu, gw4[c], h);
    }
    gb4 += __shfl_xor_sync(0xffffffffu, gb4, h);
    loss += __shfl_xor_sync(0xffffffffu, loss, h);
  }
  if (lo == 0) {
#pragma unroll
    for (int c = 0; c < 4; c++) {
      part[P_B1 + i0 + c] = gb1[c];
      part[P_B2 + i0 + c] = gb2[c];
      part[P_B3 + i0 + c] = gb3[c];
      part[P_W4 + i0 + c] = gw4[c];
    }
  }
  if (t == 0) {
    part[P_B4] = gb4;
    g.loss_part[unit] = loss * inv_b;
  }
}

// CTAs of a batch, and the units that write a partial gradient
int grad_grid(int batch) { return std::min((batch + NS - 1) / NS, kGradSMs); }
int grad_units(int batch) { return std::min((batch + NS - 1) / NS, 2 * kGradSMs); }

struct AdamArgs {
  const float *part;
  const float *loss_part;
  int nunit;
  float *master, *m, *v;
  __nv_bfloat16 *wb;
  float *grad_out;  // optional: the summed gradient
  float *loss_hist;
  const int *step;  // null: step 0
  float lr, beta1, beta2, eps;
  int apply;        // 0: only sum the gradient (and loss)
};

// Sum the partial gradients in a fixed order, 32 parameters a block and every eighth
// partial a thread, all loads coalesced (one thread a parameter over 1,024 partials:
// 41 us, bound by the latency of its loads; 5.8 us over 296); Adam on the FP32 master
// weights.
constexpr int kAdamP = 32, kAdamK = 8;
__global__ void __launch_bounds__(kAdamP *kAdamK) mlp_adam_kernel(AdamArgs a) {
  __shared__ float sum[kAdamK][kAdamP];
  const int c = threadIdx.x % kAdamP, k = threadIdx.x / kAdamP;
  const int p = blockIdx.x * kAdamP + c;
  const int t = (a.step ? *a.step : 0) + 1;
  float part = 0.f;
  if (p < NPARAM) {
#pragma unroll 8
    for (int b = k; b < a.nunit; b += kAdamK) part += a.part[(size_t)b * NPARAM + p];
  }
  sum[k][c] = part;
  __syncthreads();
  if (k == 0 && p < NPARAM) {
    float g = 0.f;
    for (int i = 0; i < kAdamK; i++) g += sum[i][c];
    if (a.grad_out) a.grad_out[p] = g;
    if (a.apply) {
      const float m = a.beta1 * a.m[p] + (1.f - a.beta1) * g;
      const float v = a.beta2 * a.v[p] + (1.f - a.beta2) * g * g;
      a.m[p] = m;
      a.v[p] = v;
      const float mh = m / (1.f - powf(a.beta1, (float)t));
      const float vh = v / (1.f - powf(a.beta2, (float)t));
      const float th = a.master[p] - a.lr * mh / (sqrtf(vh) + a.eps);
      a.master[p] = th;
      a.wb[p] = __float2bfloat16_rn(th);
    }
  }
  if (blockIdx.x == 0 && k == 1) {
    float l = 0.f;
    for (int b = c; b < a.nunit; b += 32) l += a.loss_part[b];
    for (int h = 16; h > 0; h >>= 1) l += __shfl_xor_sync(0xffffffffu, l, h);
    if (c == 0 && a.loss_hist) a.loss_hist[t - 1] = l;
  }
}
constexpr unsigned kAdamGrid = (NPARAM + kAdamP - 1) / kAdamP;

__global__ void mlp_step_kernel(int *step) { *step += 1; }

__global__ void to_bf16_kernel(const float *__restrict__ m, __nv_bfloat16 *__restrict__ wb, int n) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < n) wb[p] = __float2bfloat16_rn(m[p]);
}

// inference: w = exp(sigma * out + mu) per sample
__global__ void __launch_bounds__(NT) mlp_infer_kernel(const float *__restrict__ x, long long n,
                                                       const __nv_bfloat16 *__restrict__ wb,
                                                       float mu, float sigma,
                                                       float *__restrict__ yhat,
                                                       double *__restrict__ wout) {
  extern __shared__ __align__(16) unsigned char smem[];
  Weights &w = *reinterpret_cast<Weights *>(smem);
  Acts &a = *reinterpret_cast<Acts *>(smem + sizeof(Weights));
  load_weights(w, wb);
  for (long long b0 = (long long)blockIdx.x * NS; b0 < n; b0 += (long long)gridDim.x * NS) {
    const int cnt = (int)min((long long)NS, n - b0);
    __syncthreads();
    for (int e = threadIdx.x; e < NS * NIN; e += NT) {
      const int s = e / NIN, j = e % NIN;
      a.X[s][j] = s < cnt ? x[(b0 + s) * NIN + j] : 0.f;
    }
    __syncthreads();
    forward(w, a);
    if (threadIdx.x < cnt) {
      const float o = a.out[threadIdx.x];
      if (yhat) yhat[b0 + threadIdx.x] = o;
      if (wout) wout[b0 + threadIdx.x] = exp((double)sigma * (double)o + (double)mu);
    }
  }
}

// ------------------------------------------------------------------------
// Inference on the tensor cores: mma.sync m16n8k16, BF16 operands, FP32
// accumulation.  A warp takes 16 samples at a time; the weights are exact
// BF16 (B operands, row-major W[out][in] is the column-major B the
// instruction wants), the FP32 activations enter as the sum of NTERM BF16
// terms (hi, then the BF16 rounding of each remainder), smallest term first,
// so that the products carry the activations to about 8 NTERM bits.  The D
// fragments of n-tiles 2k and 2k+1 are the A fragment of k-tile k of the next
// layer, so the activations stay in registers from layer to layer.
// Fragment layout (PTX ISA, m16n8k16 .bf16): g = lane / 4, t = lane % 4;
// A: a0 (row g, cols 2t, 2t+1), a1 (row g + 8), a2 (cols 2t + 8, 2t + 9),
// a3 (row g + 8, cols 2t + 8, 2t + 9); B: b0 (k 2t, 2t+1; n g), b1 (k 2t + 8,
// 2t + 9; n g); C/D: c0, c1 (row g, cols 2t, 2t+1), c2, c3 (row g + 8).
constexpr int MW1 = 40;  // W1 rows in shared memory: 18 inputs, zero-padded to 32, + 8 pad
constexpr int MWH = 72;  // W2, W3 rows: 64 + 8 pad (conflict-free B loads)

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0,
                                         uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t pack_bf16(__nv_bfloat16 lo, __nv_bfloat16 hi) {
  return (uint32_t)__bfloat16_as_ushort(lo) | ((uint32_t)__bfloat16_as_ushort(hi) << 16);
}

// the NTERM BF16 terms of (v0, v1) packed as pairs, term 0 the largest
template <int NTERM>
__device__ __forceinline__ void split_pair(float v0, float v1, uint32_t (&t)[NTERM]) {
#pragma unroll
  for (int k = 0; k < NTERM; k++) {
    const __nv_bfloat16 h0 = __float2bfloat16_rn(v0), h1 = __float2bfloat16_rn(v1);
    t[k] = pack_bf16(h0, h1);
    v0 -= __bfloat162float(h0);
    v1 -= __bfloat162float(h1);
  }
}

// A fragments (NTERM terms) of k-tile kt from the previous layer's D fragments
template <int NTERM>
__device__ __forceinline__ void a_from_d(const float (&h)[8][4], int kt, uint32_t (&a)[NTERM][4]) {
  uint32_t t0[NTERM], t1[NTERM], t2[NTERM], t3[NTERM];
  split_pair<NTERM>(h[2 * kt][0], h[2 * kt][1], t0);
  split_pair<NTERM>(h[2 * kt][2], h[2 * kt][3], t1);
  split_pair<NTERM>(h[2 * kt + 1][0], h[2 * kt + 1][1], t2);
  split_pair<NTERM>(h[2 * kt + 1][2], h[2 * kt + 1][3], t3);
#pragma unroll
  for (int k = 0; k < NTERM; k++) {
    a[k][0] = t0[k];
    a[k][1] = t1[k];
    a[k][2] = t2[k];
    a[k][3] = t3[k];
  }
}

// out[8][4] = bias + A W^T over KT k-tiles (A given per k-tile by `afrag`)
template <int NTERM, int KT, int LDW, class AF>
__device__ __forceinline__ void mma_layer(const __nv_bfloat16 *__restrict__ W, const float *bias,
                                          AF afrag, float (&out)[8][4]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int nt = 0; nt < 8; nt++) {
    const float b0 = bias[nt * 8 + 2 * t], b1 = bias[nt * 8 + 2 * t + 1];
    out[nt][0] = b0;
    out[nt][1] = b1;
    out[nt][2] = b0;
    out[nt][3] = b1;
  }
#pragma unroll
  for (int kt = 0; kt < KT; kt++) {
    uint32_t a[NTERM][4];
    afrag(kt, a);
#pragma unroll
    for (int nt = 0; nt < 8; nt++) {
      const __nv_bfloat16 *wr = W + (nt * 8 + g) * LDW + kt * 16 + 2 * t;
      const uint32_t b0 = *reinterpret_cast<const uint32_t *>(wr);
      const uint32_t b1 = *reinterpret_cast<const uint32_t *>(wr + 8);
#pragma unroll
      for (int k = NTERM - 1; k >= 0; k--) mma_bf16(out[nt], a[k], b0, b1);
    }
  }
}

__device__ __forceinline__ void relu8(float (&h)[8][4]) {
#pragma unroll
  for (int nt = 0; nt < 8; nt++)
#pragma unroll
    for (int e = 0; e < 4; e++) h[nt][e] = fmaxf(h[nt][e], 0.f);
}

template <int NTERM>
__global__ void __launch_bounds__(NT, 2) mlp_infer_mma_kernel(const float *__restrict__ x, long long n,
                                                           const __nv_bfloat16 *__restrict__ wb,
                                                           float mu, float sigma,
                                                           float *__restrict__ yhat,
                                                           double *__restrict__ wout) {
  __shared__ __align__(16) __nv_bfloat16 sW1[HID * MW1];
  __shared__ __align__(16) __nv_bfloat16 sW2[HID * MWH];
  __shared__ __align__(16) __nv_bfloat16 sW3[HID * MWH];
  __shared__ float sb1[HID], sb2[HID], sb3[HID], sW4[HID];
  __shared__ float sb4;
  for (int e = threadIdx.x; e < HID * 32; e += NT) {
    const int r = e / 32, k = e % 32;
    sW1[r * MW1 + k] = k < NIN ? wb[P_W1 + r * NIN + k] : __float2bfloat16_rn(0.f);
  }
  for (int e = threadIdx.x; e < HID * HID; e += NT) {
    sW2[(e / HID) * MWH + e % HID] = wb[P_W2 + e];
    sW3[(e / HID) * MWH + e % HID] = wb[P_W3 + e];
  }
  for (int e = threadIdx.x; e < HID; e += NT) {
    sb1[e] = __bfloat162float(wb[P_B1 + e]);
    sb2[e] = __bfloat162float(wb[P_B2 + e]);
    sb3[e] = __bfloat162float(wb[P_B3 + e]);
    sW4[e] = __bfloat162float(wb[P_W4 + e]);
  }
  if (threadIdx.x == 0) sb4 = __bfloat162float(wb[P_B4]);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const long long ngrp = (n + 15) / 16;
  for (long long grp = (long long)blockIdx.x * (NT / 32) + warp; grp < ngrp;
       grp += (long long)gridDim.x * (NT / 32)) {
    const long long r0 = grp * 16 + g, r1 = r0 + 8;
    // the features of rows r0, r1 at this lane's columns (zero past 18 and past n)
    auto feat = [&](long long r, int k) -> float {
      return (r < n && k < NIN) ? __ldg(x + r * NIN + k) : 0.f;
    };
    float h1[8][4], h2[8][4];
    mma_layer<NTERM, 2, MW1>(sW1, sb1, [&](int kt, uint32_t (&a)[NTERM][4]) {
      const int k0 = kt * 16 + 2 * t;
      uint32_t t0[NTERM], t1[NTERM], t2[NTERM], t3[NTERM];
      split_pair<NTERM>(feat(r0, k0), feat(r0, k0 + 1), t0);
      split_pair<NTERM>(feat(r1, k0), feat(r1, k0 + 1), t1);
      split_pair<NTERM>(feat(r0, k0 + 8), feat(r0, k0 + 9), t2);
      split_pair<NTERM>(feat(r1, k0 + 8), feat(r1, k0 + 9), t3);
#pragma unroll
      for (int k = 0; k < NTERM; k++) {
        a[k][0] = t0[k];
        a[k][1] = t1[k];
        a[k][2] = t2[k];
        a[k][3] = t3[k];
      }
    }, h1);
    relu8(h1);
    mma_layer<NTERM, 4, MWH>(sW2, sb2, [&](int kt, uint32_t (&a)[NTERM][4]) {
      a_from_d<NTERM>(h1, kt, a);
    }, h2);
    relu8(h2);
    mma_layer<NTERM, 4, MWH>(sW3, sb3, [&](int kt, uint32_t (&a)[NTERM][4]) {
      a_from_d<NTERM>(h2, kt, a);
    }, h1);
    relu8(h1);
    // output unit: the quad of lanes sharing g holds all 64 columns of rows r0, r1
    float o0 = 0.f, o1 = 0.f;
#pragma unroll
    for (int nt = 0; nt < 8; nt++) {
      const float w0 = sW4[nt * 8 + 2 * t], w1 = sW4[nt * 8 + 2 * t + 1];
      o0 = fmaf(w0, h1[nt][0], fmaf(w1, h1[nt][1], o0));
      o1 = fmaf(w0, h1[nt][2], fmaf(w1, h1[nt][3], o1));
    }
    o0 += __shfl_xor_sync(0xffffffffu, o0, 1);
    o1 += __shfl_xor_sync(0xffffffffu, o1, 1);
    o0 += __shfl_xor_sync(0xffffffffu, o0, 2);
    o1 += __shfl_xor_sync(0xffffffffu, o1, 2);
    if (t == 0) {
      o0 += sb4;
      o1 += sb4;
      if (r0 < n) {
        if (yhat) yhat[r0] = o0;
        if (wout) wout[r0] = exp((double)sigma * (double)o0 + (double)mu);
      }
      if (r1 < n) {
        if (yhat) yhat[r1] = o1;
        if (wout) wout[r1] = exp((double)sigma * (double)o1 + (double)mu);
      }
    }
  }
}

constexpr size_t kGradSmem = sizeof(GradSmem);
static_assert(kGradSmem <= 227 * 1024, "one CTA an SM");
constexpr size_t kInferSmem = sizeof(Weights) + sizeof(Acts);

}  // namespace

struct mirt_mlp {
  DMem master, m, v, wb, part, loss_part, step, grad, losses;
  int nunit_cap = 0;
  int tensor_cores = 1;  // inference on mma.sync (1) or on the FP32 pipes (0)
  float lr = 1e-3f, beta1 = 0.9f, beta2 = 0.999f, eps = 1e-8f;
};

namespace {

int ensure_batch(mirt_mlp *q, int batch) {
  const int nunit = grad_units(batch);
  if (nunit > q->nunit_cap) {
    MCK(q->part.alloc((size_t)nunit * NPARAM * sizeof(float)));
    MCK(q->loss_part.alloc((size_t)nunit * sizeof(float)));
    q->nunit_cap = nunit;
  }
  return MIRT_OK;
}

int set_attrs() {
  static bool done = false;
  if (done) return MIRT_OK;
  MCK(cudaFuncSetAttribute(mlp_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)kGradSmem));
  MCK(cudaFuncSetAttribute(mlp_infer_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)kInferSmem));
  done = true;
  return MIRT_OK;
}

GradArgs grad_args(mirt_mlp *q, const float *x, const float *y, long long n, int batch,
                   unsigned long long seed, const int *step) {
  GradArgs g{};
  g.x = x;
  g.y = y;
  g.n = n;
  g.batch = batch;
  g.seed = seed;
  g.step = step;
  g.wb = q->wb.as<__nv_bfloat16>();
  g.part = q->part.as<float>();
  g.loss_part = q->loss_part.as<float>();
  return g;
}

AdamArgs adam_args(mirt_mlp *q, int nunit, int apply, float *grad_out, float *loss_hist,
                   const int *step) {
  AdamArgs a{};
  a.part = q->part.as<float>();
  a.loss_part = q->loss_part.as<float>();
  a.nunit = nunit;
  a.master = q->master.as<float>();
  a.m = q->m.as<float>();
  a.v = q->v.as<float>();
  a.wb = q->wb.as<__nv_bfloat16>();
  a.grad_out = grad_out;
  a.loss_hist = loss_hist;
  a.step = step;
  a.lr = q->lr;
  a.beta1 = q->beta1;
  a.beta2 = q->beta2;
  a.eps = q->eps;
  a.apply = apply;
  return a;
}

}  // namespace

extern "C" {

int mirt_mlp_create(mirt_mlp **out, const float *params) {
  if (!out || !params) return api_fail(MIRT_ERR_ARG, "NULL argument");
  *out = nullptr;
  int rc = set_attrs();
  if (rc) return rc;
  auto *q = new mirt_mlp();
  auto bail = [&](int code) {
    delete q;
    return code;
  };
  if (q->master.alloc(NPARAM * sizeof(float)) || q->m.alloc(NPARAM * sizeof(float)) ||
      q->v.alloc(NPARAM * sizeof(float)) || q->wb.alloc(NPARAM * sizeof(__nv_bfloat16)) ||
      q->step.alloc(sizeof(int)) || q->grad.alloc((NPARAM + 1) * sizeof(float)))
    return bail(api_fail(MIRT_ERR_ALLOC, "MLP parameter buffers"));
  cudaError_t e = cudaMemcpy(q->master.p, params, NPARAM * sizeof(float), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemset(q->m.p, 0, NPARAM * sizeof(float));
  if (e == cudaSuccess) e = cudaMemset(q->v.p, 0, NPARAM * sizeof(float));
  if (e == cudaSuccess) e = cudaMemset(q->step.p, 0, sizeof(int));
  if (e == cudaSuccess) {
    to_bf16_kernel<<<(NPARAM + 255) / 256, 256>>>(q->master.as<float>(),
                                                  q->wb.as<__nv_bfloat16>(), NPARAM);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaDeviceSynchronize();
  if (e != cudaSuccess) return bail(api_fail(MIRT_ERR_CUDA, cudaGetErrorString(e)));
  *out = q;
  return MIRT_OK;
}

int mirt_mlp_params(mirt_mlp *q, float *params) {
  if (!q || !params) return api_fail(MIRT_ERR_ARG, "NULL argument");
  MCK(cudaMemcpy(params, q->master.p, NPARAM * sizeof(float), cudaMemcpyDeviceToHost));
  return MIRT_OK;
}

int mirt_mlp_grad(mirt_mlp *q, const float *x, const float *y, int64_t n, float *grad,
                  float *loss, void *stream) try {
  if (!q || !x || !y || !grad) return api_fail(MIRT_ERR_ARG, "NULL argument");
  if (n < 1 || n > (1 << 30)) return api_fail(MIRT_ERR_ARG, "need 1 <= n <= 2^30");
  cudaStream_t st = as_stream(stream);
  int rc = ensure_batch(q, (int)n);
  if (rc) return rc;
  // the loss behind the gradient, so that one copy brings both
  std::vector<float> host(NPARAM + 1);
  float *dg = q->grad.as<float>();
  mlp_grad_kernel<<<grad_grid((int)n), 2 * GU, kGradSmem, st>>>(
      grad_args(q, x, y, n, (int)n, 0, nullptr));
  MCK(cudaGetLastError());
  mlp_adam_kernel<<<kAdamGrid, kAdamP * kAdamK, 0, st>>>(
      adam_args(q, grad_units((int)n), 0, dg, dg + NPARAM, nullptr));
  MCK(cudaGetLastError());
  MCK(cudaMemcpyAsync(host.data(), dg, host.size() * sizeof(float), cudaMemcpyDeviceToHost, st));
  MCK(cudaStreamSynchronize(st));
  std::copy(host.begin(), host.end() - 1, grad);
  const float l = host[NPARAM];
  if (loss) *loss = l;
  return MIRT_OK;
} catch (const std::bad_alloc &) {
  return api_fail(MIRT_ERR_ALLOC, "out of host memory");
}

int mirt_mlp_train(mirt_mlp *q, const float *x, const float *y, int64_t n, int32_t batch,
                   int32_t steps, float lr, uint64_t seed, float *loss_hist, void *stream) try {
  if (!q || !x || !y) return api_fail(MIRT_ERR_ARG, "NULL argument");
  if (n < 1 || batch < 1 || batch > (1 << 24) || steps < 0 || !(lr > 0.f))
    return api_fail(MIRT_ERR_ARG, "need n >= 1, 1 <= batch <= 2^24, steps >= 0, lr > 0");
  cudaStream_t st = as_stream(stream);
  int rc = ensure_batch(q, batch);
  if (rc) return rc;
  q->lr = lr;
  int step0 = 0;
  MCK(cudaMemcpyAsync(&step0, q->step.p, sizeof(int), cudaMemcpyDeviceToHost, st));
  MCK(cudaStreamSynchronize(st));
  MCK(q->losses.alloc((size_t)(step0 + steps + 1) * sizeof(float)));
  const int *step = q->step.as<int>();
  const GradArgs g = grad_args(q, x, y, n, batch, seed, step);
  const AdamArgs a = adam_args(q, grad_units(batch), 1, nullptr, q->losses.as<float>(), step);
  const unsigned grid = (unsigned)grad_grid(batch);
  // one training step = three launches; capture a block of steps in a CUDA
  // graph and replay it (the step counter lives on the device)
  const int chunk = steps < 64 ? steps : 64;
  cudaGraphExec_t exec = nullptr;
  if (chunk > 0) {
    cudaStream_t cs;
    MCK(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
    cudaGraph_t graph;
    cudaError_t e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
    for (int i = 0; i < chunk && e == cudaSuccess; i++) {
      mlp_grad_kernel<<<grid, 2 * GU, kGradSmem, cs>>>(g);
      mlp_adam_kernel<<<kAdamGrid, kAdamP * kAdamK, 0, cs>>>(a);
      mlp_step_kernel<<<1, 1, 0, cs>>>(q->step.as<int>());
    }
    cudaError_t e2 = cudaStreamEndCapture(cs, &graph);
    if (e == cudaSuccess) e = e2;
    if (e == cudaSuccess) e = cudaGraphInstantiate(&exec, graph, 0);
    if (e2 == cudaSuccess) cudaGraphDestroy(graph);
    cudaStreamDestroy(cs);
    if (e != cudaSuccess) return api_fail(MIRT_ERR_CUDA, std::string("training graph: ") + cudaGetErrorString(e));
  }
  int done = 0;
  cudaError_t e = cudaSuccess;
  while (e == cudaSuccess && done + chunk <= steps && chunk > 0) {
    e = cudaGraphLaunch(exec, st);
    done += chunk;
  }
  for (; e == cudaSuccess && done < steps; done++) {
    mlp_grad_kernel<<<grid, 2 * GU, kGradSmem, st>>>(g);
    mlp_adam_kernel<<<kAdamGrid, kAdamP * kAdamK, 0, st>>>(a);
    mlp_step_kernel<<<1, 1, 0, st>>>(q->step.as<int>());
    e = cudaGetLastError();
  }
  if (exec) cudaGraphExecDestroy(exec);
  MCK(e);
  if (loss_hist && steps > 0)
    MCK(cudaMemcpyAsync(loss_hist, q->losses.as<float>() + step0, steps * sizeof(float),
                        cudaMemcpyDeviceToHost, st));
  MCK(cudaStreamSynchronize(st));
  return MIRT_OK;
} catch (const std::bad_alloc &) {
  return api_fail(MIRT_ERR_ALLOC, "out of host memory");
}

int mirt_mlp_infer(mirt_mlp *q, const float *x, int64_t n, float mu, float sigma, float *yhat,
                   double *w, void *stream) {
  if (!q || !x || (!yhat && !w)) return api_fail(MIRT_ERR_ARG, "NULL argument");
  if (n < 0) return api_fail(MIRT_ERR_ARG, "n must be >= 0");
  if (n == 0) return MIRT_OK;
  cudaStream_t st = as_stream(stream);
  if (q->tensor_cores) {
    // tensor-core inference: 8 warps of 16 samples per CTA and pass
    long long nb = (n + 127) / 128;
    if (nb > 148 * 8) nb = 148 * 8;
    mlp_infer_mma_kernel<3><<<(unsigned)nb, NT, 0, st>>>(x, n, q->wb.as<__nv_bfloat16>(), mu,
                                                          sigma, yhat, w);
  } else {
    long long nb = (n + NS - 1) / NS;
    if (nb > 148 * 8) nb = 148 * 8;
    mlp_infer_kernel<<<(unsigned)nb, NT, kInferSmem, st>>>(x, n, q->wb.as<__nv_bfloat16>(), mu,
                                                            sigma, yhat, w);
  }
  MCK(cudaGetLastError());
  return MIRT_OK;
}

int mirt_mlp_set_tensor_cores(mirt_mlp *q, int32_t on) {
  if (!q) return api_fail(MIRT_ERR_ARG, "NULL argument");
  q->tensor_cores = on ? 1 : 0;
  return MIRT_OK;
}

int mirt_mlp_destroy(mirt_mlp *q) {
  if (q) {
    cudaDeviceSynchronize();
    delete q;
  }
  return MIRT_OK;
}

}  // extern "C"
