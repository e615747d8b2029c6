// sense.cu -- batched CG-SENSE on the device NUFFT.
//
// System (systems/Asense.m:53-56): A = [G diag(s_1); ...; G diag(s_C)], G the
// table NUFFT of the plan (one slice per problem, ncol = C coils).  Penalty
// (penalty/Reg1.m with its defaults: first-order differences, offsets
// [1 nx nx+1 nx-1] of penalty/penalty_offsets.m, 'tight' edges and
// distance_power 1 of penalty/Rweights.m): R = C'C = sum_m C_m' diag(w_m) C_m,
// w_m = beta / |offset_m|, over pixel pairs that are both inside the image.
// Solver (wls/qpwls_pcg1.m:94-189 with precon = 1): Fletcher-Reeves directions
// and the real step (ddir' ngrad) / (Adir' W Adir + ddir' R ddir), with Ax
// and R x carried along as the reference carries Ax and Cx.
//
// Every problem of the batch has its own scalars; all reductions are FP64
// (deterministic); vectors are complex64.  The iteration runs without host round
// trips.
//
// Each inner product is formed by the kernel that writes one of its vectors: the
// image kernels run on a grid of P blocks x S problems, a block leaves its sum in
// part[s][block], and the last block of a problem to finish adds the sums in block
// order and updates the problem's scalars.  (One CTA per problem read each vector
// again before: 131 us per product of 5 problems of 24 x 29,184 samples; the
// iteration's vector passes of those problems 0.75 ms -> 0.11 ms.)
#include "../../include/mirt_b200.h"

#include <cmath>
#include <new>
#include <string>
#include <vector>

#include "runtime.cuh"
#include "toeplitz.cuh"

using namespace mirt;

namespace {

#define SCK(call)                                                                     \
  do {                                                                                \
    cudaError_t e_ = (call);                                                          \
    if (e_ != cudaSuccess)                                                            \
      return api_fail(e_ == cudaErrorMemoryAllocation ? MIRT_ERR_ALLOC : MIRT_ERR_CUDA, \
                      std::string(#call) + ": " + cudaGetErrorString(e_));            \
  } while (0)

enum { SC_NEW = 0, SC_OLD, SC_GAMMA, SC_STEP, SC_DEN, SC_NUM, SC_DENR, SC_N };

unsigned nblocks(long long n, int t = 256) {
  long long b = (n + t - 1) / t;
  if (b > 148 * 16) b = 148 * 16;
  return (unsigned)(b < 1 ? 1 : b);
}

// z[s][p][c] = sens[s][p][c] x[s][p]
__global__ void k_expand(const float2 *__restrict__ x, const float2 *__restrict__ sens,
                         float2 *__restrict__ z, long long n, int C) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
       e += (long long)gridDim.x * blockDim.x) {
    const float2 v = x[e / C], s = sens[e];
    z[e] = make_float2(s.x * v.x - s.y * v.y, s.x * v.y + s.y * v.x);
  }
}

// The sum of v over the block (256 threads), in a fixed order, on thread 0.
__device__ __forceinline__ double block_sum(double v) {
  __shared__ double w[8];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  __syncthreads();  // an earlier call's sums are read
  if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0)
    for (int k = 1; k < 8; k++) v += w[k];
  return v;
}

// Partial sums and counters of one inner product per problem: block b of
// problem s = blockIdx.y leaves its sum in part[s][b]; the last one calls
// done(total) on one thread and clears the counter for the next product.
struct DotBuf {
  double *part;
  int *count;
};

template <class F>
__device__ __forceinline__ void finish_dot(DotBuf d, double acc, F done) {
  const int s = blockIdx.y, P = gridDim.x;
  __shared__ bool last;
  acc = block_sum(acc);
  if (threadIdx.x == 0) {
    d.part[s * P + blockIdx.x] = acc;
    __threadfence();
    last = atomicAdd(d.count + s, 1) == P - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double v = 0.0;
  for (int b = threadIdx.x; b < P; b += blockDim.x) v += __ldcg(d.part + s * P + b);
  v = block_sum(v);
  if (threadIdx.x == 0) {
    d.count[s] = 0;
    done(v);
  }
}

// this block's share [q0, q1) of n elements
__device__ __forceinline__ void share(long long n, long long &q0, long long &q1) {
  const long long per = (n + gridDim.x - 1) / gridDim.x;
  q0 = min(n, per * blockIdx.x);
  q1 = min(n, q0 + per);
}

// the scalars of a new gradient product: gamma = new / old (0 on the first
// iteration or old = 0)
__device__ __forceinline__ void new_product(double *c, double v, int first) {
  c[SC_NEW] = v;
  c[SC_GAMMA] = (first || c[SC_OLD] == 0.0) ? 0.0 : v / c[SC_OLD];
  c[SC_OLD] = v;
}

// out[s][p] = sum_c conj(sens) z  (- sub[s][p] when sub is given); eight lanes
// a pixel.  DOT: with <out, out> as the iteration's new gradient product.
template <bool DOT>
__global__ void __launch_bounds__(256) k_combine(const float2 *__restrict__ z,
                                                 const float2 *__restrict__ sens,
                                                 const float2 *__restrict__ sub,
                                                 float2 *__restrict__ out, long long np, int C,
                                                 DotBuf dot, double *sc, int first) {
  const long long base = (long long)blockIdx.y * np;
  long long q0, q1;
  share(np, q0, q1);
  const int l = threadIdx.x & 7;
  double acc = 0.0;
  for (long long b = q0; b < q1; b += 32) {
    const long long q = b + (threadIdx.x >> 3);
    float ar = 0.f, ai = 0.f;
    if (q < q1) {
      const float2 *zp = z + (base + q) * C, *sp = sens + (base + q) * C;
      for (int c = l; c < C; c += 8) {
        const float2 a = sp[c], v = zp[c];
        ar = fmaf(a.x, v.x, fmaf(a.y, v.y, ar));
        ai = fmaf(a.x, v.y, fmaf(-a.y, v.x, ai));
      }
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
      ar += __shfl_xor_sync(0xffffffffu, ar, o);
      ai += __shfl_xor_sync(0xffffffffu, ai, o);
    }
    if (q < q1 && l == 0) {
      if (sub) {
        ar -= sub[base + q].x;
        ai -= sub[base + q].y;
      }
      out[base + q] = make_float2(ar, ai);
      if (DOT) acc += (double)ar * ar + (double)ai * ai;
    }
  }
  if (DOT)
    finish_dot(dot, acc, [&](double v) { new_product(sc + blockIdx.y * SC_N, v, first); });
}

// out[s][p][c] = sens[s][p][c] sn[p]
__global__ void k_maps_sn(const float2 *__restrict__ sens, const float2 *__restrict__ sn,
                          float2 *__restrict__ out, long long n, long long np, int C) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
       e += (long long)gridDim.x * blockDim.x)
    out[e] = cmul(sens[e], sn[e / C % np]);
}

// r = W (y - Ax), W per sample (all coils) or 1
__global__ void k_resid(const float2 *__restrict__ y, const float2 *__restrict__ Ax,
                        const float *__restrict__ W, float2 *__restrict__ r, long long n, int C) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
       e += (long long)gridDim.x * blockDim.x) {
    const float w = W ? W[e / C] : 1.f;
    r[e] = make_float2(w * (y[e].x - Ax[e].x), w * (y[e].y - Ax[e].y));
  }
}

// out = C'C x for the four offsets (1,0) (0,1) (1,1) (-1,1) in (n1, n2).  DOT:
// with <x, out> as the penalty's share of the curvature.
template <bool DOT>
__global__ void __launch_bounds__(256) k_reg(const float2 *__restrict__ x, float2 *__restrict__ out,
                                             int N1, int N2, const double *__restrict__ beta,
                                             DotBuf dot, double *sc) {
  const long long np = (long long)N1 * N2;
  const int s = blockIdx.y;
  const float b = (float)beta[s];
  const float bd = (float)(beta[s] / sqrt(2.0));
  const float2 *xs = x + (long long)s * np;
  long long q0, q1;
  share(np, q0, q1);
  double acc = 0.0;
  for (long long q = q0 + threadIdx.x; q < q1; q += 256) {
    const int i2 = (int)((unsigned)q / (unsigned)N1), i1 = (int)q - i2 * N1;
    const float2 v = xs[q];
    float ar = 0.f, ai = 0.f;
    const int d1[4] = {1, 0, 1, -1}, d2[4] = {0, 1, 1, 1};
#pragma unroll
    for (int m = 0; m < 4; m++) {
      const float w = m < 2 ? b : bd;
      // pair (n, n - d)
      int j1 = i1 - d1[m], j2 = i2 - d2[m];
      if (j1 >= 0 && j1 < N1 && j2 >= 0) {
        const float2 u = xs[(long long)j2 * N1 + j1];
        ar += w * (v.x - u.x);
        ai += w * (v.y - u.y);
      }
      // pair (n + d, n)
      j1 = i1 + d1[m];
      j2 = i2 + d2[m];
      if (j1 >= 0 && j1 < N1 && j2 < N2) {
        const float2 u = xs[(long long)j2 * N1 + j1];
        ar += w * (v.x - u.x);
        ai += w * (v.y - u.y);
      }
    }
    out[(long long)s * np + q] = make_float2(ar, ai);
    if (DOT) acc += (double)v.x * ar + (double)v.y * ai;
  }
  if (DOT) finish_dot(dot, acc, [&](double v) { sc[s * SC_N + SC_DENR] = v; });
}

// out[s * stride] = Re sum conj(a) b over [off[s], off[s+1]) in FP64 (weights
// per element group of C when W is given).  WHAT: 0 only that; 1 the gradient
// product; 2 the data curvature, with the step (ddir' ngrad) / (data curvature
// + ddir' R ddir).
template <int WHAT>
__global__ void __launch_bounds__(256) k_segdot(const float2 *__restrict__ a,
                                                const float2 *__restrict__ b,
                                                const long long *__restrict__ off,
                                                const float *__restrict__ W, int C,
                                                double *__restrict__ out, int stride, DotBuf dot,
                                                double *sc, int first) {
  const int s = blockIdx.y;
  const long long e0 = off[s];
  long long q0, q1;
  share(off[s + 1] - e0, q0, q1);
  double acc = 0.0;
  for (long long q = q0 + threadIdx.x; q < q1; q += 256) {
    const float2 u = a[e0 + q], v = b[e0 + q];
    double t = (double)u.x * v.x + (double)u.y * v.y;
    if (W) t *= (double)W[(e0 + q) / C];
    acc += t;
  }
  finish_dot(dot, acc, [&](double v) {
    double *c = sc + s * SC_N;
    if (WHAT == 0) out[s * stride] = v;
    if (WHAT == 1) new_product(c, v, first);
    if (WHAT == 2) {
      const double den = v + c[SC_DENR];
      c[SC_DEN] = v;
      c[SC_STEP] = den == 0.0 ? 0.0 : c[SC_NUM] / den;
    }
  });
}

// The Gram form's negative gradient out = b - u - v.  DOT: with <out, out> as
// the iteration's new gradient product.
template <bool DOT>
__global__ void __launch_bounds__(256) k_sub2(const float2 *__restrict__ b,
                                              const float2 *__restrict__ u,
                                              const float2 *__restrict__ v,
                                              float2 *__restrict__ out, long long np, DotBuf dot,
                                              double *sc, int first) {
  const long long base = (long long)blockIdx.y * np;
  long long q0, q1;
  share(np, q0, q1);
  double acc = 0.0;
  for (long long q = base + q0 + threadIdx.x; q < base + q1; q += 256) {
    const float2 g = make_float2(b[q].x - u[q].x - v[q].x, b[q].y - u[q].y - v[q].y);
    out[q] = g;
    if (DOT) acc += (double)g.x * g.x + (double)g.y * g.y;
  }
  if (DOT)
    finish_dot(dot, acc, [&](double w) { new_product(sc + blockIdx.y * SC_N, w, first); });
}

// Fletcher-Reeves: ddir = pregrad + gamma ddir, with <ddir, ngrad>
__global__ void __launch_bounds__(256) k_dir(const float2 *__restrict__ pgrad,
                                             const float2 *__restrict__ ngrad,
                                             float2 *__restrict__ ddir, long long np, DotBuf dot,
                                             double *sc, int first) {
  double *c = sc + blockIdx.y * SC_N;
  const long long base = (long long)blockIdx.y * np;
  const float gf = (float)c[SC_GAMMA];
  long long q0, q1;
  share(np, q0, q1);
  double acc = 0.0;
  for (long long q = base + q0 + threadIdx.x; q < base + q1; q += 256) {
    float2 d = pgrad[q];
    const float2 g = ngrad[q];
    if (!first) {
      const float2 o = ddir[q];
      d = make_float2(d.x + gf * o.x, d.y + gf * o.y);
    }
    ddir[q] = d;
    acc += (double)d.x * g.x + (double)d.y * g.y;
  }
  finish_dot(dot, acc, [&](double v) { c[SC_NUM] = v; });
}

__global__ void k_scal_step(double *sc, int S) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= S) return;
  double *c = sc + s * SC_N;
  const double den = c[SC_DEN] + c[SC_DENR];
  c[SC_STEP] = den == 0.0 ? 0.0 : c[SC_NUM] / den;
}

__device__ __forceinline__ float2 axpy2(float st, float2 d, float2 v) {
  return make_float2(fmaf(st, d.x, v.x), fmaf(st, d.y, v.y));
}

// v += step d (and v2 += step2 d2, v3 likewise, when given) over the problems'
// image vectors
__global__ void __launch_bounds__(256) k_step_image(float2 *__restrict__ v,
                                                    const float2 *__restrict__ d,
                                                    float2 *__restrict__ v2,
                                                    const float2 *__restrict__ d2,
                                                    float2 *__restrict__ v3,
                                                    const float2 *__restrict__ d3,
                                                    const double *__restrict__ sc, long long np) {
  const float st = (float)sc[blockIdx.y * SC_N + SC_STEP];
  const long long base = (long long)blockIdx.y * np;
  long long q0, q1;
  share(np, q0, q1);
  for (long long q = base + q0 + threadIdx.x; q < base + q1; q += 256) {
    v[q] = axpy2(st, d[q], v[q]);
    if (v2) v2[q] = axpy2(st, d2[q], v2[q]);
    if (v3) v3[q] = axpy2(st, d3[q], v3[q]);
  }
}

// Ax += step Adir over the problems' data, and the next residual r = W (y - Ax)
__global__ void __launch_bounds__(256) k_step_data(float2 *__restrict__ Ax,
                                                   const float2 *__restrict__ Adir,
                                                   const float2 *__restrict__ y,
                                                   const float *__restrict__ W,
                                                   float2 *__restrict__ r,
                                                   const long long *__restrict__ off, int C,
                                                   const double *__restrict__ sc) {
  const int s = blockIdx.y;
  const float st = (float)sc[s * SC_N + SC_STEP];
  const long long e0 = off[s];
  long long q0, q1;
  share(off[s + 1] - e0, q0, q1);
  for (long long q = e0 + q0 + threadIdx.x; q < e0 + q1; q += 256) {
    const float2 a = axpy2(st, Adir[q], Ax[q]), b = y[q];
    const float w = W ? W[q / C] : 1.f;
    Ax[q] = a;
    r[q] = make_float2(w * (b.x - a.x), w * (b.y - a.y));
  }
}

// per-slice ||x - xref||^2 (FP64), xref = 0 when not given
__global__ void __launch_bounds__(256) k_errnorm(const float2 *__restrict__ x,
                                                 const float2 *__restrict__ xr, long long np,
                                                 double *__restrict__ out, DotBuf dot) {
  const long long base = (long long)blockIdx.y * np;
  long long q0, q1;
  share(np, q0, q1);
  double acc = 0.0;
  for (long long q = base + q0 + threadIdx.x; q < base + q1; q += 256) {
    const float2 u = x[q], v = xr ? xr[q] : make_float2(0.f, 0.f);
    const double dx = (double)u.x - v.x, dy = (double)u.y - v.y;
    acc += dx * dx + dy * dy;
  }
  finish_dot(dot, acc, [&](double w) { out[blockIdx.y] = w; });
}

// Blocks per problem of a kernel over n elements a problem: about kBlocks in all
// (16 blocks of 256 threads per SM: two waves), at least 512 elements each.
constexpr int kBlocks = 148 * 16;
unsigned problem_blocks(long long n, int S) {
  const long long p = std::min((kBlocks + S - 1ll) / S, (n + 511) / 512);
  return (unsigned)std::max(1ll, p);
}

}  // namespace

namespace mirt {
cudaError_t launch_coil_combine(const float2 *z, const float2 *sens, float2 *out, long long np, int C,
                                int S, cudaStream_t st) {
  k_combine<false><<<dim3(problem_blocks(np * 8, S), S), 256, 0, st>>>(z, sens, nullptr, out, np, C,
                                                                      DotBuf{}, nullptr, 0);
  return cudaGetLastError();
}
}  // namespace mirt

struct mirt_sense {
  mirt_nufft *G = nullptr;
  int S = 0, C = 0, N1 = 0, N2 = 0;
  long long np = 0, M = 0;
  DMem sens, beta, z, ioff, soff;
  // sens .* sn where the NUFFT's FFT runs as fused passes: A's first pass reads it
  // times the image, so that the coil images are never written
  DMem sens_sn;
  std::vector<double> beta_host;
  mirt_toeplitz *T = nullptr;  // Gram operator and preconditioner (mirt_sense_toeplitz)
  ~mirt_sense() { delete T; }
};

namespace {

// the inner products' buffers of one call
struct DotMem {
  DMem part, count;
  DotBuf buf{};
  cudaError_t alloc(int S, cudaStream_t st) {
    cudaError_t e = part.alloc((size_t)S * ((kBlocks + S - 1) / S) * sizeof(double));
    if (!e) e = count.alloc(S * sizeof(int));
    if (!e) e = cudaMemsetAsync(count.p, 0, S * sizeof(int), st);
    buf = DotBuf{part.as<double>(), count.as<int>()};
    return e;
  }
};

int sense_A(mirt_sense *op, const float2 *x, float2 *y, cudaStream_t st) {
  mirt_nufft *G = op->G;
  if (op->sens_sn.p) {
    SCK(fft_nufft_forward(G->nf, op->sens_sn.as<float2>(), G->grid.as<float2>(), 0, op->S, st, x));
    return mirt_interp_plan_forward(G->ip, G->grid.p, y, st);
  }
  const long long n = (long long)op->S * op->np * op->C;
  k_expand<<<nblocks(n), 256, 0, st>>>(x, op->sens.as<float2>(), op->z.as<float2>(), n, op->C);
  SCK(cudaGetLastError());
  return mirt_nufft_forward(op->G, op->z.p, y, st);
}

// x = A'y (- sub); with dot: and <x, x> as the new gradient product
int sense_At(mirt_sense *op, const float2 *y, float2 *x, const float2 *sub, cudaStream_t st,
             DotBuf *dot = nullptr, double *sc = nullptr, int first = 0) {
  int rc = mirt_nufft_adjoint(op->G, y, op->z.p, st);
  if (rc) return rc;
  const dim3 grid(problem_blocks(op->np * 8, op->S), op->S);
  if (dot)
    k_combine<true><<<grid, 256, 0, st>>>(op->z.as<float2>(), op->sens.as<float2>(), sub, x, op->np,
                                          op->C, *dot, sc, first);
  else
    k_combine<false><<<grid, 256, 0, st>>>(op->z.as<float2>(), op->sens.as<float2>(), sub, x,
                                           op->np, op->C, DotBuf{}, nullptr, 0);
  SCK(cudaGetLastError());
  return MIRT_OK;
}

// rx = R x; with dot: and <x, rx> as the penalty's share of the curvature
int sense_R(mirt_sense *op, const float2 *x, float2 *rx, cudaStream_t st, DotBuf *dot = nullptr,
            double *sc = nullptr) {
  const dim3 grid(problem_blocks(op->np, op->S), op->S);
  if (dot)
    k_reg<true><<<grid, 256, 0, st>>>(x, rx, op->N1, op->N2, op->beta.as<double>(), *dot, sc);
  else
    k_reg<false><<<grid, 256, 0, st>>>(x, rx, op->N1, op->N2, op->beta.as<double>(), DotBuf{},
                                       nullptr);
  SCK(cudaGetLastError());
  return MIRT_OK;
}

}  // namespace

extern "C" {

int mirt_sense_create(mirt_sense **out, mirt_nufft *G, const void *sens, const double *beta,
                      void *stream) {
  if (!out || !G || !sens || !beta) return api_fail(MIRT_ERR_ARG, "NULL argument");
  *out = nullptr;
  if (G->gg.D != 2) return api_fail(MIRT_ERR_ARG, "CG-SENSE is provided for 2D plans");
  if (G->nslice > 1024) return api_fail(MIRT_ERR_ARG, "at most 1024 problems per plan");
  cudaStream_t st = as_stream(stream);
  auto *op = new mirt_sense();
  auto bail = [&](int code) {
    delete op;
    return code;
  };
  op->G = G;
  op->S = G->nslice;
  op->C = G->C;
  op->N1 = G->gg.N[0];
  op->N2 = G->gg.N[1];
  op->np = G->gg.npix;
  op->M = G->Mtot;
  const size_t nimg = (size_t)op->S * op->np;
  if (op->sens.alloc(nimg * op->C * sizeof(float2)) || op->beta.alloc(op->S * sizeof(double)) ||
      op->z.alloc(nimg * op->C * sizeof(float2)) ||
      op->ioff.alloc((op->S + 1) * sizeof(long long)) ||
      op->soff.alloc((op->S + 1) * sizeof(long long)))
    return bail(api_fail(MIRT_ERR_ALLOC, "CG-SENSE buffers"));
  std::vector<long long> io(op->S + 1), so(op->S + 1);
  for (int s = 0; s <= op->S; s++) {
    io[s] = (long long)s * op->np;
    so[s] = G->ip->moff_host[s] * op->C;
  }
  cudaError_t e = cudaMemcpyAsync(op->sens.p, sens, nimg * op->C * sizeof(float2),
                                  cudaMemcpyDeviceToDevice, st);
  op->beta_host.assign(beta, beta + op->S);
  if (!e) e = cudaMemcpyAsync(op->beta.p, beta, op->S * sizeof(double), cudaMemcpyHostToDevice, st);
  if (!e) e = cudaMemcpyAsync(op->ioff.p, io.data(), io.size() * sizeof(long long),
                              cudaMemcpyHostToDevice, st);
  if (!e) e = cudaMemcpyAsync(op->soff.p, so.data(), so.size() * sizeof(long long),
                              cudaMemcpyHostToDevice, st);
  if (!e && G->own_fft && op->S > 0 && op->C > 0) {
    const long long n = (long long)nimg * op->C;
    // (no room for a second set of maps: A expands the coil images)
    if (op->sens_sn.alloc(n * sizeof(float2)) == cudaSuccess) {
      k_maps_sn<<<nblocks(n), 256, 0, st>>>(op->sens.as<float2>(), G->sn.as<float2>(),
                                            op->sens_sn.as<float2>(), n, op->np, op->C);
      e = cudaGetLastError();
    }
  }
  if (!e) e = cudaStreamSynchronize(st);
  if (e) return bail(api_fail(MIRT_ERR_CUDA, cudaGetErrorString(e)));
  *out = op;
  return MIRT_OK;
}

int mirt_sense_forward(mirt_sense *op, const void *x, void *y, void *stream) {
  if (!op || !x || !y) return api_fail(MIRT_ERR_ARG, "NULL argument");
  return sense_A(op, static_cast<const float2 *>(x), static_cast<float2 *>(y), as_stream(stream));
}

int mirt_sense_adjoint(mirt_sense *op, const void *y, void *x, void *stream) {
  if (!op || !x || !y) return api_fail(MIRT_ERR_ARG, "NULL argument");
  return sense_At(op, static_cast<const float2 *>(y), static_cast<float2 *>(x), nullptr,
                  as_stream(stream));
}

int mirt_sense_reg(mirt_sense *op, const void *x, void *rx, void *stream) {
  if (!op || !x || !rx) return api_fail(MIRT_ERR_ARG, "NULL argument");
  return sense_R(op, static_cast<const float2 *>(x), static_cast<float2 *>(rx), as_stream(stream));
}

int mirt_sense_pcg(mirt_sense *op, void *x_, const void *y_, const float *W, int32_t niter,
                   int32_t flags, const void *xref_, double *nrmse, float *ms, void *stream) try {
  if (!op || !x_ || !y_) return api_fail(MIRT_ERR_ARG, "NULL argument");
  if (niter < 0) return api_fail(MIRT_ERR_ARG, "niter must be >= 0");
  const bool precon = flags & MIRT_PCG_CIRCULANT, gram = flags & MIRT_PCG_TOEPLITZ;
  if ((precon || gram) && !op->T)
    return api_fail(MIRT_ERR_ARG, "attach the Toeplitz operator first (mirt_sense_toeplitz)");
  if (gram && W) return api_fail(MIRT_ERR_ARG, "the Toeplitz Gram form takes no data weights");
  cudaStream_t st = as_stream(stream);
  const int S = op->S, C = op->C;
  const long long ni = (long long)S * op->np, ns = op->M * C;
  float2 *x = static_cast<float2 *>(x_);
  const float2 *y = static_cast<const float2 *>(y_);
  const float2 *xref = static_cast<const float2 *>(xref_);
  // data-side vectors: Ax, Adir, residual (form 1) or A'y, Gx, Gdir (Gram form)
  DMem Ax, Adir, r, Rx, Rdir, ngrad, pgrad, ddir, sc, err, refn;
  if (gram) {
    SCK(Ax.alloc(ni * sizeof(float2)));    // G x
    SCK(Adir.alloc(ni * sizeof(float2)));  // G ddir
    SCK(r.alloc(ni * sizeof(float2)));     // b = A'y
  } else {
    SCK(Ax.alloc(std::max<long long>(ns, 1) * sizeof(float2)));
    SCK(Adir.alloc(std::max<long long>(ns, 1) * sizeof(float2)));
    SCK(r.alloc(std::max<long long>(ns, 1) * sizeof(float2)));
  }
  SCK(Rx.alloc(ni * sizeof(float2)));
  SCK(Rdir.alloc(ni * sizeof(float2)));
  SCK(ngrad.alloc(ni * sizeof(float2)));
  if (precon) SCK(pgrad.alloc(ni * sizeof(float2)));
  SCK(ddir.alloc(ni * sizeof(float2)));
  SCK(sc.alloc(S * SC_N * sizeof(double)));
  SCK(cudaMemsetAsync(sc.p, 0, S * SC_N * sizeof(double), st));
  DotMem dm;
  SCK(dm.alloc(S, st));
  const dim3 gi(problem_blocks(op->np, S), S), gs(problem_blocks(std::max<long long>(ns / S, 1), S), S);
  const bool track = xref && nrmse;
  if (track) {
    SCK(err.alloc((size_t)(niter + 1) * S * sizeof(double)));
    SCK(refn.alloc(S * sizeof(double)));
    k_errnorm<<<gi, 256, 0, st>>>(xref, nullptr, op->np, refn.as<double>(), dm.buf);
    k_errnorm<<<gi, 256, 0, st>>>(x, xref, op->np, err.as<double>(), dm.buf);
    SCK(cudaGetLastError());
  }
  std::vector<cudaEvent_t> ev;
  if (ms) {
    ev.resize(niter + 1);
    for (auto &e : ev) SCK(cudaEventCreate(&e));
    SCK(cudaEventRecord(ev[0], st));
  }
  auto cleanup = [&]() {
    for (auto &e : ev) cudaEventDestroy(e);
  };
  auto gram_apply = [&](const float2 *v, float2 *out) {
    return toep_gram_sense(op->T, v, op->sens.as<float2>(), out, st);
  };
  // data term and penalty of the initial estimate
  int rc = MIRT_OK;
  if (gram) {
    rc = sense_At(op, y, r.as<float2>(), nullptr, st);  // b = A'y
    if (!rc) rc = gram_apply(x, Ax.as<float2>());
  } else {
    rc = sense_A(op, x, Ax.as<float2>(), st);
    if (!rc) k_resid<<<nblocks(ns), 256, 0, st>>>(y, Ax.as<float2>(), W, r.as<float2>(), ns, C);
  }
  if (!rc) rc = sense_R(op, x, Rx.as<float2>(), st);
  const long long *ioff = op->ioff.as<long long>(), *soff = op->soff.as<long long>();
  double *scp = sc.as<double>();
  for (int it = 1; it <= niter && !rc; it++) {
    const int first = it == 1;
    // negative gradient and, without a preconditioner, its product
    if (gram) {
      if (precon)
        k_sub2<false><<<gi, 256, 0, st>>>(r.as<float2>(), Ax.as<float2>(), Rx.as<float2>(),
                                          ngrad.as<float2>(), op->np, dm.buf, scp, first);
      else
        k_sub2<true><<<gi, 256, 0, st>>>(r.as<float2>(), Ax.as<float2>(), Rx.as<float2>(),
                                         ngrad.as<float2>(), op->np, dm.buf, scp, first);
    } else {
      rc = sense_At(op, r.as<float2>(), ngrad.as<float2>(), Rx.as<float2>(), st,
                    precon ? nullptr : &dm.buf, scp, first);
      if (rc) break;
    }
    // preconditioned gradient and the Fletcher-Reeves direction
    const float2 *pg = ngrad.as<float2>();
    if (precon) {
      rc = toep_precon_apply(op->T, ngrad.as<float2>(), pgrad.as<float2>(), st);
      if (rc) break;
      pg = pgrad.as<float2>();
      k_segdot<1><<<gi, 256, 0, st>>>(ngrad.as<float2>(), pg, ioff, nullptr, 1, nullptr, 0, dm.buf,
                                      scp, first);
    }
    k_dir<<<gi, 256, 0, st>>>(pg, ngrad.as<float2>(), ddir.as<float2>(), op->np, dm.buf, scp, first);
    // step: (ddir' ngrad) / (data curvature + ddir' R ddir)
    rc = sense_R(op, ddir.as<float2>(), Rdir.as<float2>(), st, &dm.buf, scp);
    if (rc) break;
    if (gram) {
      rc = gram_apply(ddir.as<float2>(), Adir.as<float2>());
    } else {
      rc = sense_A(op, ddir.as<float2>(), Adir.as<float2>(), st);
    }
    if (rc) break;
    if (gram) {
      k_segdot<2><<<gi, 256, 0, st>>>(ddir.as<float2>(), Adir.as<float2>(), ioff, nullptr, 1,
                                      nullptr, 0, dm.buf, scp, first);
      k_step_image<<<gi, 256, 0, st>>>(x, ddir.as<float2>(), Rx.as<float2>(), Rdir.as<float2>(),
                                       Ax.as<float2>(), Adir.as<float2>(), scp, op->np);
    } else {
      k_segdot<2><<<gs, 256, 0, st>>>(Adir.as<float2>(), Adir.as<float2>(), soff, W, C, nullptr, 0,
                                      dm.buf, scp, first);
      k_step_image<<<gi, 256, 0, st>>>(x, ddir.as<float2>(), Rx.as<float2>(), Rdir.as<float2>(),
                                       nullptr, nullptr, scp, op->np);
      if (it < niter)
        k_step_data<<<gs, 256, 0, st>>>(Ax.as<float2>(), Adir.as<float2>(), y, W, r.as<float2>(),
                                        soff, C, scp);
    }
    if (track)
      k_errnorm<<<gi, 256, 0, st>>>(x, xref, op->np, err.as<double>() + (size_t)it * S, dm.buf);
    cudaError_t e = cudaGetLastError();
    if (e) rc = api_fail(MIRT_ERR_CUDA, std::string("CG iteration: ") + cudaGetErrorString(e));
    if (ms) cudaEventRecord(ev[it], st);
  }
  if (rc) {
    cleanup();
    return rc;
  }
  cudaError_t e = cudaStreamSynchronize(st);
  if (e) {
    cleanup();
    return api_fail(MIRT_ERR_CUDA, cudaGetErrorString(e));
  }
  if (ms)
    for (int it = 1; it <= niter; it++) cudaEventElapsedTime(&ms[it - 1], ev[0], ev[it]);
  cleanup();
  if (track) {
    std::vector<double> h((size_t)(niter + 1) * S), rn(S);
    SCK(cudaMemcpy(h.data(), err.p, h.size() * sizeof(double), cudaMemcpyDeviceToHost));
    SCK(cudaMemcpy(rn.data(), refn.p, S * sizeof(double), cudaMemcpyDeviceToHost));
    for (size_t i = 0; i < h.size(); i++) {
      const double d = rn[i % S];
      nrmse[i] = d > 0 ? std::sqrt(h[i] / d) : std::sqrt(h[i]);
    }
  }
  return MIRT_OK;
} catch (const std::bad_alloc &) {
  return api_fail(MIRT_ERR_ALLOC, "out of host memory");
}

int mirt_sense_cg(mirt_sense *op, void *x, const void *y, const float *W, int32_t niter,
                  const void *xref, double *nrmse, float *ms, void *stream) {
  return mirt_sense_pcg(op, x, y, W, niter, 0, xref, nrmse, ms, stream);
}

namespace {
__global__ void k_square(const double *__restrict__ w, double *__restrict__ w2, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    w2[i] = w[i] * w[i];
}
}  // namespace

int mirt_sense_precon_dcf(mirt_sense *op, const double *om, const double *w, double blend,
                          void *stream) {
  if (!op || !om || !w) return api_fail(MIRT_ERR_ARG, "NULL argument");
  if (!op->T) return api_fail(MIRT_ERR_ARG, "mirt_sense_toeplitz must run first");
  if (!(blend >= 0.0 && blend <= 1.0)) return api_fail(MIRT_ERR_ARG, "blend must be in [0, 1]");
  cudaStream_t st = as_stream(stream);
  mirt_interp_plan *P = op->G->ip;
  const int Nd[2] = {op->N1, op->N2}, Kd[2] = {P->a.g.K[0], P->a.g.K[1]};
  const int Jd[2] = {P->a.g.J[0], P->a.g.J[1]}, Ld[2] = {P->a.g.L[0], P->a.g.L[1]};
  DMem w2;
  cudaError_t e = w2.alloc(std::max<long long>(op->M, 1) * sizeof(double));
  if (e) return api_fail(MIRT_ERR_ALLOC, "DCF preconditioner weights");
  if (op->M > 0) {
    long long nb = (op->M + 255) / 256;
    if (nb > 148 * 16) nb = 148 * 16;
    k_square<<<(unsigned)nb, 256, 0, st>>>(w, w2.as<double>(), op->M);
    e = cudaGetLastError();
    if (e) return api_fail(MIRT_ERR_CUDA, cudaGetErrorString(e));
  }
  mirt_toeplitz *Tw = nullptr;
  int rc = toep_create(&Tw, om, op->M, P->moff_host.data(), op->S, Nd, Kd, Jd, Ld,
                       w2.as<double>(), 1, st);
  if (rc) return rc;
  rc = toep_precon_dcf(op->T, Tw, blend, st);
  delete Tw;
  return rc;
}

int mirt_sense_toeplitz(mirt_sense *op, const double *om, void *stream) {
  if (!op || !om) return api_fail(MIRT_ERR_ARG, "NULL argument");
  cudaStream_t st = as_stream(stream);
  mirt_interp_plan *P = op->G->ip;
  const int Nd[2] = {op->N1, op->N2}, Kd[2] = {P->a.g.K[0], P->a.g.K[1]};
  const int Jd[2] = {P->a.g.J[0], P->a.g.J[1]}, Ld[2] = {P->a.g.L[0], P->a.g.L[1]};
  mirt_toeplitz *T = nullptr;
  int rc = toep_create(&T, om, op->M, P->moff_host.data(), op->S, Nd, Kd, Jd, Ld, nullptr, op->C,
                       st);
  if (rc) return rc;
  // mean coil power per problem, for the preconditioner
  std::vector<long long> off(op->S + 1);
  for (int s = 0; s <= op->S; s++) off[s] = (long long)s * op->np * op->C;
  DMem doff, pw;
  cudaError_t e = doff.alloc((op->S + 1) * sizeof(long long));
  if (!e) e = pw.alloc(op->S * sizeof(double));
  if (!e) e = cudaMemcpyAsync(doff.p, off.data(), off.size() * sizeof(long long),
                              cudaMemcpyHostToDevice, st);
  if (e) {
    delete T;
    return api_fail(MIRT_ERR_CUDA, cudaGetErrorString(e));
  }
  DotMem dm;
  e = dm.alloc(op->S, st);
  if (e) {
    delete T;
    return api_fail(MIRT_ERR_CUDA, cudaGetErrorString(e));
  }
  k_segdot<0><<<dim3(problem_blocks(op->np * op->C, op->S), op->S), 256, 0, st>>>(
      op->sens.as<float2>(), op->sens.as<float2>(), doff.as<long long>(), nullptr, 1,
      pw.as<double>(), 1, dm.buf, nullptr, 0);
  std::vector<double> lam(op->S);
  e = cudaMemcpyAsync(lam.data(), pw.p, op->S * sizeof(double), cudaMemcpyDeviceToHost, st);
  if (!e) e = cudaStreamSynchronize(st);
  if (e) {
    delete T;
    return api_fail(MIRT_ERR_CUDA, cudaGetErrorString(e));
  }
  for (auto &v : lam) v /= (double)op->np;
  rc = toep_precon_build(T, lam.data(), op->beta_host.data(), st);
  if (rc) {
    delete T;
    return rc;
  }
  delete op->T;
  op->T = T;
  return MIRT_OK;
}

int mirt_sense_warm_start(mirt_sense *op, void *x_, const void *y_, const float *W,
                          void *stream) {
  if (!op || !x_ || !y_) return api_fail(MIRT_ERR_ARG, "NULL argument");
  cudaStream_t st = as_stream(stream);
  const int S = op->S, C = op->C;
  const long long ni = (long long)S * op->np, ns = op->M * C;
  float2 *x = static_cast<float2 *>(x_);
  const float2 *y = static_cast<const float2 *>(y_);
  DMem zero, r, Ax, sc;
  SCK(zero.alloc(std::max<long long>(ns, 1) * sizeof(float2)));
  SCK(r.alloc(std::max<long long>(ns, 1) * sizeof(float2)));
  SCK(Ax.alloc(std::max<long long>(ns, 1) * sizeof(float2)));
  SCK(sc.alloc(S * SC_N * sizeof(double)));
  SCK(cudaMemsetAsync(zero.p, 0, std::max<long long>(ns, 1) * sizeof(float2), st));
  // x = A'(W y): the density-compensated "conjugate phase" image
  k_resid<<<nblocks(ns), 256, 0, st>>>(y, zero.as<float2>(), W, r.as<float2>(), ns, C);
  int rc = sense_At(op, r.as<float2>(), x, nullptr, st);
  if (!rc) rc = sense_A(op, x, Ax.as<float2>(), st);
  if (rc) return rc;
  // per problem: x *= Re<Ax, y> / ||Ax||^2 (the least-squares scale)
  double *scp = sc.as<double>();
  DotMem dm;
  SCK(dm.alloc(S, st));
  SCK(cudaMemsetAsync(sc.p, 0, S * SC_N * sizeof(double), st));
  const dim3 gs(problem_blocks(std::max<long long>(ns / S, 1), S), S);
  k_segdot<0><<<gs, 256, 0, st>>>(Ax.as<float2>(), y, op->soff.as<long long>(), nullptr, 1,
                                  scp + SC_NUM, SC_N, dm.buf, scp, 0);
  k_segdot<0><<<gs, 256, 0, st>>>(Ax.as<float2>(), Ax.as<float2>(), op->soff.as<long long>(),
                                  nullptr, 1, scp + SC_DEN, SC_N, dm.buf, scp, 0);
  k_scal_step<<<1, 64 * ((S + 63) / 64), 0, st>>>(scp, S);
  // x = 0 + step x
  DMem xc;
  SCK(xc.alloc(ni * sizeof(float2)));
  SCK(cudaMemcpyAsync(xc.p, x, ni * sizeof(float2), cudaMemcpyDeviceToDevice, st));
  SCK(cudaMemsetAsync(x, 0, ni * sizeof(float2), st));
  k_step_image<<<dim3(problem_blocks(op->np, S), S), 256, 0, st>>>(
      x, xc.as<float2>(), nullptr, nullptr, nullptr, nullptr, scp, op->np);
  SCK(cudaGetLastError());
  SCK(cudaStreamSynchronize(st));
  return MIRT_OK;
}

int mirt_sense_destroy(mirt_sense *op) {
  if (op) {
    cudaDeviceSynchronize();
    delete op;
  }
  return MIRT_OK;
}

}  // extern "C"
