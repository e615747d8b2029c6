// dcf.cu -- density compensation weights on the project's NUFFT.
//
// Pipe & Menon iteration (mri/ir_mri_density_comp.m:203-281): starting from
// w = 1, repeat  goal = real(P P' w),  w = w ./ goal  until
// max |goal - 1| <= thresh, with at most niter + 1 updates (the reference
// tests `iter > niter` after the update), then scale w so that the point
// spread function G' w sums to prod(N ./ fov).  P is the table interpolator
// with the NUFFT's phase shift (nufft/nufft_table_interp.m:75-78 and
// nufft/nufft_table_adj.m:47-50), G the full NUFFT.  The one-step weights
// w = 1 ./ real(P (P' 1)) of ir_mri_dcf_jackson (:160-180) are here too.
//
// Precision: the spread / gather run in FP32 (the plan's kernels); the weights,
// the ratio update, the residual and the scaling sums are FP64.  A batch of
// slices (trajectories of uneven length in one plan) iterates together in one
// launch sequence; each slice stops on its own residual and is then frozen on
// the device, so no host round trip is needed per iteration.
#include "../../include/mirt_b200.h"

#include <cmath>
#include <string>
#include <vector>

#include "runtime.cuh"

using namespace mirt;

namespace {

#define DCK(call)                                                                     \
  do {                                                                                \
    cudaError_t e_ = (call);                                                          \
    if (e_ != cudaSuccess)                                                            \
      return api_fail(e_ == cudaErrorMemoryAllocation ? MIRT_ERR_ALLOC : MIRT_ERR_CUDA, \
                      std::string(#call) + ": " + cudaGetErrorString(e_));            \
  } while (0)

constexpr int kUpdThreads = 256, kUpdPer = 2;  // update: samples a thread, block-strided

__global__ void fill_ones_kernel(double *w, long long M) {
  for (long long m = blockIdx.x * (long long)blockDim.x + threadIdx.x; m < M;
       m += (long long)gridDim.x * blockDim.x)
    w[m] = 1.0;
}

// FP64 weights -> complex64 samples for the spread
__global__ void w_to_c64_kernel(const double *__restrict__ w, long long M, float2 *__restrict__ f) {
  for (long long m = blockIdx.x * (long long)blockDim.x + threadIdx.x; m < M;
       m += (long long)gridDim.x * blockDim.x)
    f[m] = make_float2((float)w[m], 0.f);
}

// w <- w / real(g) on the active slices, and the next pass's samples f = w; residual
// max |goal - 1| per slice by an atomic max on the bit pattern (order-free for
// non-negative doubles): one per block where its samples lie in one slice, else one
// per warp and slice.  The last block to finish records the residual and iteration
// of each active slice, freezes the slices that met the threshold and counts the
// ones still active.  Bound by its loads and stores (36 bytes a sample): 29 us with
// each thread on its own run of samples and 5.5 us more for the cast and the
// bookkeeping, 8.3 us so (6 slices, 491,520 samples).
struct PipeState {
  int *active;
  unsigned long long *resid_bits;
  double *resid;
  int *iters, *bad, *nactive;
  unsigned *done;
};

__global__ void __launch_bounds__(kUpdThreads)
    pipe_update_kernel(const float2 *__restrict__ g, const int *__restrict__ slice_of, long long M,
                       double *__restrict__ w, float2 *__restrict__ f, PipeState P, int nslice,
                       int it, double thresh) {
  __shared__ unsigned long long smax;
  __shared__ int last, cnt;
  const long long m0 = (long long)blockIdx.x * (kUpdThreads * kUpdPer);
  const long long m1 = min(M, m0 + kUpdThreads * kUpdPer) - 1;
  const int s0 = slice_of && m0 <= m1 ? slice_of[m0] : 0;
  const bool one = !slice_of || m0 > m1 || slice_of[m1] == s0;
  const bool act0 = m0 <= m1 && P.active[s0];
  if (threadIdx.x == 0) smax = 0ull;
  __syncthreads();
  // all loads of the thread's samples before the first store
  int sl[kUpdPer];
  bool act[kUpdPer];
  double goal[kUpdPer], wv[kUpdPer];
#pragma unroll
  for (int k = 0; k < kUpdPer; k++) {
    const long long m = m0 + k * kUpdThreads + threadIdx.x;
    const bool in = m <= m1;
    sl[k] = in && !one ? slice_of[m] : s0;
    goal[k] = in ? (double)g[m].x : 1.0;
    wv[k] = in ? w[m] : 0.0;
    act[k] = in && (one ? act0 : P.active[sl[k]] != 0);
  }
  unsigned long long rmax = 0ull;
  bool neg = false;
#pragma unroll
  for (int k = 0; k < kUpdPer; k++) {
    const long long m = m0 + k * kUpdThreads + threadIdx.x;
    if (!one) rmax = 0ull;
    if (act[k]) {
      if (goal[k] > 0.0) {
        const double v = wv[k] / goal[k];
        w[m] = v;
        f[m] = make_float2((float)v, 0.f);
        const double r = fabs(goal[k] - 1.0);
        rmax = max(rmax, (unsigned long long)__double_as_longlong(r));
      } else {
        neg = true;
      }
    }
    if (!one) {
      const unsigned same = __match_any_sync(0xffffffffu, act[k] ? sl[k] : -1);
      for (int h = 16; h > 0; h >>= 1) {
        const unsigned long long o = __shfl_xor_sync(0xffffffffu, rmax, h);
        if (same == 0xffffffffu) rmax = max(rmax, o);
      }
      if (act[k] && (same != 0xffffffffu || (threadIdx.x & 31) == 0))
        atomicMax(P.resid_bits + sl[k], rmax);
    }
  }
  if (__syncthreads_or(neg) && threadIdx.x == 0) atomicOr(P.bad, 1);
  if (one) {
    for (int h = 16; h > 0; h >>= 1)
      rmax = max(rmax, __shfl_xor_sync(0xffffffffu, rmax, h));
    if ((threadIdx.x & 31) == 0) atomicMax(&smax, rmax);
    __syncthreads();
    if (threadIdx.x == 0 && smax) atomicMax(P.resid_bits + s0, smax);
  }
  if (!one || threadIdx.x == 0) __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    cnt = 0;
    last = atomicAdd(P.done, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (int s = threadIdx.x; s < nslice; s += blockDim.x) {
    if (P.active[s]) {
      const double r = __longlong_as_double((long long)__ldcg(P.resid_bits + s));
      P.resid[s] = r;
      P.iters[s] = it;
      if (r <= thresh)
        P.active[s] = 0;
      else
        atomicAdd(&cnt, 1);
    }
    P.resid_bits[s] = 0ull;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    *P.nactive = cnt;
    *P.done = 0u;
  }
}

// Per-slice FP64 sum of real(x) over npix pixels, fixed summation order.
__global__ void psf_sum_kernel(const float2 *__restrict__ x, long long npix,
                               double *__restrict__ sums) {
  __shared__ double part[256];
  const float2 *xs = x + (long long)blockIdx.x * npix;
  double acc = 0.0;
  for (long long i = threadIdx.x; i < npix; i += blockDim.x) acc += (double)xs[i].x;
  part[threadIdx.x] = acc;
  __syncthreads();
  for (int h = blockDim.x / 2; h > 0; h >>= 1) {
    if (threadIdx.x < h) part[threadIdx.x] += part[threadIdx.x + h];
    __syncthreads();
  }
  if (threadIdx.x == 0) sums[blockIdx.x] = part[0];
}

// w <- (target / sum_s) w per slice
__global__ void dcf_scale_kernel(double *__restrict__ w, const int *__restrict__ slice_of,
                                 long long M, const double *__restrict__ sums, double target) {
  for (long long m = blockIdx.x * (long long)blockDim.x + threadIdx.x; m < M;
       m += (long long)gridDim.x * blockDim.x) {
    const int s = slice_of ? slice_of[m] : 0;
    w[m] *= target / sums[s];
  }
}

__global__ void recip_real_kernel(const float2 *__restrict__ g, long long M, double *__restrict__ w,
                                  int *bad) {
  for (long long m = blockIdx.x * (long long)blockDim.x + threadIdx.x; m < M;
       m += (long long)gridDim.x * blockDim.x) {
    const double v = (double)g[m].x;
    if (v == 0.0) atomicOr(bad, 1);
    w[m] = 1.0 / v;
  }
}

unsigned grid_for(long long n, int threads) {
  long long b = (n + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > 148 * 32) b = 148 * 32;
  return (unsigned)b;
}

struct DcfBuffers {
  DMem f, g, slice_of;
  int alloc(mirt_nufft *p, cudaStream_t st) {
    const long long M = p->Mtot;
    DCK(f.alloc(std::max<long long>(M, 1) * sizeof(float2)));
    DCK(g.alloc(std::max<long long>(M, 1) * sizeof(float2)));
    if (p->nslice > 1) {
      DCK(slice_of.alloc(std::max<long long>(M, 1) * sizeof(int)));
      DCK(launch_fill_slice(p->ip->moff.as<long long>(), p->nslice, M, slice_of.as<int>(), st));
    }
    return MIRT_OK;
  }
};

// g = P P' f  (spread into the plan's grid, gather back; phase applied by the plan)
int ppt(mirt_nufft *p, const float2 *f, float2 *g, cudaStream_t st) {
  mirt_interp_plan *P = p->ip;
  DCK(launch_spread(P->a, P->t, P->ls, P->bin_start.as<int>(), f, p->grid.as<float2>(), st));
  DCK(launch_gather(P->ag, P->lg, p->grid.as<float2>(), g, st));
  return MIRT_OK;
}

// scale: sum(real(G' w)) = prod(N ./ fov) per slice (mri/ir_mri_density_comp.m:258-261)
int scale_to_psf(mirt_nufft *p, double *w, const double *fov, DcfBuffers &b, cudaStream_t st) {
  const long long M = p->Mtot;
  const int S = p->nslice;
  double target = 1.0;
  for (int d = 0; d < p->gg.D; d++) {
    const double fv = fov ? fov[d] : 1.0;
    if (!(fv > 0.0)) return api_fail(MIRT_ERR_ARG, "fov must be positive");
    target *= p->gg.N[d] / fv;
  }
  DMem x, sums;
  DCK(x.alloc((size_t)S * p->gg.npix * sizeof(float2)));
  DCK(sums.alloc(S * sizeof(double)));
  w_to_c64_kernel<<<grid_for(M, 256), 256, 0, st>>>(w, M, b.f.as<float2>());
  DCK(cudaGetLastError());
  int rc = mirt_nufft_adjoint(p, b.f.p, x.p, st);
  if (rc) return rc;
  psf_sum_kernel<<<S, 256, 0, st>>>(x.as<float2>(), p->gg.npix, sums.as<double>());
  DCK(cudaGetLastError());
  const int *slice_of = S > 1 ? b.slice_of.as<int>() : nullptr;
  dcf_scale_kernel<<<grid_for(M, 256), 256, 0, st>>>(w, slice_of, M, sums.as<double>(), target);
  DCK(cudaGetLastError());
  return MIRT_OK;
}

int check_plan(mirt_nufft *p, const double *w) {
  if (!p) return api_fail(MIRT_ERR_ARG, "nufft is NULL");
  if (!w) return api_fail(MIRT_ERR_ARG, "w is NULL");
  if (p->C != 1)
    return api_fail(MIRT_ERR_ARG,
                    "density compensation needs a single-column NUFFT plan (ncol = 1)");
  return MIRT_OK;
}

}  // namespace

extern "C" {

int mirt_dcf_pipe(mirt_nufft *p, double *w, int32_t init_ones, int32_t niter, double thresh,
                  const double *fov, int32_t *iters, double *resid, void *stream) {
  int rc = check_plan(p, w);
  if (rc) return rc;
  if (niter < 0 || !(thresh >= 0.0)) return api_fail(MIRT_ERR_ARG, "need niter >= 0, thresh >= 0");
  cudaStream_t st = as_stream(stream);
  const long long M = p->Mtot;
  const int S = p->nslice;
  DcfBuffers b;
  rc = b.alloc(p, st);
  if (rc) return rc;
  DMem active, rbits, rdev, idev, flags;
  DCK(active.alloc(S * sizeof(int)));
  DCK(rbits.alloc(S * sizeof(unsigned long long)));
  DCK(rdev.alloc(S * sizeof(double)));
  DCK(idev.alloc(S * sizeof(int)));
  DCK(flags.alloc(3 * sizeof(int)));  // non-positive goal seen, slices still active, blocks done
  {
    std::vector<int> ones(S, 1);
    DCK(cudaMemcpyAsync(active.p, ones.data(), S * sizeof(int), cudaMemcpyHostToDevice, st));
  }
  DCK(cudaMemsetAsync(rbits.p, 0, S * sizeof(unsigned long long), st));
  DCK(cudaMemsetAsync(rdev.p, 0, S * sizeof(double), st));
  DCK(cudaMemsetAsync(idev.p, 0, S * sizeof(int), st));
  DCK(cudaMemsetAsync(flags.p, 0, 3 * sizeof(int), st));
  const int *slice_of = p->nslice > 1 ? b.slice_of.as<int>() : nullptr;
  if (init_ones) fill_ones_kernel<<<grid_for(M, 256), 256, 0, st>>>(w, M);
  DCK(cudaGetLastError());
  w_to_c64_kernel<<<grid_for(M, 256), 256, 0, st>>>(w, M, b.f.as<float2>());
  DCK(cudaGetLastError());
  int *fl = flags.as<int>();
  const PipeState ps{active.as<int>(), rbits.as<unsigned long long>(), rdev.as<double>(),
                     idev.as<int>(), fl, fl + 1, reinterpret_cast<unsigned *>(fl + 2)};
  const long long per = kUpdThreads * kUpdPer;
  const unsigned nblk = (unsigned)std::max<long long>((M + per - 1) / per, 1);
  for (int it = 1; it <= niter + 1; it++) {
    rc = ppt(p, b.f.as<float2>(), b.g.as<float2>(), st);
    if (rc) return rc;
    pipe_update_kernel<<<nblk, kUpdThreads, 0, st>>>(b.g.as<float2>(), slice_of, M, w,
                                                     b.f.as<float2>(), ps, S, it, thresh);
    DCK(cudaGetLastError());
    if (it % 4 == 0 || it == niter + 1) {
      int h[2];
      DCK(cudaMemcpyAsync(h, flags.p, sizeof h, cudaMemcpyDeviceToHost, st));
      DCK(cudaStreamSynchronize(st));
      if (h[0]) return api_fail(MIRT_ERR_ARG, "pipe bug: non-positive P P' w");
      if (h[1] == 0) break;
    }
  }
  {
    int h[2];
    DCK(cudaMemcpyAsync(h, flags.p, sizeof h, cudaMemcpyDeviceToHost, st));
    DCK(cudaStreamSynchronize(st));
    if (h[0]) return api_fail(MIRT_ERR_ARG, "pipe bug: non-positive P P' w");
  }
  rc = scale_to_psf(p, w, fov, b, st);
  if (rc) return rc;
  if (iters) DCK(cudaMemcpyAsync(iters, idev.p, S * sizeof(int), cudaMemcpyDeviceToHost, st));
  if (resid) DCK(cudaMemcpyAsync(resid, rdev.p, S * sizeof(double), cudaMemcpyDeviceToHost, st));
  DCK(cudaStreamSynchronize(st));
  return MIRT_OK;
}

int mirt_dcf_scale(mirt_nufft *p, double *w, const double *fov, void *stream) {
  int rc = check_plan(p, w);
  if (rc) return rc;
  cudaStream_t st = as_stream(stream);
  DcfBuffers b;
  rc = b.alloc(p, st);
  if (rc) return rc;
  rc = scale_to_psf(p, w, fov, b, st);
  if (rc) return rc;
  DCK(cudaStreamSynchronize(st));
  return MIRT_OK;
}

int mirt_dcf_jackson(mirt_nufft *p, double *w, void *stream) {
  int rc = check_plan(p, w);
  if (rc) return rc;
  cudaStream_t st = as_stream(stream);
  const long long M = p->Mtot;
  DcfBuffers b;
  rc = b.alloc(p, st);
  if (rc) return rc;
  DMem flags;
  DCK(flags.alloc(sizeof(int)));
  DCK(cudaMemsetAsync(flags.p, 0, sizeof(int), st));
  fill_ones_kernel<<<grid_for(M, 256), 256, 0, st>>>(w, M);
  w_to_c64_kernel<<<grid_for(M, 256), 256, 0, st>>>(w, M, b.f.as<float2>());
  DCK(cudaGetLastError());
  rc = ppt(p, b.f.as<float2>(), b.g.as<float2>(), st);
  if (rc) return rc;
  recip_real_kernel<<<grid_for(M, 256), 256, 0, st>>>(b.g.as<float2>(), M, w, flags.as<int>());
  DCK(cudaGetLastError());
  int h = 0;
  DCK(cudaMemcpyAsync(&h, flags.p, sizeof h, cudaMemcpyDeviceToHost, st));
  DCK(cudaStreamSynchronize(st));
  if (h) return api_fail(MIRT_ERR_ARG, "jackson: P P' 1 has a zero entry");
  return MIRT_OK;
}

}  // extern "C"
