// features.cu -- per-sample trajectory features for the learned density
// compensation: normalised radius |omega| / pi, angle atan2(omega_2,
// omega_1) / pi, and log1p of a 16-bin histogram of the distances to the
// other samples of the same trajectory within 2 grid cells (bins of 1/8
// cell, distances in units of the oversampled grid, t = omega / (2 pi / K),
// no periodic wrap).
//
// Samples are bucketed into 2 x 2-cell hash cells by the library's stable
// radix sort (slice-major keys), so the neighbours of a sample lie in the 3 x
// 3 hash cells around its own; the scan reads the sorted coordinate copy
// contiguously.  Squared distances are formed in FP64 with explicitly rounded
// operations and compared with the exact squared bin edges, so the counts are
// reproducible bit for bit by an FP64 restatement.
#include "../../include/mirt_b200.h"

#include <new>
#include <string>

#include "runtime.cuh"

using namespace mirt;

namespace {

#define FCK(call)                                                                     \
  do {                                                                                \
    cudaError_t e_ = (call);                                                          \
    if (e_ != cudaSuccess)                                                            \
      return api_fail(e_ == cudaErrorMemoryAllocation ? MIRT_ERR_ALLOC : MIRT_ERR_CUDA, \
                      std::string(#call) + ": " + cudaGetErrorString(e_));            \
  } while (0)

struct FeatGeom {
  double scale[2];  // K / (2 pi): omega -> grid units
  int K[2];
  int nc[2];        // hash cells per dimension (2 grid units each)
  int ncells;       // nc[0] * nc[1]
};

__device__ __forceinline__ int cell_of(double t, int K, int nc) {
  // t in [-K/2, K/2) for omega in [-pi, pi); clamp the rest onto the edge cells
  int c = (int)floor((t + 0.5 * K) * 0.5);
  return c < 0 ? 0 : (c >= nc ? nc - 1 : c);
}

// grid coordinates and sort key (slice-major, then hash cell) of each sample
__global__ void feat_keys_kernel(const double *__restrict__ om, long long M,
                                 const int *__restrict__ slice_of, FeatGeom g,
                                 double2 *__restrict__ t, uint32_t *__restrict__ keys) {
  const long long m = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (m >= M) return;
  const double t0 = __dmul_rn(om[m], g.scale[0]);
  const double t1 = __dmul_rn(om[M + m], g.scale[1]);
  t[m] = make_double2(t0, t1);
  const int s = slice_of ? slice_of[m] : 0;
  const int c = cell_of(t0, g.K[0], g.nc[0]) + g.nc[0] * cell_of(t1, g.K[1], g.nc[1]);
  keys[m] = (uint32_t)((long long)s * g.ncells + c);
}

// what the histogram needs of each sorted position: coordinates, {first bin of its
// slice, hash cell, sample} and the two polar features
__global__ void feat_gather_kernel(const double *__restrict__ om, const double2 *__restrict__ t,
                                   const int *__restrict__ perm, const int *__restrict__ slice_of,
                                   long long M, FeatGeom g, double2 *__restrict__ ts,
                                   int4 *__restrict__ info, float2 *__restrict__ polar) {
  const long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (p >= M) return;
  const int m = perm[p];
  const double2 tp = t[m];
  const double w0 = om[m], w1 = om[M + m];
  ts[p] = tp;
  info[p] = make_int4((slice_of ? slice_of[m] : 0) * g.ncells, cell_of(tp.x, g.K[0], g.nc[0]),
                      cell_of(tp.y, g.K[1], g.nc[1]), m);
  polar[p] = make_float2((float)(sqrt(w0 * w0 + w1 * w1) / M_PI), (float)(atan2(w1, w0) / M_PI));
}

// Eight lanes per sorted position over the candidates of its 3 x 3 hash cells (three
// runs of the sort order, walked as one), four positions a warp with their histograms
// in shared memory; the warp writes their rows.  The bin of a distance is its FP32
// square root, put right by FP64 comparisons with the exact edges (b / 8)^2, so the
// counts stay those of the FP64 comparisons.  Bound by the chain of dependent loads
// and FP64 operations of the short walks (27 candidates on average, 600 at the
// trajectory's centre; 8 slices of 101 spokes x 512): 204 us with one thread a sample
// and 15 comparisons a candidate, 87 us so.
// floor(8 sqrt(d2)) or one off it, 0 <= d2 < 4: the double's bits cut to FP32 (below
// 2^-126 to zero), an approximate root and a rounding by a large constant, as the
// conversions between FP64, FP32 and integers run at a fraction of the rate
__device__ __forceinline__ int bin_guess(double d2) {
  const int hi = max(__double2hiint(d2) - 0x38000000, 0);
  const float f = __uint_as_float(__funnelshift_l(__double2loint(d2), hi, 3));
  float r;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(f));
  const int b = __float_as_int(fmaf(8.f, r, 8388607.5f)) & 31;
  return b > 15 ? (b > 16 ? 0 : 15) : b;
}

constexpr int kFeatLanes = 8, kFeatBlock = 256, kFeatPos = 32 / kFeatLanes;

__global__ void __launch_bounds__(kFeatBlock)
    feat_hist_kernel(const double2 *__restrict__ ts, const int4 *__restrict__ info,
                     const float2 *__restrict__ polar, const int *__restrict__ bin_start,
                     long long M, FeatGeom g, float *__restrict__ feat) {
  __shared__ int hist[kFeatBlock / 32][16 * kFeatPos];
  __shared__ double edge[17];  // exact squared bin edges
  const int warp = threadIdx.x >> 5, ln = threadIdx.x & 31;
  const int pos = ln / kFeatLanes, lane = ln % kFeatLanes;
  int *h = hist[warp];
  if (threadIdx.x < 17) edge[threadIdx.x] = (threadIdx.x * 0.125) * (threadIdx.x * 0.125);
  h[ln] = 0;
  h[32 + ln] = 0;
  __syncthreads();
  const long long p0 = ((long long)blockIdx.x * (kFeatBlock / 32) + warp) * kFeatPos;
  if (p0 >= M) return;
  const int np = (int)min((long long)kFeatPos, M - p0);
  const long long p = p0 + pos;
  int m = 0;
  if (pos < np) {
    const int4 in = info[p];
    const double2 tp = ts[p];
    m = in.w;
    const int *bs = bin_start + in.x;
    const int ca = max(in.y - 1, 0), cb = min(in.y + 1, g.nc[0] - 1);
    int first[3], n[3];
#pragma unroll
    for (int r = 0; r < 3; r++) {
      // the three cells of a row are contiguous in the sort order
      const int cc1 = in.z + r - 1;
      const bool ok = cc1 >= 0 && cc1 < g.nc[1];
      const int *b = bs + (ok ? (long long)cc1 * g.nc[0] : 0);
      first[r] = ok ? b[ca] : 0;
      n[r] = ok ? b[cb + 1] - first[r] : 0;
    }
    const int n01 = n[0] + n[1], total = n01 + n[2];
    const int a1 = first[1] - n[0], a2 = first[2] - n01;
    for (int i = lane; i < total; i += kFeatLanes) {
      const int q = i + (i < n[0] ? first[0] : i < n01 ? a1 : a2);
      const double2 tq = ts[q];
      const double dx = __dsub_rn(tq.x, tp.x), dy = __dsub_rn(tq.y, tp.y);
      const double d2 = __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy));
      if (d2 < 4.0 && q != p) {
        // bin b: (b/8)^2 <= d2 < ((b+1)/8)^2, edges exact in binary
        int b = bin_guess(d2);
        b += (d2 >= edge[b + 1]) - (d2 < edge[b]);
        atomicAdd(h + b * kFeatPos + pos, 1);
      }
    }
  }
  __syncwarp();
#pragma unroll
  for (int e = 0; e < 16 * kFeatPos; e += 32)
    h[e + ln] = __float_as_int(log1pf((float)h[e + ln]));
  __syncwarp();
  for (int e = ln; e < ((np * MIRT_DCF_NFEAT + 31) & ~31); e += 32) {
    const int r = e / MIRT_DCF_NFEAT, j = e - r * MIRT_DCF_NFEAT;
    const int mr = __shfl_sync(0xffffffffu, m, (r < np ? r : 0) * kFeatLanes);
    if (r < np) {
      float v;
      if (j < 2) {
        const float2 pl = polar[p0 + r];
        v = j ? pl.y : pl.x;
      } else {
        v = __int_as_float(h[(j - 2) * kFeatPos + r]);
      }
      feat[(long long)mr * MIRT_DCF_NFEAT + j] = v;
    }
  }
}

}  // namespace

extern "C" int mirt_dcf_features(const double *om, int64_t M, const int64_t *slice_moff,
                                 int32_t nslice, const int32_t *K, float *feat, void *stream) try {
  if (!om || !K || !feat) return api_fail(MIRT_ERR_ARG, "NULL argument");
  if (M < 0 || nslice < 1) return api_fail(MIRT_ERR_ARG, "need M >= 0 and nslice >= 1");
  if (M >= (1ll << 31)) return api_fail(MIRT_ERR_ARG, "M too large");
  if (K[0] < 2 || K[1] < 2) return api_fail(MIRT_ERR_ARG, "K must be >= 2");
  FeatGeom g{};
  for (int d = 0; d < 2; d++) {
    g.K[d] = K[d];
    g.scale[d] = K[d] / (2.0 * M_PI);
    g.nc[d] = (K[d] + 1) / 2;
  }
  g.ncells = g.nc[0] * g.nc[1];
  const long long nbins = (long long)g.ncells * nslice;
  if (nbins >= (1ll << 31) - 1) return api_fail(MIRT_ERR_ARG, "too many hash cells (K, nslice)");
  std::vector<long long> moff(nslice + 1);
  if (slice_moff) {
    for (int s = 0; s <= nslice; s++) moff[s] = slice_moff[s];
    if (moff[0] != 0 || moff[nslice] != M)
      return api_fail(MIRT_ERR_ARG, "slice offsets must start at 0 and end at M");
    for (int s = 0; s < nslice; s++)
      if (moff[s + 1] < moff[s]) return api_fail(MIRT_ERR_ARG, "slice offsets must not decrease");
  } else if (nslice != 1) {
    return api_fail(MIRT_ERR_ARG, "slice offsets required for nslice > 1");
  }
  if (M == 0) return MIRT_OK;
  cudaStream_t st = as_stream(stream);
  DMem dmoff, slice, t, ts, keys, perm, bstart, tmp, info, polar;
  const int *slice_of = nullptr;
  if (nslice > 1) {
    FCK(dmoff.alloc((nslice + 1) * sizeof(long long)));
    FCK(cudaMemcpyAsync(dmoff.p, moff.data(), (nslice + 1) * sizeof(long long),
                        cudaMemcpyHostToDevice, st));
    FCK(slice.alloc(M * sizeof(int)));
    FCK(launch_fill_slice(dmoff.as<long long>(), nslice, M, slice.as<int>(), st));
    slice_of = slice.as<int>();
  }
  FCK(t.alloc(M * sizeof(double2)));
  FCK(ts.alloc(M * sizeof(double2)));
  FCK(info.alloc(M * sizeof(int4)));
  FCK(polar.alloc(M * sizeof(float2)));
  FCK(keys.alloc(M * sizeof(uint32_t)));
  FCK(perm.alloc(M * sizeof(int)));
  FCK(bstart.alloc((nbins + 1) * sizeof(int)));
  FCK(tmp.alloc(radix_sort_tmp_bytes(M)));
  const unsigned blk = (unsigned)((M + 255) / 256);
  feat_keys_kernel<<<blk, 256, 0, st>>>(om, M, slice_of, g, t.as<double2>(), keys.as<uint32_t>());
  FCK(cudaGetLastError());
  FCK(radix_sort_bins(keys.as<uint32_t>(), M, (int)nbins, tmp.p, perm.as<int>(), bstart.as<int>(),
                      st));
  feat_gather_kernel<<<blk, 256, 0, st>>>(om, t.as<double2>(), perm.as<int>(), slice_of, M, g,
                                          ts.as<double2>(), info.as<int4>(), polar.as<float2>());
  FCK(cudaGetLastError());
  const long long per = kFeatBlock / 32 * kFeatPos;
  feat_hist_kernel<<<(unsigned)((M + per - 1) / per), kFeatBlock, 0, st>>>(
      ts.as<double2>(), info.as<int4>(), polar.as<float2>(), bstart.as<int>(), M, g, feat);
  FCK(cudaGetLastError());
  FCK(cudaStreamSynchronize(st));
  return MIRT_OK;
} catch (const std::bad_alloc &) {
  return mirt::api_fail(MIRT_ERR_ALLOC, "out of host memory");
}
