// interp.cu -- bin keys, the stable bin sort, and the public launchers of the
// table-interpolation kernels (templates in interp_impl.cuh, instantiated per
// dimension in interp_d{1,2,3}.cu).
#include "interp_impl.cuh"

namespace mirt {
// ------------------------------------------------------------------------
// bin keys
// ------------------------------------------------------------------------
__global__ void bin_keys_kernel(InterpArgs a, Tiling t, uint32_t *keys) {
  const long long m = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (m >= a.Mtot) return;
  int bin = 0, mul = 1;
  for (int d = 0; d < a.g.D; d++) {
    const double td = a.tm[(long long)d * a.Mtot + m];
    const int k0 = wrapk(koff_of(td, a.g.J[d]), a.g.K[d]);
    bin += (k0 / t.B[d]) * mul;
    mul *= t.nbin[d];
  }
  const int s = a.slice_id ? a.slice_id[m] : 0;
  keys[m] = (uint32_t)s * (uint32_t)t.nbins + (uint32_t)bin;
}

cudaError_t launch_bin_keys(const InterpArgs &a, const Tiling &t, uint32_t *keys,
                            cudaStream_t st) {
  if (a.Mtot == 0) return cudaSuccess;
  const int thr = 256;
  const long long blocks = (a.Mtot + thr - 1) / thr;
  bin_keys_kernel<<<(unsigned)blocks, thr, 0, st>>>(a, t, keys);
  return cudaGetLastError();
}

// ------------------------------------------------------------------------
// stable LSD radix sort of bin keys (8-bit digits), deterministic
// ------------------------------------------------------------------------
namespace {
constexpr int RS_THREADS = 256;
constexpr int RS_WARPS = RS_THREADS / 32;
// Elements per block: the scatter walks its chunk 256 elements at a time, so few
// samples take short chunks that fill the SMs (413,696 samples: 12.5 -> 6.4 us a
// pass), many take long ones that keep the table of counts small.
int rs_chunk(long long n) { return n <= 148ll * 8 * 1024 ? 1024 : 4096; }
constexpr unsigned FULL = 0xffffffffu;

__global__ void rs_hist(const uint32_t *keys, long long n, int shift, int nblk, int chunk,
                        int *hist) {
  __shared__ int cnt[256];
  cnt[threadIdx.x] = 0;
  __syncthreads();
  const long long beg = (long long)blockIdx.x * chunk;
  const long long end = min(beg + chunk, n);
  for (long long i = beg + threadIdx.x; i < end; i += RS_THREADS)
    atomicAdd(&cnt[(keys[i] >> shift) & 255u], 1);
  __syncthreads();
  hist[threadIdx.x * nblk + blockIdx.x] = cnt[threadIdx.x];
}

// Exclusive scan of 256 ints by a block of 256 threads (wsum: 8 ints of shared
// memory; the caller separates two uses with a barrier)
__device__ __forceinline__ int block_scan256(int x, int *wsum, int *total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int s = x;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(FULL, s, o);
    if (lane >= o) s += y;
  }
  if (lane == 31) wsum[w] = s;
  __syncthreads();
  int base = 0, all = 0;
  for (int i = 0; i < RS_WARPS; i++) {
    if (i < w) base += wsum[i];
    all += wsum[i];
  }
  *total = all;
  return base + s - x;
}

// Exclusive scan of each digit's row of block counts, one block a digit, and the
// row's total; the scatter adds the scan of the totals (one block over the whole
// table took 19.8 us a pass at 413,696 samples, latency of serial loads; 2.6 us so).
__global__ void rs_scan_rows(int *v, int nblk, int *tot) {
  __shared__ int wsum[RS_WARPS];
  int *row = v + (size_t)blockIdx.x * nblk;
  int run = 0;
  for (int i0 = 0; i0 < nblk; i0 += RS_THREADS) {
    const int i = i0 + threadIdx.x;
    const int x = i < nblk ? row[i] : 0;
    int all;
    const int e = block_scan256(x, wsum, &all);
    if (i < nblk) row[i] = run + e;
    run += all;
    __syncthreads();
  }
  if (threadIdx.x == 0) tot[blockIdx.x] = run;
}

// Stable scatter: elements keep their input order within a digit.  Each warp
// ranks its 32 elements with match_any; warps are then ordered by a per-digit
// prefix over the warp counts, and the block's running digit offsets advance.
__global__ void rs_scatter(const uint32_t *kin, const int *vin, long long n, int shift, int nblk,
                           int chunk, const int *offs, const int *tot, uint32_t *kout, int *vout) {
  __shared__ int run[256];
  __shared__ int wcnt[RS_WARPS][256];
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  {
    int all;
    run[tid] = offs[tid * nblk + blockIdx.x] + block_scan256(tot[tid], &wcnt[0][0], &all);
  }
  __syncthreads();
  const long long beg = (long long)blockIdx.x * chunk;
  const long long end = min(beg + chunk, n);
  const unsigned lt = (1u << lane) - 1u;
  for (long long base = beg; base < end; base += RS_THREADS) {
    for (int i = tid; i < RS_WARPS * 256; i += RS_THREADS) (&wcnt[0][0])[i] = 0;
    __syncthreads();
    const long long i = base + tid;
    const bool valid = i < end;
    const uint32_t key = valid ? kin[i] : 0u;
    const int val = valid ? (vin ? vin[i] : (int)i) : 0;
    const unsigned dig = valid ? ((key >> shift) & 255u) : 256u;
    const unsigned peers = __match_any_sync(FULL, dig);
    const int rank = __popc(peers & lt);
    if (valid && rank == 0) wcnt[w][dig] = __popc(peers);
    __syncthreads();
    {
      int acc = run[tid];
      for (int ww = 0; ww < RS_WARPS; ww++) {
        const int c = wcnt[ww][tid];
        wcnt[ww][tid] = acc;
        acc += c;
      }
      run[tid] = acc;
    }
    __syncthreads();
    if (valid) {
      const int pos = wcnt[w][dig] + rank;
      kout[pos] = key;
      vout[pos] = val;
    }
    __syncthreads();
  }
}

__global__ void rs_bin_start(const uint32_t *ks, long long n, int nbins, int *bin_start) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const long long k = ks[i];
  const long long kp = i > 0 ? (long long)ks[i - 1] : -1;
  for (long long b = kp + 1; b <= k; b++) bin_start[b] = (int)i;
  if (i == n - 1)
    for (long long b = k + 1; b <= nbins; b++) bin_start[b] = (int)n;
}

__global__ void fill_int(int *p, int n, int v) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] = v;
}
}  // namespace

size_t radix_sort_tmp_bytes(long long n) {
  const long long nblk = (n + rs_chunk(n) - 1) / rs_chunk(n) + 1;
  return (size_t)(4 * n * 4) + (size_t)(256 * nblk * 4) + 1024;
}

cudaError_t radix_sort_bins(const uint32_t *keys, long long n, int nbins, void *tmp, int *perm,
                            int *bin_start, cudaStream_t st) {
  if (n == 0) {
    fill_int<<<(nbins + 1 + 255) / 256, 256, 0, st>>>(bin_start, nbins + 1, 0);
    return cudaGetLastError();
  }
  const int chunk = rs_chunk(n);
  const int nblk = (int)((n + chunk - 1) / chunk);
  char *p = static_cast<char *>(tmp);
  uint32_t *kA = reinterpret_cast<uint32_t *>(p);
  uint32_t *kB = kA + n;
  int *vA = reinterpret_cast<int *>(kB + n);
  int *vB = vA + n;
  int *hist = vB + n, *tot = hist + 256 * (size_t)nblk;
  int bits = 1;
  while (bits < 32 && (1ll << bits) < (long long)nbins) bits++;
  const int npass = (bits + 7) / 8;
  const uint32_t *kin = keys;
  const int *vin = nullptr;
  for (int ps = 0; ps < npass; ps++) {
    const int shift = 8 * ps;
    uint32_t *kout = (ps & 1) ? kB : kA;
    int *vout = (ps == npass - 1) ? perm : ((ps & 1) ? vB : vA);
    rs_hist<<<nblk, RS_THREADS, 0, st>>>(kin, n, shift, nblk, chunk, hist);
    rs_scan_rows<<<256, RS_THREADS, 0, st>>>(hist, nblk, tot);
    rs_scatter<<<nblk, RS_THREADS, 0, st>>>(kin, vin, n, shift, nblk, chunk, hist, tot, kout, vout);
    kin = kout;
    vin = vout;
  }
  rs_bin_start<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(kin, n, nbins, bin_start);
  return cudaGetLastError();
}

// ------------------------------------------------------------------------
// visit lists of the 3D line sweep
// ------------------------------------------------------------------------
namespace {
// Per bin column, the samples of the bin lines around the block (lane l keeps lines l
// and l + 32) in line and sort order, then the column's dense bins in line order: one
// warp a column counts them (count), one warp a part lists its columns (64^3, a million
// samples: 84 and 167 us).
__global__ void sweep3_list_kernel(InterpArgs a, Tiling t, const int *__restrict__ bin_start, int B2,
                                   int B3, long long n, const int4 *__restrict__ part,
                                   const long long *__restrict__ off, int *__restrict__ count,
                                   int *__restrict__ pos, unsigned char *__restrict__ line) {
  const long long i = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
  if (i >= n) return;
  const int lane = threadIdx.x & 31;
  const int K1 = a.g.K[0], K2 = a.g.K[1], K3 = a.g.K[2];
  const int4 pt = count ? make_int4((int)(i / K1), (int)(i % K1), (int)(i % K1) + 1, 0) : part[i];
  const long long block = pt.x;
  const int Q2 = B2 + 5, nl = Q2 * (B3 + 5);
  const int nby = (K2 + B2 - 1) / B2, nbz = (K3 + B3 - 1) / B3;
  const int y0 = (int)(block % nby) * B2;
  const int z0 = (int)(block / nby % nbz) * B3;
  const long long slice = block / ((long long)nby * nbz);
  const int *bs = bin_start + slice * t.nbins;
  const int *dof = t.dense_of ? t.dense_of + slice * t.nbins : nullptr;
  const int dmin = t.dense_of ? t.dense_min : 0x7fffffff;
  long long base[2];
  for (int h = 0; h < 2; h++) {
    const int l = lane + 32 * h;
    int r = (y0 - 5 + l % Q2) % K2, z = (z0 - 5 + l / Q2) % K3;
    if (r < 0) r += K2;
    if (z < 0) z += K3;
    base[h] = l < nl ? ((long long)z * K2 + r) * K1 : -1;
  }
  long long at = count ? 0 : off[i];
  for (int x = pt.y; x < pt.z; x++) {
    for (int h = 0; h < 2; h++) {
      const int b0 = base[h] >= 0 ? bs[base[h] + x] : 0;
      const int n = base[h] >= 0 ? bs[base[h] + x + 1] - b0 : 0;
      const int s = n >= dmin ? 0 : n;
      int inc = s;
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(FULL, inc, o);
        if (lane >= o) inc += u;
      }
      if (pos)
        for (int k = 0; k < s; k++) {
          pos[at + inc - s + k] = b0 + k;
          line[at + inc - s + k] = (unsigned char)(lane + 32 * h);
        }
      at += __shfl_sync(FULL, inc, 31);
    }
    for (int h = 0; h < 2 && dof; h++) {
      const int n = base[h] >= 0 ? bs[base[h] + x + 1] - bs[base[h] + x] : 0;
      const unsigned m = __ballot_sync(FULL, n >= dmin && n > 0);
      if (pos && n >= dmin && n > 0) {
        const long long i = at + __popc(m & ((1u << lane) - 1u));
        pos[i] = ~dof[base[h] + x];
        line[i] = (unsigned char)(lane + 32 * h);
      }
      at += __popc(m);
    }
  }
  if (count && lane == 0) count[i] = (int)at;
}
}  // namespace

cudaError_t launch_sweep3_list(const InterpArgs &a, const Tiling &t, const int *bin_start, int B2,
                               int B3, long long n, const int4 *part, const long long *off,
                               int *count, int *pos, unsigned char *line, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  sweep3_list_kernel<<<(unsigned)((n + 7) / 8), 256, 0, st>>>(a, t, bin_start, B2, B3, n, part, off,
                                                             count, pos, line);
  return cudaGetLastError();
}

// ------------------------------------------------------------------------
// per-position tap data
// ------------------------------------------------------------------------
cudaError_t launch_prep_taps(const InterpArgs &a, float2 *W, int4 *K0, cudaStream_t st) {
  if (a.Mtot == 0) return cudaSuccess;
  const unsigned blocks = (unsigned)((a.Mtot + 255) / 256);
  if (a.real_tab)
    detail::prep_taps_kernel<true><<<blocks, 256, 0, st>>>(a, W, K0);
  else
    detail::prep_taps_kernel<false><<<blocks, 256, 0, st>>>(a, W, K0);
  return cudaGetLastError();
}

// ------------------------------------------------------------------------
// public launchers
// ------------------------------------------------------------------------
namespace {
cudaError_t dispatch(detail::Req &r) {
  switch (r.a->g.D) {
    case 1: return detail::dispatch_d1(r);
    case 2: return detail::dispatch_d2(r);
    case 3: return detail::dispatch_d3(r);
    default: return cudaErrorInvalidValue;
  }
}
}  // namespace

cudaError_t query_gather_grid(const InterpArgs &a, Launch &l) {
  detail::Req r{detail::GATHER_GRID, &a, nullptr, &l, nullptr, nullptr, nullptr, 0};
  return dispatch(r);
}

cudaError_t launch_gather(const InterpArgs &a, const Launch &l, const float2 *ck, float2 *fm,
                          cudaStream_t st) {
  if (a.Mtot == 0 || a.C == 0) return cudaSuccess;
  Launch lc = l;
  detail::Req r{detail::GATHER, &a, nullptr, &lc, nullptr, ck, fm, st};
  return dispatch(r);
}

namespace {
__global__ void mark_dense_kernel(const int *__restrict__ dense_bin, int n, int *dense_of) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dense_of[dense_bin[i]] = i;
}
}  // namespace

cudaError_t launch_mark_dense(const int *dense_bin, int n, int *dense_of, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  mark_dense_kernel<<<(n + 255) / 256, 256, 0, st>>>(dense_bin, n, dense_of);
  return cudaGetLastError();
}

cudaError_t launch_spread(const InterpArgs &a, const Tiling &t, const Launch &l,
                          const int *bin_start, const float2 *fm, float2 *ck, cudaStream_t st) {
  if (a.C == 0) return cudaSuccess;
  Launch lc = l;
  if (t.split && (t.sweep || !l.atomic)) {
    if (t.split_nteams) {
      Tiling ts = t;
      ts.sweep = -1;
      ts.sweep_rows = 4;
      ts.sweep_staged = 2;
      ts.dense_on = 0;
      ts.sweep_team = t.split_team;
      ts.nteams = t.split_nteams;
      ts.team_order = t.split_order;
      ts.team_next = t.split_next;
      lc.cw = 32;
      detail::Req r{detail::SPREAD, &a, &ts, &lc, bin_start, fm, ck, st};
      cudaError_t e = dispatch(r);
      if (e != cudaSuccess) return e;
    }
    return launch_spread_points(a, t, bin_start, fm, ck, st);
  }
  if (t.points && (t.sweep || !l.atomic)) return launch_spread_points(a, t, bin_start, fm, ck, st);
  detail::Req r{detail::SPREAD, &a, &t, &lc, bin_start, fm, ck, st};
  return dispatch(r);
}

}  // namespace mirt
