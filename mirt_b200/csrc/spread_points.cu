// spread_points.cu -- the adjoint spread (nufft/table/interp{1,2,3}_table1_adj.c)
// over the grid points' own samples: any D <= 3, J, K and column count.
//
// A group of lanes owns a brick of grid points (blocks of four consecutive
// points of a row, a few rows and planes of them) and keeps its points' sums in
// registers: CW lanes of NC columns each per block.  With one-point sort bins
// the samples that reach the brick are, for each of its J2 - 1 + rows times
// J3 - 1 + planes tap rows, the bins from J1 - 1 points before it to its end:
// one run of the sort order.  The group lists the runs (their first positions
// and running counts), and walks the samples S at a time: each lane finds the
// run of one sample, loads its header and copies its tap record and its columns
// times conj(phase) into the group's shared-memory stage, all loads of a chunk
// in flight together, and then every lane adds each staged sample's taps into
// its own block where the block's row and plane are among the sample's.  The
// samples are read through the sort permutation: no ordering pass and no per-plan
// copy.
//
// Dense bricks (the k-space centre of radial and kooshball trajectories): the
// plan gives each base tile of bricks a split G, a power of two, so that no
// group walks more than about pt_visits() samples: the tile becomes G CTAs of 1/G
// of its bricks, with G groups per brick that take every G-th chunk and are
// summed in a fixed order; CTAs that share a brick leave their sums in the plan's
// scratch, and the last of them to finish adds them in order (one launch of a plan at a
// time).  G depends on the trajectory alone: every grid point is summed in one order,
// bitwise reproducible, with no atomics on the sums.
//
// Bound by instruction issue (about 100 warp instructions per sample at one
// column in 2D, 46 % of the lanes of a visit useful).  Against the tiled spread,
// whose 32 lanes held the 6 taps of one column and whose warps walked a dense
// tile alone: 2D, one column, 8,192 samples on K = 128^2 1314 -> 15 us; 491,520
// samples on 6 x 512^2 1730 -> 110 us; 16 columns, 115,968 samples on 384^2 2457
// -> 112 us; 24 columns, 145,920 samples on 5 x 384^2 2481 -> 197 us (the
// unstaged row sweep with its dense-bin patches 570 us there); 3D, one column,
// 216,000 samples on 144 x 120 x 96 4530 -> 287 us.
#include <algorithm>

#include "interp_impl.cuh"

namespace mirt {
namespace {

constexpr int PT_THREADS = 128;
constexpr int PT_X = 4;          // grid points per block
constexpr int PT_SHARE = 6;      // log2 of the CTAs that may share a brick
// Samples a group walks before its tile is split: 32 in 1D and 2D (64 there:
// image of K = 128^2 21 us, 32: 15 us; a batch of 6 slices of K = 512^2 107 and
// 110 us), 64 in 3D, where listing a brick's runs costs more (K = 144 x 120 x 96:
// 290 us, 32: 356 us).
inline int pt_visits(int D) { return D == 3 ? 64 : 32; }

// Lane shape of CW column lanes: LB blocks per group (brick), GL lanes, S
// samples staged at a time, LS lanes copying one sample's record.
template <int CW>
struct PtShape {
  static constexpr int LB = CW <= 2 ? 8 : 4;
  static constexpr int GL = CW * LB;
  static constexpr int NGRP = PT_THREADS / GL;
  static constexpr int S = GL == 32 ? 16 : 8;
  static constexpr int LS = GL / S;
};
inline int pt_lb(int cw) { return cw <= 2 ? 8 : 4; }

// blocks of a brick per dimension
template <int D, int LB>
struct PtBrick {
  static constexpr int BZ = D == 3 ? 2 : 1;
  static constexpr int BY = D == 1 ? 1 : D == 2 ? 4 : LB == 8 ? 4 : 2;
  static constexpr int BX = LB / (BY * BZ);
};

// A plan's base tiles: bricks per tile and tiles per dimension, the brick's
// extent in points.
struct PtTile {
  int W, R2, R3;
  int bx, by, bz;
  int nt1, nt2, nt3;
};

inline PtTile pt_tile(const Geom &g, int cw) {
  const int lb = pt_lb(cw), ng = PT_THREADS / (cw * lb);
  PtTile t;
  t.bz = g.D == 3 ? 2 : 1;
  t.by = g.D == 1 ? 1 : g.D == 2 ? 4 : lb == 8 ? 4 : 2;
  t.bx = lb / (t.by * t.bz) * PT_X;
  t.R2 = g.D > 1 && ng >= 4 ? 2 : 1;
  t.R3 = g.D > 2 && ng >= 8 ? 2 : 1;
  t.W = ng / (t.R2 * t.R3);
  auto up = [](int n, int d) { return (n + d - 1) / d; };
  t.nt1 = up(g.K[0], t.W * t.bx);
  t.nt2 = up(g.K[1], t.R2 * t.by);
  t.nt3 = up(g.K[2], t.R3 * t.bz);
  return t;
}

// Shared memory of a group: the run list, then the stage.
struct PtSmem {
  int ne;                  // runs: the tap rows of a brick
  int o2, o3, rs;          // record offsets of the 2nd and 3rd dimension's taps, stride (float2)
  int off_rec, off_f, off_d, bytes;
};

inline PtSmem pt_smem(const Geom &g, const PtTile &t, int cw, int nc) {
  const int gl = cw * pt_lb(cw), S = gl == 32 ? 16 : 8;
  PtSmem s;
  s.ne = (t.by + g.J[1] - 1) * (t.bz + g.J[2] - 1);
  s.o2 = (4 + g.J[0] + 3 + 1) & ~1;
  s.o3 = s.o2 + ((g.J[1] + 1) & ~1);
  int e = g.D == 1 ? s.o2 : g.D == 2 ? s.o3 : s.o3 + ((g.J[2] + 1) & ~1);
  s.rs = (e / 2) | 1;
  s.rs *= 2;
  s.off_rec = (s.ne * 2 * 4 + 4 + 15) & ~15;
  s.off_f = s.off_rec + S * s.rs * 8;
  s.off_d = (s.off_f + S * cw * nc * 8 + 15) & ~15;
  s.bytes = s.off_d + S * 24;
  return s;
}

// header of every position: first tap, caller's sample index, phase
__global__ void point_header_kernel(InterpArgs a, int4 *__restrict__ hdr) {
  const long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (p >= a.Mtot) return;
  const float2 ph = a.phase ? a.phase[p] : make_float2(1.f, 0.f);
  hdr[p] = make_int4(a.K0[p].x, a.perm ? a.perm[p] : (int)p, __float_as_int(ph.x),
                     __float_as_int(ph.y));
}

// the most samples that reach one brick, of every base tile
__global__ void point_count_kernel(InterpArgs a, Tiling t, PtTile pt, int ngrp,
                                   const int *__restrict__ bin_start, long long ntile,
                                   int *__restrict__ most) {
  const long long tile = blockIdx.x;
  if (tile >= ntile) return;
  const Geom &g = a.g;
  long long r = tile;
  const int t1 = (int)(r % pt.nt1);
  r /= pt.nt1;
  const int t2 = (int)(r % pt.nt2);
  r /= pt.nt2;
  const int t3 = (int)(r % pt.nt3);
  const int s = (int)(r / pt.nt3);
  const int *bs = bin_start + (long long)s * t.nbins;
  const int K1 = g.K[0], K2 = g.K[1], K3 = g.K[2];
  __shared__ int cnt[PT_THREADS / 8];
  if (threadIdx.x < ngrp) cnt[threadIdx.x] = 0;
  __syncthreads();
  const int nq2 = pt.by + g.J[1] - 1, nq = nq2 * (pt.bz + g.J[2] - 1);
  for (int i = threadIdx.x; i < ngrp * nq; i += blockDim.x) {
    const int b = i / nq, q = i - b * nq;
    const int X0 = (t1 * pt.W + b % pt.W) * pt.bx;
    const int Y0 = (t2 * pt.R2 + b / pt.W % pt.R2) * pt.by;
    const int Z0 = (t3 * pt.R3 + b / (pt.W * pt.R2)) * pt.bz;
    const int y = Y0 - g.J[1] + 1 + q % nq2, z = Z0 - g.J[2] + 1 + q / nq2;
    if (X0 >= K1 || Y0 >= K2 || Z0 >= K3 || y >= K2 || z >= K3) continue;
    const int *row = bs + (long long)((z < 0 ? z + K3 : z) * K2 + (y < 0 ? y + K2 : y)) * K1;
    const int u = X0 - g.J[0] + 1;
    int v = row[min(X0 + pt.bx, K1)] - row[max(u, 0)];
    if (u < 0) v += row[K1] - row[u + K1];
    atomicAdd(&cnt[b], v);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int m = 0;
    for (int b = 0; b < ngrp; b++) m = max(m, cnt[b]);
    most[tile] = m;
  }
}

// One lane's sums again, tap by tap from global memory, over the samples of its
// group's share (chunks part, part + 2^lg, ... of S samples of the brick's runs) in
// the walk's order and operations: X points from (x, y, z), columns c, c + cw, ...
// below C.  Called where the walk left a sum that is not finite; kept out of line, so
// that the walk's registers don't pay for it (without and with it: one real column,
// 63,114 samples on 402 x 350 22.0 and 23.0 us; 12 columns on 6 x 512^2 481 and 502; 16 on
// 384^2 121 and 118; 24 on 5 x 384^2 197 and 199; a test in the walk cost 2 to 5 % of the
// one- to 24-column passes).
template <int D, int NC, bool REAL>
__device__ __noinline__ void points_redo(const InterpArgs &a, const Tiling &t, const int *bin_start,
                                         const float2 *fm, int slice, int X0, int Y0, int Z0, int bw,
                                         int by0, int bz0, int part, int lg, int S, int x, int y,
                                         int z, int c, int cw, float2 *acc) {
  const Geom &g = a.g;
  const int *bs = bin_start + (long long)slice * t.nbins;
  const int J1 = g.J[0], J2 = D > 1 ? g.J[1] : 1, J3 = D > 2 ? g.J[2] : 1;
  const int K1 = g.K[0], K2 = D > 1 ? g.K[1] : 1, K3 = D > 2 ? g.K[2] : 1;
  const int nq2 = by0 + J2 - 1, nq = nq2 * (bz0 + J3 - 1);
  for (int k = 0; k < NC * PT_X; k++) acc[k] = make_float2(0.f, 0.f);
  for (int ps = 0; ps < 2; ps++) {
    int base = 0;  // samples of the runs before this one
    for (int e = 0; e < nq; e++) {
      const int yq = Y0 - J2 + 1 + e % nq2, zq = Z0 - J3 + 1 + e / nq2;
      if (yq >= K2 || zq >= K3) continue;
      const int *row = bs + ((zq < 0 ? zq + K3 : zq) * K2 + (yq < 0 ? yq + K2 : yq)) * K1;
      const int u = X0 - J1 + 1;
      int l = 0, n = 0;
      if (ps == 0) {
        l = row[max(u, 0)];
        n = row[min(X0 + bw, K1)] - l;
      } else if (u < 0) {
        l = row[u + K1];
        n = row[K1] - l;
      }
      const int j2 = y - yq, j3 = z - zq;
      for (int v = base; v < base + n; v++) {
        const int chunk = v / S;
        if ((chunk & ((1 << lg) - 1)) != part) {  // to the share's next chunk
          v = (chunk + ((part - chunk) & ((1 << lg) - 1))) * S - 1;
          continue;
        }
        if (j2 < 0 || j2 >= J2 || j3 < 0 || j3 >= J3) continue;
        const long long p = l + (v - base);
        const int4 h = t.pt_hdr[p];
        const float2 *w = a.W + p * a.SJ;
        float2 wo = D > 1 ? w[J1 + j2] : make_float2(1.f, 0.f);
        if (D > 2) {
          const float2 w3 = w[J1 + J2 + j3];
          wo = REAL ? make_float2(wo.x * w3.x, 0.f) : cmul(wo, w3);
        }
        for (int m = 0; m < NC; m++) {
          if (c + m * cw >= a.C) break;
          float2 f = fm[(long long)h.y * a.C + c + m * cw];
          if (a.phase) f = cmulc(make_float2(__int_as_float(h.z), __int_as_float(h.w)), f);
          if (D > 1) f = detail::cw_mul<REAL>(wo, f);
          for (int k = 0; k < PT_X; k++) {
            const int j1 = x + k - h.x + (ps ? K1 : 0);
            if (j1 >= 0 && j1 < J1) detail::cmac_conj<REAL>(acc[m * PT_X + k], w[j1], f);
          }
        }
      }
      base += n;
    }
  }
}

template <int D, int CW, int NC, bool REAL>
__global__ void __launch_bounds__(PT_THREADS, D == 3 ? 5 : NC <= 2 ? 8 : 6)
    spread_points_kernel(const __grid_constant__ InterpArgs a, const __grid_constant__ Tiling t,
                         PtTile pt, PtSmem sm, const int *__restrict__ bin_start,
                         const float2 *__restrict__ fm, float2 *__restrict__ ck) {
  using Sh = PtShape<CW>;
  constexpr int LB = Sh::LB, GL = Sh::GL, NGRP = Sh::NGRP, S = Sh::S, LS = Sh::LS, X = PT_X;
  constexpr int BX = PtBrick<D, LB>::BX, BY = PtBrick<D, LB>::BY, BZ = PtBrick<D, LB>::BZ;
  constexpr unsigned FULLM = 0xffffffffu;
  extern __shared__ __align__(16) unsigned char smem[];
  const Geom &g = a.g;
  const int J1 = g.J[0], J2 = D > 1 ? g.J[1] : 1, J3 = D > 2 ? g.J[2] : 1;
  const int K1 = g.K[0], K2 = D > 1 ? g.K[1] : 1, K3 = D > 2 ? g.K[2] : 1;
  const int grp = threadIdx.x / GL, gl = threadIdx.x % GL;
  const int blk = gl / CW, cl = gl % CW;
  unsigned char *gsm = smem + (size_t)grp * sm.bytes;
  int *lo = reinterpret_cast<int *>(gsm);   // [ne] first position minus running count
  int *cum = lo + sm.ne;                    // [ne + 1] running counts
  float2 *rec = reinterpret_cast<float2 *>(gsm + sm.off_rec);
  float2 *sf = reinterpret_cast<float2 *>(gsm + sm.off_f);
  int4 *sd = reinterpret_cast<int4 *>(gsm + sm.off_d);
  float2 *sph = reinterpret_cast<float2 *>(sd + S);  // phases (column chunks of 8 and more)
  // the task: part of base tile tk.x, split G = 2^lg: 1/G of its bricks with G
  // groups each, or (G > NGRP) one brick shared by G / NGRP CTAs
  const int4 tk = t.pt_task[blockIdx.x];
  constexpr int LN = NGRP == 4 ? 2 : NGRP == 8 ? 3 : NGRP == 16 ? 4 : 5;
  static_assert(1 << LN == NGRP, "groups per CTA");
  const int lg = tk.y >> 16, G = 1 << lg, ts = tk.y & 0xffff;
  const int brick = lg <= LN ? ts * (NGRP >> lg) + (grp >> lg) : ts >> (lg - LN);
  const int part = lg <= LN ? grp & (G - 1) : (ts & ((G >> LN) - 1)) * NGRP + grp;
  int r = tk.x;
  const int t1 = r % pt.nt1;
  r /= pt.nt1;
  const int t2 = r % pt.nt2;
  r /= pt.nt2;
  const int t3 = r % pt.nt3;
  const int slice = r / pt.nt3;
  const int X0 = (t1 * pt.W + brick % pt.W) * (BX * X);
  const int Y0 = (t2 * pt.R2 + brick / pt.W % pt.R2) * BY;
  const int Z0 = (t3 * pt.R3 + brick / (pt.W * pt.R2)) * BZ;
  const bool brick_on = X0 < K1 && Y0 < K2 && Z0 < K3;
  const int *bs = bin_start + (long long)slice * t.nbins;
  // this lane's block
  const int bx = blk % BX * X, by = blk / BX % BY, bz = blk / (BX * BY);
  const int C = a.C, c0 = blockIdx.y * CW * NC;

  float2 acc[NC][X];
#pragma unroll
  for (int n = 0; n < NC; n++)
#pragma unroll
    for (int k = 0; k < X; k++) acc[n][k] = make_float2(0.f, 0.f);
  // the records' padding stays zero
  for (int i = gl; i < S * sm.rs; i += GL) rec[i] = make_float2(0.f, 0.f);
  const int SJ = a.SJ;
  const bool pairs = ((J1 | (D > 1 ? J2 : 0) | (D > 2 ? J3 : 0)) & 1) == 0;
  const int nq2 = BY + J2 - 1, nq = nq2 * (BZ + J3 - 1);
  const int ci = gl / LS, sub = gl % LS;  // the staged sample this lane copies, and its share
  // pass 0: the tap rows' bins up to the brick's end; pass 1 (tiles that start
  // within J1 - 1 points of the grid's start, of which there may be several: a tile
  // is 8 points wide or more): their bins before 0, at the end of the periodic row
  const int npass = t1 * pt.W * (BX * X) < J1 - 1 ? 2 : 1;
  for (int ps = 0; ps < npass; ps++) {
    int total = 0;
    for (int e0 = 0; e0 < nq; e0 += GL) {
      const int e = e0 + gl;
      const int y = Y0 - J2 + 1 + e % nq2, z = Z0 - J3 + 1 + e / nq2;
      int l = 0, n = 0;
      if (e < nq && brick_on && y < K2 && z < K3) {
        const int *row = bs + ((z < 0 ? z + K3 : z) * K2 + (y < 0 ? y + K2 : y)) * K1;
        const int u = X0 - J1 + 1;
        if (ps == 0) {
          l = __ldg(row + max(u, 0));
          n = __ldg(row + min(X0 + BX * X, K1)) - l;
        } else if (u < 0) {
          l = __ldg(row + u + K1);
          n = __ldg(row + K1) - l;
        }
      }
      int inc = n;
#pragma unroll
      for (int o = 1; o < GL; o <<= 1) {
        const int v = __shfl_up_sync(FULLM, inc, o, GL);
        if (gl >= o) inc += v;
      }
      if (e < nq) {
        cum[e] = total + inc - n;
        lo[e] = l - (total + inc - n);
      }
      total += __shfl_sync(FULLM, inc, GL - 1, GL);
    }
    __syncwarp();
    // chunks part, part + G, ... of S samples; the warp's groups in step.  The
    // headers of the next chunk are on their way while a chunk is summed.
    const int nch = (total + S - 1) / S;
    const int trips = __reduce_max_sync(FULLM, (nch - part + G - 1) >> lg);
    int p = 0, e = 0;
    int4 h = make_int4(0, 0, 0, 0);
    auto header = [&](int it) {
      const int v = (part + it * G) * S + ci;
      if (v < total) {
        e = 0;  // the last run that starts at or before v
        for (int step = 1 << (31 - __clz(nq)); step > 0; step >>= 1)
          if (e + step < nq && cum[e + step] <= v) e += step;
        p = lo[e] + v;
        h = __ldg(t.pt_hdr + p);
      }
    };
    header(0);
    for (int it = 0; it < trips; it++) {
      const int n = min(S, total - (part + it * G) * S);  // <= 0: this group is done
      if (ci < n) {
        const float2 *w = a.W + (long long)p * SJ;
        float2 *d = rec + ci * sm.rs;
        if (pairs) {
          const float4 *w4 = reinterpret_cast<const float4 *>(w);
          float4 *d4 = reinterpret_cast<float4 *>(d);
          for (int k = sub; k < J1 / 2; k += LS) d4[2 + k] = __ldg(w4 + k);
          if (D > 1)
            for (int k = sub; k < J2 / 2; k += LS) d4[sm.o2 / 2 + k] = __ldg(w4 + J1 / 2 + k);
          if (D > 2)
            for (int k = sub; k < J3 / 2; k += LS)
              d4[sm.o3 / 2 + k] = __ldg(w4 + (J1 + J2) / 2 + k);
        } else {
          for (int k = sub; k < J1; k += LS) d[4 + k] = __ldg(w + k);
          if (D > 1)
            for (int k = sub; k < J2; k += LS) d[sm.o2 + k] = __ldg(w + J1 + k);
          if (D > 2)
            for (int k = sub; k < J3; k += LS) d[sm.o3 + k] = __ldg(w + J1 + J2 + k);
        }
        if constexpr (CW * NC < 8) {
          const float2 ph = make_float2(__int_as_float(h.z), __int_as_float(h.w));
          const float2 *f = fm + (long long)h.y * C + c0;
#pragma unroll
          for (int c = 0; c < CW * NC; c++)
            if (c % LS == sub) {
              const float2 v2 = c0 + c < C ? __ldg(f + c) : make_float2(0.f, 0.f);
              sf[ci * (CW * NC) + c] = a.phase ? cmulc(ph, v2) : v2;
            }
        }
        // first tap relative to the brick (after 4 pad entries), tap row and plane
        if (sub == 0) {
          sd[ci] = make_int4(4 + X0 - h.x + (ps ? K1 : 0), e % nq2 | e / nq2 << 16, h.y, 0);
          if (CW * NC >= 8) sph[ci] = make_float2(__int_as_float(h.z), __int_as_float(h.w));
        }
      }
      __syncwarp();
      if constexpr (CW * NC >= 8) {
        // the chunk's columns, the group's lanes along them, four loads in flight
        constexpr int CN = CW * NC, U = 4;
        for (int i0 = gl; i0 < n * CN; i0 += U * GL) {
          float2 v2[U];
#pragma unroll
          for (int u = 0; u < U; u++) {
            const int i = i0 + u * GL, j = i / CN, c = i % CN;
            v2[u] = make_float2(0.f, 0.f);
            if (i < n * CN && c0 + c < C) v2[u] = __ldg(fm + (long long)sd[j].z * C + c0 + c);
          }
#pragma unroll
          for (int u = 0; u < U; u++) {
            const int i = i0 + u * GL;
            if (i < n * CN) sf[i] = a.phase ? cmulc(sph[i / CN], v2[u]) : v2[u];
          }
        }
        __syncwarp();
      }
      header(it + 1);
      for (int j = 0; j < n; j++) {
        const int4 hj = sd[j];
        const int o = hj.x + bx;  // record entry of this block's first point
        const int j2 = by + J2 - 1 - (hj.y & 0xffff), j3 = bz + J3 - 1 - (hj.y >> 16);
        const bool ok = (D < 2 || (unsigned)j2 < (unsigned)J2) &&
                        (D < 3 || (unsigned)j3 < (unsigned)J3) &&
                        (unsigned)(o - 1) < (unsigned)(J1 + 3);
        if (ok) {
          const float2 *w = rec + j * sm.rs;
          float2 wo = make_float2(1.f, 0.f);
          if (D > 1) wo = w[sm.o2 + j2];
          if (D > 2) {
            const float2 w3 = w[sm.o3 + j3];
            wo = REAL ? make_float2(wo.x * w3.x, 0.f) : cmul(wo, w3);
          }
          float2 fv[NC];
#pragma unroll
          for (int m = 0; m < NC; m++) {
            fv[m] = sf[j * (CW * NC) + m * CW + cl];
            if (D > 1) fv[m] = detail::cw_mul<REAL>(wo, fv[m]);
          }
#pragma unroll
          for (int k = 0; k < X; k++) {
            const float2 w1 = w[o + k];
#pragma unroll
            for (int m = 0; m < NC; m++) detail::cmac_conj<REAL>(acc[m][k], w1, fv[m]);
          }
        }
      }
      __syncwarp();
    }
  }
  // A block's four points take the zeros beside the taps as well, which would make NaN
  // of an infinite or NaN product.  Such a product never leaves a sum finite.
  {
    float chk[X] = {};  // 0 x of any sum: NaN where one is not finite; four short chains
#pragma unroll
    for (int m = 0; m < NC; m++)
#pragma unroll
      for (int k = 0; k < X; k++)
        chk[k] = fmaf(0.f, acc[m][k].x, fmaf(0.f, acc[m][k].y, chk[k]));
    static_assert(X == 4, "sums of a block");
    const float bad = (chk[0] + chk[1]) + (chk[2] + chk[3]);
    if (__builtin_expect(bad != 0.f, 0)) {
      float2 again[NC * X];
      points_redo<D, NC, REAL>(a, t, bin_start, fm, slice, X0, Y0, Z0, BX * X, BY, BZ, part, lg, S,
                               X0 + bx, Y0 + by, Z0 + bz, c0 + cl, CW, again);
#pragma unroll
      for (int m = 0; m < NC; m++)
#pragma unroll
        for (int k = 0; k < X; k++) acc[m][k] = again[m * X + k];
    }
  }
  // sum a brick's groups in order: those of this CTA, then those of the CTAs that
  // share it
  if (lg > 0) {
    __syncthreads();
    float2 *red = reinterpret_cast<float2 *>(smem);  // [NGRP][NC X][GL]
#pragma unroll
    for (int m = 0; m < NC; m++)
#pragma unroll
      for (int k = 0; k < X; k++) red[(grp * (NC * X) + m * X + k) * GL + gl] = acc[m][k];
    __syncthreads();
    const int Gc = min(G, NGRP);  // groups of a brick in this CTA
    if ((grp & (Gc - 1)) == 0)
      for (int q = 1; q < Gc; q++)
#pragma unroll
        for (int m = 0; m < NC; m++)
#pragma unroll
          for (int k = 0; k < X; k++) {
            const float2 w = red[((grp + q) * (NC * X) + m * X + k) * GL + gl];
            acc[m][k].x += w.x;
            acc[m][k].y += w.y;
          }
    if (G > NGRP) {
      // this CTA's sum of the brick to its slot; the last CTA adds the slots
      const int nc = G >> LN;
      constexpr int NV = NC * X * GL;
      float2 *slot = t.pt_scratch + ((size_t)blockIdx.y * t.pt_slots + tk.z) * NV;
      if (grp == 0)
#pragma unroll
        for (int m = 0; m < NC; m++)
#pragma unroll
          for (int k = 0; k < X; k++) slot[(m * X + k) * GL + gl] = acc[m][k];
      __shared__ int last;
      __threadfence();
      __syncthreads();
      if (threadIdx.x == 0) {
        // (counts round: zero again once every CTA has counted, whatever launch it is of)
        int *c = t.pt_count + (size_t)blockIdx.y * t.pt_slots + tk.w;
        last = atomicInc(reinterpret_cast<unsigned *>(c), (unsigned)nc - 1u) == (unsigned)nc - 1u;
      }
      __syncthreads();
      if (!last || grp) return;
      __threadfence();
      const float2 *s0 = t.pt_scratch + ((size_t)blockIdx.y * t.pt_slots + tk.w) * NV;
#pragma unroll
      for (int m = 0; m < NC; m++)
#pragma unroll
        for (int k = 0; k < X; k++) acc[m][k] = make_float2(0.f, 0.f);
      for (int q = 0; q < nc; q++)
#pragma unroll
        for (int m = 0; m < NC; m++)
#pragma unroll
          for (int k = 0; k < X; k++) {
            const float2 w = __ldcg(s0 + (size_t)q * NV + (m * X + k) * GL + gl);
            acc[m][k].x += w.x;
            acc[m][k].y += w.y;
          }
    }
  }
  const int x = X0 + bx, y = Y0 + by, z = Z0 + bz;
  if ((lg <= LN && part) || grp % min(G, NGRP) || x >= K1 || y >= K2 || z >= K3) return;
  long long pt0 = x;
  if (D > 1) pt0 += (long long)y * K1;
  if (D > 2) pt0 += (long long)z * K1 * K2;
  float2 *out = ck + (long long)slice * a.grid_elems + pt0 * C + c0 + cl;
#pragma unroll
  for (int m = 0; m < NC; m++)
    if (c0 + m * CW + cl < C)
#pragma unroll
      for (int k = 0; k < X; k++)
        if (x + k < K1) out[(long long)k * C + m * CW] = acc[m][k];
}

template <class F>
cudaError_t pt_by_shape(int points, F &&f) {
  using std::integral_constant;
#define PT_CASE(CW, NC) \
  case CW * 8 + NC: return f(integral_constant<int, CW>{}, integral_constant<int, NC>{});
  switch (points) {
    PT_CASE(1, 1)
    PT_CASE(1, 2)
    PT_CASE(1, 3)
    PT_CASE(1, 4)
    PT_CASE(2, 3)
    PT_CASE(2, 4)
    PT_CASE(4, 3)
    PT_CASE(4, 4)
    PT_CASE(8, 3)
    PT_CASE(8, 4)
    default: return cudaErrorInvalidValue;
  }
#undef PT_CASE
}

// dynamic shared memory of a CTA: the groups' stages, or the split's sums
size_t pt_bytes(const Geom &g, const PtTile &pt, int cw, int nc) {
  const size_t stage = (size_t)(PT_THREADS / (cw * pt_lb(cw))) * pt_smem(g, pt, cw, nc).bytes;
  return std::max(stage, (size_t)PT_THREADS * nc * PT_X * sizeof(float2));
}

}  // namespace

// Column lanes and columns per lane, 8 CW + NC: the columns of a lane share
// its walk, its index arithmetic and its tap loads; the smallest chunk that
// holds the columns, chunks of 24 or 32 beyond (the one with fewer idle lanes).
int points_shape(int C) {
  auto code = [](int cw, int nc) { return cw * 8 + nc; };
  if (C <= 4) return code(1, C < 1 ? 1 : C);
  if (C <= 8) return code(2, C <= 6 ? 3 : 4);
  if (C <= 16) return code(4, C <= 12 ? 3 : 4);
  return (C + 23) / 24 * 24 < (C + 31) / 32 * 32 ? code(8, 3) : code(8, 4);
}

long long points_tiles(const InterpArgs &a, int shape, int nslice) {
  const PtTile t = pt_tile(a.g, shape / 8);
  if (pt_bytes(a.g, t, shape / 8, shape % 8) > 200 * 1024) return 0;
  return (long long)t.nt1 * t.nt2 * t.nt3 * nslice;
}

int points_cta_log2(int shape) {
  int l = 0;
  while ((2 << l) * (shape / 8) * pt_lb(shape / 8) <= PT_THREADS) l++;
  return l;
}

size_t points_slot_bytes(int shape) {
  return (size_t)(shape / 8) * pt_lb(shape / 8) * (shape % 8) * PT_X * sizeof(float2);
}

int points_chunks(int shape, int C) {
  const int n = (shape / 8) * (shape % 8);
  return (C + n - 1) / n;
}

void points_tile_extent(const InterpArgs &a, int shape, int *ext, int *n) {
  const PtTile t = pt_tile(a.g, shape / 8);
  ext[0] = t.W * t.bx;
  ext[1] = t.R2 * t.by;
  ext[2] = t.R3 * t.bz;
  n[0] = t.nt1;
  n[1] = t.nt2;
  n[2] = t.nt3;
}

cudaError_t launch_points_count(const InterpArgs &a, const Tiling &t, int shape, int nslice,
                                const int *bin_start, int *most, int4 *hdr, cudaStream_t st) {
  const PtTile pt = pt_tile(a.g, shape / 8);
  const int ngrp = PT_THREADS / (shape / 8 * pt_lb(shape / 8));
  const long long n = points_tiles(a, shape, nslice);
  point_count_kernel<<<(unsigned)n, 128, 0, st>>>(a, t, pt, ngrp, bin_start, n, most);
  if (a.Mtot > 0)
    point_header_kernel<<<(unsigned)((a.Mtot + 255) / 256), 256, 0, st>>>(a, hdr);
  return cudaGetLastError();
}

int points_split(const InterpArgs &a, int shape, int most, long long ntile) {
  const int lc = points_cta_log2(shape);
  int l = 0;
  // few tiles: split them all until there are two CTAs per SM
  while (l < lc && (ntile * points_chunks(shape, a.C) << l) < 296) l++;
  while (l < lc + PT_SHARE && (most >> l) > pt_visits(a.g.D)) l++;
  return l;
}

cudaError_t launch_spread_points(const InterpArgs &a, const Tiling &t, const int *bin_start,
                                 const float2 *fm, float2 *ck, cudaStream_t st) {
  if (t.n_pt_task == 0) return cudaSuccess;
  return pt_by_shape(t.points, [&](auto w, auto v) -> cudaError_t {
    constexpr int CW = decltype(w)::value, NC = decltype(v)::value;
    const PtTile pt = pt_tile(a.g, CW);
    const PtSmem sm = pt_smem(a.g, pt, CW, NC);
    const size_t bytes = pt_bytes(a.g, pt, CW, NC);
    const dim3 grid((unsigned)t.n_pt_task, (unsigned)points_chunks(t.points, a.C));
    auto go = [&](auto kern) -> cudaError_t {
      cudaError_t e =
          cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
      if (e != cudaSuccess) return e;
      kern<<<grid, PT_THREADS, bytes, st>>>(a, t, pt, sm, bin_start, fm, ck);
      return cudaGetLastError();
    };
    switch (a.g.D) {
      case 1:
        return a.real_tab ? go(spread_points_kernel<1, CW, NC, true>)
                          : go(spread_points_kernel<1, CW, NC, false>);
      case 2:
        return a.real_tab ? go(spread_points_kernel<2, CW, NC, true>)
                          : go(spread_points_kernel<2, CW, NC, false>);
      default:
        return a.real_tab ? go(spread_points_kernel<3, CW, NC, true>)
                          : go(spread_points_kernel<3, CW, NC, false>);
    }
  });
}

}  // namespace mirt
