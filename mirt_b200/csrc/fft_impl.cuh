// fft_impl.cuh -- batched DFT passes of the NUFFT's oversampled FFT (see fft.cuh),
// included by the translation units that instantiate the lengths (fft.cu, fft_l*.cu).
//
// A pass transforms lines of length n = R1 * R2 in two radix stages (the
// four-step factorisation): with k = R2 k1 + q and p = p1 + R1 p2,
//   X[p1 + R1 p2] = sum_q W_R2^{p2 q} W_n^{p1 q} sum_k1 W_R1^{p1 k1} x[R2 k1 + q].
// Stage 1 loads the R1 elements of one (line, q) from global memory into
// registers, runs the radix-R1 DFT, multiplies by the twiddles W_n^{p1 q} and
// stores to shared memory; stage 2 reads the R2 values of one (line, p1),
// runs the radix-R2 DFT and stores the outputs to global memory.  Every
// element is read from global memory once and written once, and every read of
// a line precedes the block barrier that precedes its writes, so the passes
// along dimensions >= 2 run in place.
//
// A line's elements are vectors of vw consecutive complex values (coils, or
// consecutive grid points of the faster dimensions); lane v of a group serves
// element v of the vector, so every global access of a warp is a run of
// consecutive complex values and every shared-memory access is conflict-free
// (rows padded when vw < 16).
//
// Zero padding and crop: the forward passes read only the nin < n input
// elements that hold data; when nin <= n/2 the radix-R1 stage drops its first
// decimation-in-frequency butterfly level (half its inputs are zero).  The
// adjoint passes write only the nout outputs the crop keeps; when nout <= n/2
// the radix-R2 stage forms only the first half of its outputs.
//
// In-register DFTs: recursive radix-4/2 decimation in time with the twiddle
// constants cos(2 pi e/R), sin(2 pi e/R) evaluated by the compiler from their
// Taylor series in FP64; the pass twiddles W_n^{p1 q} come from an FP64-built
// table.  Arithmetic is FP32.
#pragma once
#include <algorithm>
#include <type_traits>
#include <utility>

#include "common.cuh"
#include "fft.cuh"

namespace mirt {
namespace fftk {

constexpr int kThreads = 256;
constexpr int kMaxLpb = 32;

// ---- compile-time twiddle constants ---------------------------------------
constexpr double kTwoPi = 6.283185307179586476925286766559;

__host__ __device__ constexpr double ct_cos(double x) {
  double s = 1.0, t = 1.0;
  for (int k = 1; k <= 24; k++) {
    t = -t * x * x / ((2.0 * k - 1.0) * (2.0 * k));
    s += t;
  }
  return s;
}

__host__ __device__ constexpr double ct_sin(double x) {
  double s = x, t = x;
  for (int k = 1; k <= 24; k++) {
    t = -t * x * x / ((2.0 * k) * (2.0 * k + 1.0));
    s += t;
  }
  return s;
}

// 2 pi e / R with e reduced into (-R/2, R/2], so |angle| <= pi
template <int R, int E>
struct Angle {
  static constexpr int e0 = ((E % R) + R) % R;
  static constexpr int e = 2 * e0 > R ? e0 - R : e0;
  static constexpr double value = kTwoPi * e / R;
};

__device__ __forceinline__ float2 cadd(float2 a, float2 b) {
  return make_float2(a.x + b.x, a.y + b.y);
}
__device__ __forceinline__ float2 csub(float2 a, float2 b) {
  return make_float2(a.x - b.x, a.y - b.y);
}

// v * W_R^E with W_R = exp(-2 pi i / R) (forward) or exp(+2 pi i / R) (INV)
template <int R, int E, bool INV>
__device__ __forceinline__ float2 twmul(float2 v) {
  constexpr int e = ((E % R) + R) % R;
  if constexpr (e == 0) {
    return v;
  } else if constexpr (2 * e == R) {
    return make_float2(-v.x, -v.y);
  } else if constexpr (4 * e == R) {  // -i (forward), +i (inverse)
    return INV ? make_float2(-v.y, v.x) : make_float2(v.y, -v.x);
  } else if constexpr (4 * e == 3 * R) {  // +i (forward), -i (inverse)
    return INV ? make_float2(v.y, -v.x) : make_float2(-v.y, v.x);
  } else {
    constexpr float c = (float)ct_cos(Angle<R, E>::value);
    constexpr float s0 = (float)ct_sin(Angle<R, E>::value);
    constexpr float s = INV ? s0 : -s0;
    return make_float2(__fmaf_rn(v.x, c, -__fmul_rn(v.y, s)), __fmaf_rn(v.x, s, __fmul_rn(v.y, c)));
  }
}

// v * cos(2 pi E / R), v * sin(2 pi E / R)
template <int R, int E>
__device__ __forceinline__ float2 cosmul_add(float2 v, float2 acc) {
  constexpr float c = (float)ct_cos(Angle<R, E>::value);
  return make_float2(__fmaf_rn(c, v.x, acc.x), __fmaf_rn(c, v.y, acc.y));
}
template <int R, int E>
__device__ __forceinline__ float2 sinmul_add(float2 v, float2 acc) {
  constexpr float c = (float)ct_sin(Angle<R, E>::value);
  return make_float2(__fmaf_rn(c, v.x, acc.x), __fmaf_rn(c, v.y, acc.y));
}

// In-place DFT of R values in natural order.  R = A * B: A DFTs of length B on
// the stride-A subsequences, twiddles W_R^{a k1}, then B DFTs of length A.  Odd
// R (3, 5, 7, 9 as 3 * 3): X[m] = x[0] + sum_k cos(2 pi m k / R) (x[k] + x[R-k])
// -+ i sum_k sin(2 pi m k / R) (x[k] - x[R-k]), k = 1 .. (R-1)/2.
template <int R, bool INV>
struct Dft {
  static __device__ __forceinline__ void run(float2 *x) {
    if constexpr (R == 1) {
    } else if constexpr (R == 3 || R == 5 || R == 7) {
      constexpr int H = (R - 1) / 2;
      float2 a[H], b[H];
      sfor<H>([&](auto k) {
        a[k] = cadd(x[k + 1], x[R - 1 - k]);
        b[k] = csub(x[k + 1], x[R - 1 - k]);
      });
      const float2 x0 = x[0];
      sfor<H>([&](auto k) { x[0] = cadd(x[0], a[k]); });
      sfor<H>([&](auto m) {
        constexpr int M = decltype(m)::value + 1;
        float2 c = x0, s = make_float2(0.f, 0.f);
        sfor<H>([&](auto k) {
          constexpr int E = M * (decltype(k)::value + 1);
          c = cosmul_add<R, E>(a[k], c);
          s = sinmul_add<R, E>(b[k], s);
        });
        // c -+ i s
        const float2 lo = make_float2(c.x + s.y, c.y - s.x), hi = make_float2(c.x - s.y, c.y + s.x);
        x[M] = INV ? hi : lo;
        x[R - M] = INV ? lo : hi;
      });
    } else if constexpr (R == 2) {
      const float2 a = x[0], b = x[1];
      x[0] = cadd(a, b);
      x[1] = csub(a, b);
    } else if constexpr (R == 4) {
      const float2 t0 = cadd(x[0], x[2]), t1 = csub(x[0], x[2]);
      const float2 t2 = cadd(x[1], x[3]), t3 = twmul<4, 1, INV>(csub(x[1], x[3]));
      x[0] = cadd(t0, t2);
      x[2] = csub(t0, t2);
      x[1] = cadd(t1, t3);
      x[3] = csub(t1, t3);
    } else {
      constexpr int A = R % 2 ? 3 : (R % 16 == 0 || (R % 4 == 0 && R != 8)) ? 4 : 2;
      constexpr int B = R / A;
      float2 y[A][B];
      sfor<A>([&](auto a) { sfor<B>([&](auto b) { y[a][b] = x[A * b + a]; }); });
      sfor<A>([&](auto a) { Dft<B, INV>::run(y[a]); });
      sfor<A>([&](auto a) {
        sfor<B>([&](auto k) {
          y[a][k] = twmul<R, decltype(a)::value * decltype(k)::value, INV>(y[a][k]);
        });
      });
      sfor<B>([&](auto k1) {
        float2 z[A];
        sfor<A>([&](auto a) { z[a] = y[a][k1]; });
        Dft<A, INV>::run(z);
        sfor<A>([&](auto k2) { x[k1 + B * k2] = z[k2]; });
      });
    }
  }
};

// DFT of R values whose upper half is zero: X[2m] = DFT_{R/2}(x)[m],
// X[2m+1] = DFT_{R/2}(x[j] W_R^j)[m].
template <int R, bool INV>
__device__ __forceinline__ void dft_half_in(float2 *x) {
  constexpr int H = R / 2;
  float2 a[H], b[H];
  sfor<H>([&](auto j) {
    a[j] = x[j];
    b[j] = twmul<R, decltype(j)::value, INV>(x[j]);
  });
  Dft<H, INV>::run(a);
  Dft<H, INV>::run(b);
  sfor<H>([&](auto k) {
    x[2 * k] = a[k];
    x[2 * k + 1] = b[k];
  });
}

// The first R/2 outputs of a DFT of R values: X[k] = E[k] + W_R^k O[k] (E, O the
// DFTs of the even and odd samples).
template <int R, bool INV>
__device__ __forceinline__ void dft_half_out(float2 *x) {
  constexpr int H = R / 2;
  float2 e[H], o[H];
  sfor<H>([&](auto j) {
    e[j] = x[2 * j];
    o[j] = x[2 * j + 1];
  });
  Dft<H, INV>::run(e);
  Dft<H, INV>::run(o);
  sfor<H>([&](auto k) { x[k] = cadd(e[k], twmul<R, decltype(k)::value, INV>(o[k])); });
}

// ---- the pass kernel ---------------------------------------------------------
// PRUNE: forward with nin <= n/2, or inverse with nout <= n/2.  VW: the vector
// width at compile time (8 or 16) with the element counts exactly the transform's
// (nin = n/2 pruned or n, nout = n/2 pruned or n: no bounds tests), or 0 (any
// width and counts, read from the pass).
constexpr bool pow2(int r) { return (r & (r - 1)) == 0; }
template <int R1, int R2, bool INV, bool PRUNE, int VW>
__global__ void __launch_bounds__(kThreads, VW == 16 ? 3 : VW == 8 || !pow2(R1 * R2) ? 2 : 1)
    fft_pass_kernel(FftPass P, int lpb, int pitch_rt, int ahead) {
  constexpr bool EXACT = VW != 0;
  // the stride of the sweeps over the items: kThreads where blocks are that large, but for
  // the forward's exact form, which loses by the constant (64 slices of 512^2 x 32, two
  // passes: 1860 us with it, 1786 without; the adjoint's 1755 with it, 1782 without)
  constexpr bool FIXED = pow2(R1 * R2) && (INV || VW != 16);
  const int nthr = FIXED ? kThreads : (int)blockDim.x;
  extern __shared__ __align__(16) float2 sm[];
  __shared__ long long base_in[kMaxLpb], base_out[kMaxLpb], base_nx[kMaxLpb];
  __shared__ int snrow[kMaxLpb];
  const int vw = VW ? VW : P.vw;
  const int lvw = VW ? (VW == 16 ? 4 : 3) : __ffs(vw) - 1;
  const int pitch = VW ? R2 * VW + (VW < 16 ? VW : 0) : pitch_rt;
  const int nlines = P.nslice * P.nr2 * P.nr1 * P.nvec;
  const int g0 = blockIdx.x * lpb;
  if (threadIdx.x < lpb || (VW == 16 && ahead && threadIdx.x >= 32 && threadIdx.x < 32 + lpb)) {
    const bool nx = threadIdx.x >= 32;
    const int g = threadIdx.x & 31;
    const int gl = g0 + g + (nx ? ahead * lpb : 0);
    long long bi = -1, bo = -1;
    int row = 0;
    if (gl < nlines) {
      int o = gl / P.nvec;
      const int w = gl - o * P.nvec;
      const int r1 = o % P.nr1;
      o /= P.nr1;
      const int r2 = o % P.nr2;
      const int s = o / P.nr2;
      bi = s * P.is[0] + r2 * P.is[1] + r1 * P.is[2] + (long long)w * vw;
      bo = s * P.os[0] + r2 * P.os[1] + r1 * P.os[2] + (long long)w * vw;
      row = s * P.sn_rows + r2 * P.nr1 + r1;
    }
    if (nx) {
      base_nx[g] = bi;
    } else {
      base_in[g] = bi;
      base_out[g] = bo;
      snrow[g] = row;
    }
  }
  __syncthreads();

  // stage 1
  constexpr int KH = (PRUNE && !INV) ? R1 / 2 : R1;
  const int n1 = (lpb * R2) << lvw;
#pragma unroll 1
  for (int i = threadIdx.x; i < n1; i += nthr) {
    const int v = i & (vw - 1);
    const int q = (i >> lvw) % R2;
    const int g = (i >> lvw) / R2;
    const long long bi = base_in[g];
    if (bi < 0) continue;
    const float2 *src = P.in + bi + v;
    float2 x[R1];
    if constexpr (EXACT) {
      // element k = R2 k1 + q at a running pointer (no hoisted per-element offsets)
      const float2 *sp = src + (long long)q * P.es_in;
      const long long st = (long long)R2 * P.es_in;
#pragma unroll
      for (int k1 = 0; k1 < R1; k1++) {
        x[k1] = make_float2(0.f, 0.f);
        if (k1 < KH) {
          x[k1] = *sp;
          sp += st;
        }
      }
    } else {
#pragma unroll
      for (int k1 = 0; k1 < R1; k1++) {
        const int k = R2 * k1 + q;
        x[k1] = make_float2(0.f, 0.f);
        if (k1 < KH && k < P.nin) x[k1] = src[(long long)k * P.es_in];
      }
    }
    if (P.sn_in) {
      const float2 *sr = P.sn_in + (long long)snrow[g] * P.nin + q;
#pragma unroll
      for (int k1 = 0; k1 < KH; k1++) {
        const int k = R2 * k1 + q;
        if (EXACT || k < P.nin) x[k1] = cmul(x[k1], __ldg(sr + R2 * k1));
      }
    }
    if (P.ph_in) {
#pragma unroll
      for (int k1 = 0; k1 < KH; k1++) x[k1] = cmulc(__ldg(P.ph_in + R2 * k1 + q), x[k1]);
    }
    if constexpr (PRUNE && !INV) {
      dft_half_in<R1, INV>(x);
    } else {
      Dft<R1, INV>::run(x);
    }
    {
      // this column's twiddles, two per 16-byte load
      const float4 *tw4 = reinterpret_cast<const float4 *>(P.tw) + q * (R1 / 2);
#pragma unroll
      for (int j = 0; j < R1 / 2; j++) {
        const float4 t = __ldg(tw4 + j);
        if (j > 0 || !P.tw_unit0) x[2 * j] = cmul(x[2 * j], make_float2(t.x, t.y));
        x[2 * j + 1] = cmul(x[2 * j + 1], make_float2(t.z, t.w));
      }
    }
    float2 *d = sm + (size_t)(g * R1) * pitch + (q << lvw) + v;
#pragma unroll
    for (int p1 = 0; p1 < R1; p1++) d[p1 * pitch] = x[p1];
  }
  // The input of the block that takes this one's place, on its way to L2 meanwhile:
  // three blocks an SM keep too few loads in flight for the memory's latency (16
  // slices of 512^2 x 32: passes of 172 and 362 us -> 155 and 296, 5.4 TB/s).
  if (VW == 16 && ahead) {
    for (int i = threadIdx.x; i < lpb * P.nin; i += nthr) {
      const int g = i / P.nin;
      if (base_nx[g] >= 0)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(P.in + base_nx[g] +
                                                      (long long)(i - g * P.nin) * P.es_in));
    }
  }
  __syncthreads();

  // stage 2
  constexpr int PH = (PRUNE && INV) ? R2 / 2 : R2;
  const int n2 = (lpb * R1) << lvw;
#pragma unroll 1
  for (int i = threadIdx.x; i < n2; i += nthr) {
    const int v = i & (vw - 1);
    const int p1 = (i >> lvw) % R1;
    const int g = (i >> lvw) / R1;
    const long long bo = base_out[g];
    if (bo < 0) continue;
    float2 y[R2];
    const float2 *s = sm + (size_t)(g * R1 + p1) * pitch + v;
#pragma unroll
    for (int k2 = 0; k2 < R2; k2++) y[k2] = s[k2 << lvw];
    if constexpr (PRUNE && INV) {
      dft_half_out<R2, INV>(y);
    } else {
      Dft<R2, INV>::run(y);
    }
    float2 *dst = P.out + bo + v;
    const float2 *sr = P.sn_out ? P.sn_out + (long long)snrow[g] * P.nout : nullptr;
    if (EXACT && !sr && !P.ph_out) {
      float2 *dp = dst + (long long)p1 * P.es_out;
      const long long st = (long long)R1 * P.es_out;
#pragma unroll
      for (int p2 = 0; p2 < PH; p2++) {
        *dp = y[p2];
        dp += st;
      }
    } else {
#pragma unroll
      for (int p2 = 0; p2 < PH; p2++) {
        const int p = p1 + R1 * p2;
        if (EXACT || p < P.nout) {
          float2 val = y[p2];
          if (P.ph_out) val = cmul(val, __ldg(P.ph_out + p));
          if (sr) val = cmulc(__ldg(sr + p), val);
          dst[(long long)p * P.es_out] = val;
        }
      }
    }
  }
}

// ---- forward, spectrum, inverse ------------------------------------------------
// Stage 1 and stage 2 of the forward transform as in fft_pass_kernel (inputs
// pruned to n/2), so that thread (line, p1) holds X[p1 + R1 p2] for all p2; times
// the spectrum; then the inverse with k = p1 + R1 p2 and m = m2 + R2 m1,
//   x[m] = sum_p1 W_R1^{m1 p1} W_n^{m2 p1} sum_p2 W_R2^{m2 p2} Y[p1 + R1 p2],
// whose first radix-R2 stage stays in that thread's registers and goes back to
// the same row of shared memory, and whose radix-R1 stage forms the first half of
// its outputs (m < n/2).
template <int R1, int R2, int VW>
__global__ void __launch_bounds__(kThreads, VW == 16 ? 3 : 2)
    circulant_pass_kernel(CirculantPass P, int lpb, int pitch_rt) {
  extern __shared__ __align__(16) float2 sm[];
  const int vw = VW ? VW : P.vw;
  const int lvw = VW ? (VW == 16 ? 4 : 3) : __ffs(vw) - 1;
  const int pitch = VW ? R2 * VW + (VW < 16 ? VW : 0) : pitch_rt;
  const int nlines = P.nslice * P.nvec;
  const int g0 = blockIdx.x * lpb;
  auto line = [&](int g, int v) -> float2 * {
    const int gl = g0 + g;
    if (gl >= nlines) return nullptr;
    const int s = gl / P.nvec, w = gl - s * P.nvec;
    return P.io + s * P.slice + ((long long)w << lvw) + v;
  };
  // stage 1
  const int n1 = (lpb * R2) << lvw;
#pragma unroll 1
  for (int i = threadIdx.x; i < n1; i += blockDim.x) {
    const int v = i & (vw - 1), q = (i >> lvw) % R2, g = (i >> lvw) / R2;
    const float2 *sp = line(g, v);
    if (!sp) continue;
    float2 x[R1];
    sp += (long long)q * P.es;
    const long long st = (long long)R2 * P.es;
#pragma unroll
    for (int k1 = 0; k1 < R1; k1++) {
      x[k1] = make_float2(0.f, 0.f);
      if (k1 < R1 / 2) {
        x[k1] = *sp;
        sp += st;
      }
    }
    dft_half_in<R1, false>(x);
    const float4 *tw4 = reinterpret_cast<const float4 *>(P.tw) + q * (R1 / 2);
#pragma unroll
    for (int j = 0; j < R1 / 2; j++) {
      const float4 t = __ldg(tw4 + j);
      if (j > 0) x[2 * j] = cmul(x[2 * j], make_float2(t.x, t.y));
      x[2 * j + 1] = cmul(x[2 * j + 1], make_float2(t.z, t.w));
    }
    float2 *d = sm + (size_t)(g * R1) * pitch + (q << lvw) + v;
#pragma unroll
    for (int p1 = 0; p1 < R1; p1++) d[p1 * pitch] = x[p1];
  }
  __syncthreads();
  // stage 2, spectrum, inverse stage 1
  const int n2 = (lpb * R1) << lvw;
#pragma unroll 1
  for (int i = threadIdx.x; i < n2; i += blockDim.x) {
    const int v = i & (vw - 1), p1 = (i >> lvw) % R1, g = (i >> lvw) / R1;
    const int gl = g0 + g;
    if (gl >= nlines) continue;
    float2 y[R2];
    float2 *s = sm + (size_t)(g * R1 + p1) * pitch + v;
#pragma unroll
    for (int k = 0; k < R2; k++) y[k] = s[k << lvw];
    Dft<R2, false>::run(y);
    const int sl = gl / P.nvec, w = gl - sl * P.nvec;
    const long long h0 = ((long long)sl * P.n + p1) * P.n1 + ((w << lvw) + v) / P.C;
    const long long hs = (long long)R1 * P.n1;
    if (P.Hr) {
      const float *h = P.Hr + h0;
#pragma unroll
      for (int k = 0; k < R2; k++) {
        const float a = P.scale * __ldg(h);
        h += hs;
        y[k] = make_float2(a * y[k].x, a * y[k].y);
      }
    } else {
      const float2 *h = P.H + h0;
#pragma unroll
      for (int k = 0; k < R2; k++) {
        const float2 a = __ldg(h);
        h += hs;
        y[k] = cmul(y[k], make_float2(P.scale * a.x, P.scale * a.y));
      }
    }
    Dft<R2, true>::run(y);
    const float2 *tw = P.tw + p1;  // conj(W_n^{m2 p1})
#pragma unroll
    for (int k = 0; k < R2; k++) s[k << lvw] = k ? cmulc(__ldg(tw + k * R1), y[k]) : y[k];
  }
  __syncthreads();
  // inverse stage 2: outputs m = m2 + R2 m1, m1 < R1 / 2
#pragma unroll 1
  for (int i = threadIdx.x; i < n1; i += blockDim.x) {
    const int v = i & (vw - 1), q = (i >> lvw) % R2, g = (i >> lvw) / R2;
    float2 *dp = line(g, v);
    if (!dp) continue;
    float2 x[R1];
    const float2 *d = sm + (size_t)(g * R1) * pitch + (q << lvw) + v;
#pragma unroll
    for (int p1 = 0; p1 < R1; p1++) x[p1] = d[p1 * pitch];
    dft_half_out<R1, true>(x);
    dp += (long long)q * P.es;
    const long long st = (long long)R2 * P.es;
#pragma unroll
    for (int m1 = 0; m1 < R1 / 2; m1++) {
      *dp = x[m1];
      dp += st;
    }
  }
}

// lines per block and the block size whose sweeps over the stages' items (lpb R2
// vw twice or once, lpb R1 vw) idle least.  Few lines: fewer per block, so that they
// lie on more SMs and a thread takes one turn (1D forward, K = 560, 124 lines: 24.9 us
// in 11 blocks of 12, 15.7 us in 31 of 4)
template <int R1, int R2>
void block_shape(int vw, int stages_r2, long long nlines, int *lpb, unsigned *threads) {
  *lpb = kThreads / ((R1 < R2 ? R1 : R2) * vw);
  const int least = 64 / ((R1 < R2 ? R1 : R2) * vw) + 1;  // two warps' items
  if (*lpb > (nlines + 147) / 148) *lpb = std::max(least, (int)((nlines + 147) / 148));
  if (*lpb < 1) *lpb = 1;
  if (*lpb > kMaxLpb) *lpb = kMaxLpb;
  const unsigned n1 = *lpb * R2 * vw, n2 = *lpb * R1 * vw;
  unsigned best = ~0u;
  for (unsigned t = kThreads; t >= 96; t -= 32) {
    const unsigned work = (stages_r2 * ((n1 + t - 1) / t) + (n2 + t - 1) / t) * t;
    if (work < best) {
      best = work;
      *threads = t;
    }
  }
}

template <int R1, int R2>
cudaError_t launch_c(const CirculantPass &P, cudaStream_t st) {
  int lpb = 1;
  unsigned threads = kThreads;
  const long long nlines = (long long)P.nslice * P.nvec;
  if (nlines <= 0) return cudaSuccess;
  block_shape<R1, R2>(P.vw, 2, nlines, &lpb, &threads);
  const int pitch = R2 * P.vw + (P.vw < 16 ? P.vw : 0);
  const size_t smem = (size_t)lpb * R1 * pitch * sizeof(float2);
  const unsigned grid = (unsigned)((nlines + lpb - 1) / lpb);
  auto kern = P.vw == 16 ? circulant_pass_kernel<R1, R2, 16> : circulant_pass_kernel<R1, R2, 0>;
  cudaError_t e =
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  kern<<<grid, threads, smem, st>>>(P, lpb, pitch);
  return cudaGetLastError();
}

// EXTRA: a length off the powers of two; the exact forms only where pruned
// (K >= 2 N, the usual oversampling), the general form elsewhere
template <int R1, int R2, bool EXTRA = false>
cudaError_t launch_r(const FftPass &P, cudaStream_t st) {
  const int vw = P.vw;
  int lpb = 1;
  unsigned threads = kThreads;
  const long long nlines = (long long)P.nslice * P.nr2 * P.nr1 * P.nvec;
  if (nlines <= 0) return cudaSuccess;
  block_shape<R1, R2>(vw, 1, nlines, &lpb, &threads);
  if (!EXTRA) threads = kThreads;
  const int pitch = R2 * vw + (vw < 16 ? vw : 0);
  const size_t smem = (size_t)lpb * R1 * pitch * sizeof(float2);
  const unsigned grid = (unsigned)((nlines + lpb - 1) / lpb);
  const bool prune = P.inverse ? (2 * P.nout <= P.n) : (2 * P.nin <= P.n);
  // the exact forms: 16- or 8-wide vectors, inputs and outputs exactly the
  // (pruned) halves or all n
  const int hin = prune && !P.inverse ? P.n / 2 : P.n, hout = prune && P.inverse ? P.n / 2 : P.n;
  const int exact =
      (P.nin == hin && P.nout == hout && (vw == 16 || vw == 8) && (prune || !EXTRA)) ? vw : 0;
  auto pick = [&](auto kern) -> cudaError_t {
    cudaError_t e =
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    // Blocks prefetch for the block that follows them on their SM, one full chip of
    // blocks on, where 128-byte vectors lie close enough: strides of 4 MB put the 256
    // lines of a column on few L2 sets (3D, 256^3 x 8: 316 us without, 428 with).
    int ahead = 0;
    if (exact == 16 && P.es_in * (long long)sizeof(float2) <= (1 << 20)) {
      int per = 0;
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, threads, smem);
      if (e != cudaSuccess) return e;
      if (grid > 2u * 148u * per) ahead = 148 * per;
    }
    kern<<<grid, threads, smem, st>>>(P, lpb, pitch, ahead);
    return cudaGetLastError();
  };
  auto by_width = [&](auto k16, auto k8, auto k0) -> cudaError_t {
    return exact == 16 ? pick(k16) : exact == 8 ? pick(k8) : pick(k0);
  };
  auto by_prune = [&](auto inv) -> cudaError_t {
    constexpr bool INV = decltype(inv)::value;
    if (prune)
      return by_width(fft_pass_kernel<R1, R2, INV, true, 16>, fft_pass_kernel<R1, R2, INV, true, 8>,
                      fft_pass_kernel<R1, R2, INV, true, 0>);
    if constexpr (EXTRA)
      return pick(fft_pass_kernel<R1, R2, INV, false, 0>);
    else
      return by_width(fft_pass_kernel<R1, R2, INV, false, 16>,
                      fft_pass_kernel<R1, R2, INV, false, 8>,
                      fft_pass_kernel<R1, R2, INV, false, 0>);
  };
  return P.inverse ? by_prune(std::true_type{}) : by_prune(std::false_type{});
}

// the lengths off the powers of two, a third in each of three translation units
cudaError_t launch_l1(const FftPass &p, cudaStream_t st);
cudaError_t launch_l2(const FftPass &p, cudaStream_t st);
cudaError_t launch_l3(const FftPass &p, cudaStream_t st);
cudaError_t launch_c1(const CirculantPass &p, cudaStream_t st);
cudaError_t launch_c2(const CirculantPass &p, cudaStream_t st);
cudaError_t launch_c3(const CirculantPass &p, cudaStream_t st);

}  // namespace fftk
}  // namespace mirt
