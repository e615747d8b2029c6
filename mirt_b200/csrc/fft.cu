// fft.cu -- the passes of the NUFFT's oversampled FFT (fft.cuh): transform
// lengths and their dispatch, and the forward and adjoint pass sequences.
#include "fft_impl.cuh"

#include <algorithm>
#include <cmath>

namespace mirt {
namespace {

// Transform lengths n = R1 R2.  R1 and R2 are multiples of 4 where the length
// allows it (a folded grid phase needs it, fft_fold_ok); the lengths off the powers of
// two are K = 2 N of 26 usual image sizes N between 40 and 448; others that the same
// radices would give (140, 168, 180, 196, 216, 252, 324, 392, 432, 504) are left to cuFFT.
struct FftLen {
  int n, r1, r2, unit;  // unit: the translation unit that instantiates it (0: here)
};
constexpr FftLen kLens[] = {
    {64, 8, 8, 0},    {80, 8, 10, 1},   {96, 8, 12, 1},   {100, 10, 10, 1}, {112, 8, 14, 1},
    {120, 12, 10, 1}, {128, 8, 16, 0},  {144, 12, 12, 1}, {160, 8, 20, 1},  {192, 12, 16, 1},
    {200, 20, 10, 1}, {224, 16, 14, 1},  {240, 12, 20, 2}, {256, 16, 16, 0}, {280, 20, 14, 2},
    {288, 12, 24, 2}, {320, 16, 20, 2}, {336, 24, 14, 2}, {360, 20, 18, 2}, {384, 16, 24, 2},
    {400, 20, 20, 2}, {448, 16, 28, 2}, {480, 20, 24, 3}, {512, 16, 32, 0}, {560, 20, 28, 3},
    {576, 24, 24, 3}, {640, 20, 32, 3}, {672, 24, 28, 3}, {768, 24, 32, 3}, {896, 28, 32, 3},
    {1024, 32, 32, 0}};

const FftLen *find_len(int n) {
  for (const FftLen &l : kLens)
    if (l.n == n) return &l;
  return nullptr;
}

// largest power of two dividing v, at most 16
int vec_width(long long v) {
  int w = 1;
  while (w < 16 && v % (2 * w) == 0) w *= 2;
  return w;
}

// ... for a pass of `lines` of n: 8 where few lines of 16 would take a block two turns
int pass_width(int n, long long v, long long lines) {
  const int w = vec_width(v);
  int r1 = 0, r2 = 0;
  fft_radix(n, &r1, &r2);
  return w == 16 && lines * (v / w) < 74 && 16 * std::max(r1, r2) > fftk::kThreads ? 8 : w;
}

FftPass base_pass(const NufftFft &f, int d, int s0, int s1, bool inverse) {
  FftPass p{};
  p.nslice = s1 - s0;
  p.nr1 = p.nr2 = 1;
  p.n = f.g.K[d];
  p.inverse = inverse ? 1 : 0;
  p.tw = inverse ? f.twa[d] : f.twf[d];
  p.tw_unit0 = !inverse || !f.phase_folded;  // entry p1 = 0 is 1 for every column
  const float2 *ph = (f.gp && f.gp->tab[0] && !f.phase_folded) ? f.gp->tab[d] : nullptr;
  if (inverse)
    p.ph_in = ph;
  else
    p.ph_out = ph;
  return p;
}

}  // namespace

bool fft_len_ok(int n) { return find_len(n) != nullptr; }

bool fft_fold_ok(int n) {
  const FftLen *l = find_len(n);
  return l && l->r1 % 4 == 0 && l->r2 % 4 == 0;
}

cudaError_t launch_fft_pass(const FftPass &p, cudaStream_t st) {
  if (p.vw < 1 || p.vw > 32 || (p.vw & (p.vw - 1)) || p.nr1 < 1 || p.nr2 < 1 || p.nvec < 1)
    return cudaErrorInvalidValue;
  if ((long long)p.nslice * p.nr2 * p.nr1 * p.nvec >= (1ll << 31)) return cudaErrorInvalidValue;
  const FftLen *l = find_len(p.n);
  if (!l) return cudaErrorInvalidValue;
  switch (l->unit) {
    case 1: return fftk::launch_l1(p, st);
    case 2: return fftk::launch_l2(p, st);
    case 3: return fftk::launch_l3(p, st);
    default: break;
  }
  switch (p.n) {
    case 64: return fftk::launch_r<8, 8>(p, st);
    case 128: return fftk::launch_r<8, 16>(p, st);
    case 256: return fftk::launch_r<16, 16>(p, st);
    case 512: return fftk::launch_r<16, 32>(p, st);
    case 1024: return fftk::launch_r<32, 32>(p, st);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_circulant_pass(const CirculantPass &p, cudaStream_t st) {
  const FftLen *l = find_len(p.n);
  if (!l || p.vw < 1 || p.vw > 16 || (p.vw & (p.vw - 1)) || p.nvec < 1) return cudaErrorInvalidValue;
  if ((long long)p.nslice * p.nvec >= (1ll << 31)) return cudaErrorInvalidValue;
  switch (l->unit) {
    case 1: return fftk::launch_c1(p, st);
    case 2: return fftk::launch_c2(p, st);
    case 3: return fftk::launch_c3(p, st);
    default: break;
  }
  switch (p.n) {
    case 64: return fftk::launch_c<8, 8>(p, st);
    case 128: return fftk::launch_c<8, 16>(p, st);
    case 256: return fftk::launch_c<16, 16>(p, st);
    case 512: return fftk::launch_c<16, 32>(p, st);
    case 1024: return fftk::launch_c<32, 32>(p, st);
    default: return cudaErrorInvalidValue;
  }
}

void fft_twiddles(int n, bool inverse, std::vector<float2> &tw) {
  int r1 = 0, r2 = 0;
  fft_radix(n, &r1, &r2);
  tw.clear();
  for (int q = 0; q < r2; q++)
    for (int p1 = 0; p1 < r1; p1++) {
      const double a = fftk::kTwoPi * (double)(((long long)p1 * q) % n) / n;
      tw.push_back(make_float2((float)std::cos(a), (float)(inverse ? std::sin(a) : -std::sin(a))));
    }
}

int fft_vec_width(long long v) { return vec_width(v); }

void fft_radix(int n, int *r1, int *r2) {
  const FftLen *l = find_len(n);
  *r1 = l ? l->r1 : 0;
  *r2 = l ? l->r2 : 0;
}

int fft_nufft_passes(const NufftFft &f) { return f.g.D; }

cudaError_t fft_nufft_forward(const NufftFft &f, const float2 *x, float2 *grid, int s0, int s1,
                              cudaStream_t st, const float2 *img) {
  const GlueGeom &g = f.g;
  const long long C = f.C, xs = g.npix * C, gs = g.ngrid * C;
  if (s1 <= s0 || C == 0) return cudaSuccess;
  const int N1 = g.N[0], N2 = g.N[1], N3 = g.N[2];
  const int K1 = g.K[0], K2 = g.K[1];
  float2 *gd = grid + s0 * gs;
  // dimension 1: image rows -> grid rows (times sn)
  {
    FftPass p = base_pass(f, 0, s0, s1, false);
    p.in = x + s0 * xs;
    p.out = gd;
    p.nr1 = g.D > 1 ? N2 : 1;
    p.nr2 = g.D > 2 ? N3 : 1;
    p.is[0] = xs;
    p.is[1] = (long long)N2 * N1 * C;
    p.is[2] = (long long)N1 * C;
    p.os[0] = gs;
    p.os[1] = (long long)K2 * K1 * C;
    p.os[2] = (long long)K1 * C;
    p.es_in = p.es_out = C;
    p.vw = pass_width(p.n, C, (long long)(s1 - s0) * p.nr1 * p.nr2);
    p.nvec = (int)(C / p.vw);
    p.nin = N1;
    p.nout = K1;
    p.sn_in = img ? img + s0 * g.npix : f.sn;
    p.sn_rows = img ? N2 * N3 : 0;
    cudaError_t e = launch_fft_pass(p, st);
    if (e != cudaSuccess || g.D == 1) return e;
  }
  // dimension 2, in place: the image rows of every plane n3 < N3
  {
    FftPass p = base_pass(f, 1, s0, s1, false);
    p.in = p.out = gd;
    p.nr1 = g.D > 2 ? N3 : 1;
    p.is[0] = p.os[0] = gs;
    p.is[2] = p.os[2] = (long long)K2 * K1 * C;
    p.es_in = p.es_out = (long long)K1 * C;
    p.vw = vec_width((long long)K1 * C);
    p.nvec = (int)((long long)K1 * C / p.vw);
    p.nin = N2;
    p.nout = K2;
    cudaError_t e = launch_fft_pass(p, st);
    if (e != cudaSuccess || g.D == 2) return e;
  }
  // dimension 3, in place
  {
    FftPass p = base_pass(f, 2, s0, s1, false);
    p.in = p.out = gd;
    p.is[0] = p.os[0] = gs;
    p.es_in = p.es_out = (long long)K2 * K1 * C;
    p.vw = vec_width(p.es_in);
    p.nvec = (int)(p.es_in / p.vw);
    p.nin = N3;
    p.nout = g.K[2];
    return launch_fft_pass(p, st);
  }
}

cudaError_t fft_nufft_adjoint(const NufftFft &f, float2 *grid, float2 *x, int s0, int s1,
                              cudaStream_t st) {
  const GlueGeom &g = f.g;
  const long long C = f.C, xs = g.npix * C, gs = g.ngrid * C;
  if (s1 <= s0 || C == 0) return cudaSuccess;
  const int N1 = g.N[0], N2 = g.N[1], N3 = g.N[2];
  const int K1 = g.K[0], K2 = g.K[1];
  float2 *gd = grid + s0 * gs;
  cudaError_t e = cudaSuccess;
  if (g.D > 2) {  // dimension 3, in place: planes n3 < N3 kept
    FftPass p = base_pass(f, 2, s0, s1, true);
    p.in = p.out = gd;
    p.is[0] = p.os[0] = gs;
    p.es_in = p.es_out = (long long)K2 * K1 * C;
    p.vw = vec_width(p.es_in);
    p.nvec = (int)(p.es_in / p.vw);
    p.nin = g.K[2];
    p.nout = N3;
    e = launch_fft_pass(p, st);
    if (e != cudaSuccess) return e;
  }
  if (g.D > 1) {  // dimension 2, in place: rows n2 < N2 of planes n3 < N3 kept
    FftPass p = base_pass(f, 1, s0, s1, true);
    p.in = p.out = gd;
    p.nr1 = g.D > 2 ? N3 : 1;
    p.is[0] = p.os[0] = gs;
    p.is[2] = p.os[2] = (long long)K2 * K1 * C;
    p.es_in = p.es_out = (long long)K1 * C;
    p.vw = vec_width((long long)K1 * C);
    p.nvec = (int)((long long)K1 * C / p.vw);
    p.nin = K2;
    p.nout = N2;
    e = launch_fft_pass(p, st);
    if (e != cudaSuccess) return e;
  }
  // dimension 1: grid rows -> image rows, cropped, times conj(sn)
  FftPass p = base_pass(f, 0, s0, s1, true);
  p.in = gd;
  p.out = x + s0 * xs;
  p.nr1 = g.D > 1 ? N2 : 1;
  p.nr2 = g.D > 2 ? N3 : 1;
  p.is[0] = gs;
  p.is[1] = (long long)K2 * K1 * C;
  p.is[2] = (long long)K1 * C;
  p.os[0] = xs;
  p.os[1] = (long long)N2 * N1 * C;
  p.os[2] = (long long)N1 * C;
  p.es_in = p.es_out = C;
  p.vw = pass_width(p.n, C, (long long)(s1 - s0) * p.nr1 * p.nr2);
  p.nvec = (int)(C / p.vw);
  p.nin = K1;
  p.nout = N1;
  p.sn_out = f.sn;
  return launch_fft_pass(p, st);
}

}  // namespace mirt
