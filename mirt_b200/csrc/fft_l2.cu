// fft_l2.cu -- DFT passes of lengths off the powers of two, part 2 (fft_impl.cuh).
#include "fft_impl.cuh"

namespace mirt {
namespace fftk {

cudaError_t launch_l2(const FftPass &p, cudaStream_t st) {
  switch (p.n) {
    case 240: return launch_r<12, 20, true>(p, st);
    case 280: return launch_r<20, 14, true>(p, st);
    case 288: return launch_r<12, 24, true>(p, st);
    case 320: return launch_r<16, 20, true>(p, st);
    case 336: return launch_r<24, 14, true>(p, st);
    case 360: return launch_r<20, 18, true>(p, st);
    case 384: return launch_r<16, 24, true>(p, st);
    case 400: return launch_r<20, 20, true>(p, st);
    case 448: return launch_r<16, 28, true>(p, st);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_c2(const CirculantPass &p, cudaStream_t st) {
  switch (p.n) {
    case 240: return launch_c<12, 20>(p, st);
    case 280: return launch_c<20, 14>(p, st);
    case 288: return launch_c<12, 24>(p, st);
    case 320: return launch_c<16, 20>(p, st);
    case 336: return launch_c<24, 14>(p, st);
    case 360: return launch_c<20, 18>(p, st);
    case 384: return launch_c<16, 24>(p, st);
    case 400: return launch_c<20, 20>(p, st);
    case 448: return launch_c<16, 28>(p, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace fftk
}  // namespace mirt
