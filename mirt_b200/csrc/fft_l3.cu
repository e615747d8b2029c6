// fft_l3.cu -- DFT passes of lengths off the powers of two, part 3 (fft_impl.cuh).
#include "fft_impl.cuh"

namespace mirt {
namespace fftk {

cudaError_t launch_l3(const FftPass &p, cudaStream_t st) {
  switch (p.n) {
    case 480: return launch_r<20, 24, true>(p, st);
    case 560: return launch_r<20, 28, true>(p, st);
    case 576: return launch_r<24, 24, true>(p, st);
    case 640: return launch_r<20, 32, true>(p, st);
    case 672: return launch_r<24, 28, true>(p, st);
    case 768: return launch_r<24, 32, true>(p, st);
    case 896: return launch_r<28, 32, true>(p, st);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_c3(const CirculantPass &p, cudaStream_t st) {
  switch (p.n) {
    case 480: return launch_c<20, 24>(p, st);
    case 560: return launch_c<20, 28>(p, st);
    case 576: return launch_c<24, 24>(p, st);
    case 640: return launch_c<20, 32>(p, st);
    case 672: return launch_c<24, 28>(p, st);
    case 768: return launch_c<24, 32>(p, st);
    case 896: return launch_c<28, 32>(p, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace fftk
}  // namespace mirt
