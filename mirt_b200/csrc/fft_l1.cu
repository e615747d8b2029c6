// fft_l1.cu -- DFT passes of lengths off the powers of two, part 1 (fft_impl.cuh).
#include "fft_impl.cuh"

namespace mirt {
namespace fftk {

cudaError_t launch_l1(const FftPass &p, cudaStream_t st) {
  switch (p.n) {
    case 80: return launch_r<8, 10, true>(p, st);
    case 96: return launch_r<8, 12, true>(p, st);
    case 100: return launch_r<10, 10, true>(p, st);
    case 112: return launch_r<8, 14, true>(p, st);
    case 120: return launch_r<12, 10, true>(p, st);
    case 144: return launch_r<12, 12, true>(p, st);
    case 160: return launch_r<8, 20, true>(p, st);
    case 192: return launch_r<12, 16, true>(p, st);
    case 200: return launch_r<20, 10, true>(p, st);
    case 224: return launch_r<16, 14, true>(p, st);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_c1(const CirculantPass &p, cudaStream_t st) {
  switch (p.n) {
    case 80: return launch_c<8, 10>(p, st);
    case 96: return launch_c<8, 12>(p, st);
    case 100: return launch_c<10, 10>(p, st);
    case 112: return launch_c<8, 14>(p, st);
    case 120: return launch_c<12, 10>(p, st);
    case 144: return launch_c<12, 12>(p, st);
    case 160: return launch_c<8, 20>(p, st);
    case 192: return launch_c<12, 16>(p, st);
    case 200: return launch_c<20, 10>(p, st);
    case 224: return launch_c<16, 14>(p, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace fftk
}  // namespace mirt
