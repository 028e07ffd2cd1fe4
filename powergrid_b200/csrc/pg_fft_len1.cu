// Instantiates the FFT passes of some lengths (pg_fftkern.cuh).
#include "pg_fftkern.cuh"

namespace pg {

const FftOps* fft_ops_1(int n) {
  switch (n) {
    case 80: return fft_ops<16, 5>();
    case 96: return fft_ops<16, 6>();
    case 112: return fft_ops<16, 7>();
    case 464: return fft_ops<16, 29>();
    default: return nullptr;
  }
}

}  // namespace pg
