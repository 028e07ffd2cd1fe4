// Instantiates the FFT passes of some lengths (pg_fftkern.cuh).
#include "pg_fftkern.cuh"

namespace pg {

const FftOps* fft_ops_5(int n) {
  switch (n) {
    case 272: return fft_ops<16, 17>();
    case 288: return fft_ops<16, 18>();
    case 384: return fft_ops<16, 24>();
    case 400: return fft_ops<16, 25>();
    default: return nullptr;
  }
}

}  // namespace pg
