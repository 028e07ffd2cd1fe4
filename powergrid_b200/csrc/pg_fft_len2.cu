// Instantiates the FFT passes of some lengths (pg_fftkern.cuh).
#include "pg_fftkern.cuh"

namespace pg {

const FftOps* fft_ops_2(int n) {
  switch (n) {
    case 128: return fft_ops<16, 8>();
    case 144: return fft_ops<16, 9>();
    case 160: return fft_ops<16, 10>();
    case 368: return fft_ops<16, 23>();
    case 432: return fft_ops<16, 27>();
    default: return nullptr;
  }
}

}  // namespace pg
