// Instantiates the FFT passes of some lengths (pg_fftkern.cuh).
#include "pg_fftkern.cuh"

namespace pg {

const FftOps* fft_ops_3(int n) {
  switch (n) {
    case 176: return fft_ops<16, 11>();
    case 192: return fft_ops<16, 12>();
    case 208: return fft_ops<16, 13>();
    case 448: return fft_ops<16, 28>();
    default: return nullptr;
  }
}

}  // namespace pg
