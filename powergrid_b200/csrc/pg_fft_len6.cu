// Instantiates the FFT passes of some lengths (pg_fftkern.cuh).
#include "pg_fftkern.cuh"

namespace pg {

const FftOps* fft_ops_6(int n) {
  switch (n) {
    case 304: return fft_ops<16, 19>();
    case 320: return fft_ops<16, 20>();
    case 352: return fft_ops<16, 22>();
    case 1024: return fft_ops<32, 32>();
    default: return nullptr;
  }
}

}  // namespace pg
