// Instantiates the FFT passes of some lengths (pg_fftkern.cuh).
#include "pg_fftkern.cuh"

namespace pg {

const FftOps* fft_ops_0(int n) {
  switch (n) {
    case 16: return fft_ops<4, 4>();
    case 32: return fft_ops<8, 4>();
    case 48: return fft_ops<16, 3>();
    case 64: return fft_ops<16, 4>();
    case 496: return fft_ops<16, 31>();
    default: return nullptr;
  }
}

}  // namespace pg
