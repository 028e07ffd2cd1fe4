// Instantiates the FFT passes of some lengths (pg_fftkern.cuh).
#include "pg_fftkern.cuh"

namespace pg {

const FftOps* fft_ops_4(int n) {
  switch (n) {
    case 224: return fft_ops<16, 14>();
    case 240: return fft_ops<16, 15>();
    case 256: return fft_ops<16, 16>();
    case 416: return fft_ops<16, 26>();
    default: return nullptr;
  }
}

}  // namespace pg
