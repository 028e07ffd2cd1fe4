// Instantiates the FFT passes of some lengths (pg_fftkern.cuh).
#include "pg_fftkern.cuh"

namespace pg {

const FftOps* fft_ops_7(int n) {
  switch (n) {
    case 336: return fft_ops<16, 21>();
    case 480: return fft_ops<16, 30>();
    case 512: return fft_ops<16, 32>();
    default: return nullptr;
  }
}

}  // namespace pg
