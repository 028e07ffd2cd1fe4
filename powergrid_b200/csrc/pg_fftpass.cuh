// Pruned oversampled FFT passes with the NUFFT pre/post kernels fused in
// (pg_fftpass.cu), for 2-D and 3-D grids of 2N per axis with N a multiple of 8
// up to 256, or 512.
#pragma once

#include "pg_nufft.cuh"

namespace pg {

// The grids of one application: grid b = c * L + l of coil c0 + c, segment l.
struct FftBatch {
  int C = 1, L = 1, c0 = 0;
  const float2* S = nullptr;
  const float2* E = nullptr;
  // several images (NufftBatch): coil c0 + c belongs to image (c0 + c) / cgroup
  int cgroup = 0;
  uint64_t image_stride = 0, phase_stride = 0;
};

bool fftpass_supported(const NufftGeom& g);
// Scratch (complex elements) that either direction may need for a batch: half-
// transformed lines, then the images of the last inverse pass.  One buffer: an
// allocation costs some 0.34 ms whatever its size, and a new operator's first calls
// wait for it (208^2, 12 coils, L = 10, first forward and adjoint: 1.72 ms with the
// images on their own, 1.38 ms in one).
uint64_t fftpass_scratch(const NufftGeom& g, const FftBatch& b);
// Twiddle tables exp(-2 pi i k1 m2 / n) for the in-plane length (and z),
// made in double precision.
pg_status fftpass_twiddles(const NufftGeom& g, DevBuf<float2>* tw, cudaStream_t s);
// The groups of grid cells that the samples' taps reach, from their tap starts
// and segment windows [l0, l0 + K).
pg_status fftpass_support(const NufftGeom& g, uint64_t M, int L, int K, const uint2* start, const int* l0,
                          FftSupport* out, cudaStream_t s);
// scratch: fftpass_scratch elements.  grids: C * L grids out, their supported cells.
pg_status fftpass_forward(const NufftGeom& g, const FftBatch& b, const FftSupport& sup, const float2* x,
                          const float2* Wo, const float* deapf, const float2* tw, float2* scratch, float2* grids,
                          cudaStream_t s);
// Zeroes the supported cells of the batch's 3-D grids.
pg_status fftpass_clear(const NufftGeom& g, const FftBatch& b, const FftSupport& sup, float2* grids, cudaStream_t s);
// grids: C * L grids in (after the spread), read in their supported cells;
// with clear set the first pass zeroes each of them after reading it.
// scratch: fftpass_scratch elements; x (+)= the images' sums in a fixed order.
pg_status fftpass_adjoint(const NufftGeom& g, const FftBatch& b, const FftSupport& sup, float2* grids, int clear,
                          const float2* WoH, const float* deapf, const float2* tw, float2* scratch, int accumulate,
                          float2* x, cudaStream_t s);

}  // namespace pg
