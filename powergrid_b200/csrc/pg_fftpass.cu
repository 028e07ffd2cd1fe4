// Oversampled 2-D and 3-D FFTs for grids of 2N per axis, N a multiple of 8 up
// to 256 (or 512), written as pruned passes with the pre- and post-kernels
// fused in.
//
// The forward operator's input grid is zero outside the N x N image region
// (zero_pad, griddingSupport.cpp:372-404) and the adjoint keeps only that
// region of its output (crop_center_region, :408-460).  A library transform
// runs over the whole grid twice per direction; here
//   forward  F1  per image row: pre-kernel values (deapodization, coil map,
//                shot and segment phases, checkerboard sign) into a zero-
//                padded row, FFT along y                      -> N rows
//            F2  per grid column: the N nonzero rows, zero padded, FFT along
//                x                                             -> grid
//   adjoint  A1  per grid column: inverse FFT along x, keep the N cropped rows
//            A2  per cropped row: inverse FFT along y, keep the N cropped
//                columns, post-kernel weights (sign, deapodization, WoH,
//                conj coil map, conj shot phase), summed over grids
// In 3-D the first pass runs over the Nx*Nz image lines along y, the second
// along x over each of the Nz nonzero z-slabs, and a third along z over the
// (x, y) columns, reading only the Nz nonzero slabs; the adjoint mirrors it
// (z, keeping Nz slabs; x per slab, keeping Nx rows; y with the post weights).
// Transforms are unnormalised (FFTW/cuFFT conventions, forward sign -1).
//
// Support pruning.  A segment's grid is read (forward) or written (adjoint)
// only where the taps of that segment's samples fall.  A readout crosses
// k-space once, so a time segment covers a part of it: of a spiral's L segments
// each is an annulus, and together they cover about two discs, not L squares.
// The plan lists the groups of 8 adjacent y cells (64 bytes) with a sample
// (FftSupport); the passes compute, store, load and clear those groups only.
// The values of a supported cell do not depend on the list.  Measured on one
// B200 (operator pairs, forward + adjoint): 128^2 x 64, 2 shots, 4 coils, L = 12
// 10.45 -> 4.36 ms against passes over the whole grids; 208^2, 12 coils, L = 10
// 0.609 -> 0.361 ms and 96^2 x 16, 8 coils, L = 6 2.70 -> 1.86 ms against cuFFT.
//
// The kernels are in pg_fftkern.cuh, instantiated per length in pg_fft_len*.cu.
#include <algorithm>
#include <cmath>
#include <vector>

#include "pg_fftkern.cuh"

namespace pg {

const FftOps* fft_ops_0(int n);
const FftOps* fft_ops_1(int n);
const FftOps* fft_ops_2(int n);
const FftOps* fft_ops_3(int n);
const FftOps* fft_ops_4(int n);
const FftOps* fft_ops_5(int n);
const FftOps* fft_ops_6(int n);
const FftOps* fft_ops_7(int n);

namespace {

constexpr int kMaxGridY = 65535;

const FftOps* ops_for(int n) {
  using Fn = const FftOps* (*)(int);
  static constexpr Fn units[] = {fft_ops_0, fft_ops_1, fft_ops_2, fft_ops_3, fft_ops_4, fft_ops_5, fft_ops_6, fft_ops_7};
  for (Fn f : units)
    if (const FftOps* o = f(n)) return o;
  return nullptr;
}

// x[img][p] (+)= its `ng` partial images: 8 lanes per pixel, lane k takes images
// k, k+8, ..., added by a fixed xor butterfly.  An image whose coils began in an
// earlier batch (img * cgroup < c0) is added to.
__global__ void k_sum_images(uint64_t N, int ng, const float2* __restrict__ images, int img0, uint64_t image_stride,
                             int accumulate, int cgroup, int c0, float2* __restrict__ x) {
  pdl_wait();
  const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int k = (int)(t & 7);
  const uint64_t p = t >> 3;
  images += (uint64_t)blockIdx.y * ng * N;
  float2 acc = make_float2(0.f, 0.f);
  if (p < N)
    for (int b = k; b < ng; b += 8) acc = cadd(acc, images[(uint64_t)b * N + p]);
#pragma unroll
  for (int o = 4; o >= 1; o >>= 1) {
    acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
    acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
  }
  if (p < N && k == 0) {
    const int img = img0 + blockIdx.y;
    float2* o = x + (uint64_t)img * image_stride + p;
    *o = accumulate || (cgroup > 0 && img * cgroup < c0) ? cadd(*o, acc) : acc;
  }
}

// Grid cells (8 adjacent in y) that the taps of the samples reach in each
// segment: act[l][x][y / 8].  Every writer stores the same value.
__global__ void k_mark_support(NufftGeom g, uint64_t M, int K, const uint2* __restrict__ start,
                               const int* __restrict__ l0, uint8_t* __restrict__ act) {
  const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t i = t >> 3;
  if (i >= M) return;
  const uint32_t st = start[i].x;
  const int xx = (int)(st & 0xffff) + (int)(t & 7);
  if (xx >= g.Gx) return;
  const int y0 = (int)(st >> 16) >> 3, y1 = min((int)(st >> 16) + 7, g.Gy - 1) >> 3;
  const int nyg = g.Gy / 8, l = l0 ? l0[i] : 0;
  for (int j = 0; j < K; ++j)
    for (int y = y0; y <= y1; ++y) act[((uint64_t)(l + j) * g.Gx + xx) * nyg + y] = 1;
}

// Zeroes the supported groups of the batch's 3-D grids: four threads per
// group (64 bytes) and z plane.
__global__ void k_clear_groups(const uint32_t* __restrict__ list, int nlist, int L, uint64_t plane, int Gz, int zsplit,
                               float2* __restrict__ grids) {
  pdl_wait();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nlist * 4) return;
  const uint32_t ent = list[t >> 2];
  const int c = blockIdx.y / zsplit, part = blockIdx.y - c * zsplit;
  float2* p = grids + ((uint64_t)c * L + (ent >> 24)) * Gz * plane + (uint64_t)(ent & 0xffffffu) * 8 + (t & 3) * 2;
  for (int z = Gz * part / zsplit; z < Gz * (part + 1) / zsplit; ++z)
    *reinterpret_cast<float4*>(p + (uint64_t)z * plane) = make_float4(0.f, 0.f, 0.f, 0.f);
}

// R1 of the factorisation n = R1 * R2 (pg_fft_len*.cu).
int split_r1(int n) { return n >= 1024 ? 32 : n <= 16 ? 4 : n <= 32 ? 8 : 16; }

// W_n^(k1 m2) as [k1 < R1][m2 < R2] (forward) and as [k1 < R2][m2 < R1] (inverse).
void twiddle_table(int n, std::vector<float2>* h) {
  const int R1 = split_r1(n), R2 = n / R1;
  const double two_pi = 6.283185307179586476925286766559;
  for (int t = 0; t < 2; ++t)
    for (int k1 = 0; k1 < (t ? R2 : R1); ++k1)
      for (int m2 = 0; m2 < (t ? R1 : R2); ++m2) {
        const double a = -two_pi * (double)(k1 * m2) / (double)n;
        h->push_back(make_float2((float)std::cos(a), (float)std::sin(a)));
      }
}

// Blocks that a row pass should at least have: two per SM and a half wave more.
int wanted_blocks() { return 2 * sm_count() + sm_count() / 2; }

}  // namespace

bool fftpass_supported(const NufftGeom& g) {
  if (g.Gx != g.Gy || g.Gx != 2 * g.Nx || g.Ny != g.Nx || !ops_for(g.Gx)) return false;
  return g.dim == 2 || (g.Gz == 2 * g.Nz && ops_for(g.Gz));
}

pg_status fftpass_twiddles(const NufftGeom& g, DevBuf<float2>* tw, cudaStream_t s) {
  std::vector<float2> h;
  twiddle_table(g.Gx, &h);
  if (g.dim == 3) twiddle_table(g.Gz, &h);   // the z tables follow the in-plane ones
  return tw->upload(h.data(), h.size(), s);
}

pg_status fftpass_support(const NufftGeom& g, uint64_t M, int L, int K, const uint2* start, const int* l0,
                          FftSupport* out, cudaStream_t s) {
  const int n = g.Gx, nyg = g.Gy / 8, R1 = split_r1(n);
  const uint64_t na = (uint64_t)L * g.Gx * nyg;
  DevBuf<uint8_t> act;
  PG_TRY(act.alloc(na));
  PG_CUDA(cudaMemsetAsync(act.p, 0, na, s));
  PG_LAUNCH(k_mark_support, ceil_div(M * 8, 256), 256, 0, s, g, M, K, start, l0, act.p);
  std::vector<uint8_t> h(na);
  PG_CUDA(cudaMemcpyAsync(h.data(), act.p, na, cudaMemcpyDeviceToHost, s));
  PG_CUDA(cudaStreamSynchronize(s));
  std::vector<uint32_t> ymask((size_t)L * R1, 0u), xmask((size_t)L * nyg * R1, 0u), ylist, xylist;
  std::vector<uint8_t> any(nyg);
  for (int l = 0; l < L; ++l) {
    std::fill(any.begin(), any.end(), 0);
    for (int x = 0; x < g.Gx; ++x) {
      const uint8_t* a = h.data() + ((size_t)l * g.Gx + x) * nyg;
      for (int yg = 0; yg < nyg; ++yg)
        if (a[yg]) {
          any[yg] = 1;
          xmask[((size_t)l * nyg + yg) * R1 + x % R1] |= 1u << (x / R1);
          if (g.dim == 3) xylist.push_back((uint32_t)l << 24 | (uint32_t)(x * nyg + yg));
        }
    }
    for (int yg = 0; yg < nyg; ++yg)
      if (any[yg]) {
        ylist.push_back((uint32_t)l << 24 | (uint32_t)yg);
        for (int y = 8 * yg; y < 8 * yg + 8; ++y) ymask[(size_t)l * R1 + y % R1] |= 1u << (y / R1);
      }
  }
  out->ny = (int)ylist.size();
  out->nxy = (int)xylist.size();
  // one upload: [ymask][xmask][ylist][xylist]
  std::vector<uint32_t> all(std::move(ymask));
  const size_t ox = all.size(), oy = ox + xmask.size(), oxy = oy + ylist.size();
  all.insert(all.end(), xmask.begin(), xmask.end());
  all.insert(all.end(), ylist.begin(), ylist.end());
  all.insert(all.end(), xylist.begin(), xylist.end());
  PG_TRY(out->words.upload(all.data(), all.size(), s));
  out->ymask = out->words.p;
  out->xmask = out->words.p + ox;
  out->ylist = out->words.p + oy;
  out->xylist = out->words.p + oxy;
  PG_CUDA(cudaStreamSynchronize(s));   // the host lists are released on return
  return PG_OK;
}

// Small 2-D grids run both passes of a grid in one block while the batch is at
// most one wave.
static bool one_block_per_grid(const NufftGeom& g, const FftBatch& b, const FftOps* op) {
  return g.dim == 2 && op->grid_fwd && b.C * b.L <= sm_count();
}
// The adjoint then writes one image per grid, so every image of the batch has
// to have all of its coils in it.
static bool one_image_per_grid(const NufftGeom& g, const FftBatch& b, const FftOps* op) {
  return one_block_per_grid(g, b, op) && (b.cgroup == 0 || (b.c0 % b.cgroup == 0 && b.C % b.cgroup == 0));
}

// Elements of the half-transformed lines; none where both directions run one block
// per grid.
static uint64_t line_scratch(const NufftGeom& g, const FftBatch& b, const FftOps* op) {
  if (one_image_per_grid(g, b, op)) return 0;
  // 2-D: Nx rows of Gy per grid.  3-D: Nz*Nx rows of Gy, then Nz slabs of Gx*Gy.
  const uint64_t rows = (uint64_t)g.Nx * g.Nz * g.Gy;
  return (uint64_t)b.C * b.L * (g.dim == 2 ? rows : rows + (uint64_t)g.Nz * g.Gx * g.Gy);
}

static FftRows rows_args(const FftBatch& b, const FftSupport& sup, const float2* W, const float* deapf,
                         const float2* tw, int split, bool cluster = false) {
  return FftRows{b.L, b.C, b.c0, b.cgroup, b.image_stride, b.phase_stride, b.S, b.E, W, deapf, sup.ymask, tw, split,
                 cluster ? 1 : 0};
}

pg_status fftpass_forward(const NufftGeom& g, const FftBatch& b, const FftSupport& sup, const float2* x,
                          const float2* Wo, const float* deapf, const float2* tw, float2* scratch, float2* grids,
                          cudaStream_t s) {
  float2* P = scratch;
  const int B = b.C * b.L;
  if (B > kMaxGridY) return set_error(PG_INVALID_ARG, "fft passes: batch of %d grids", B);
  const FftOps* op = ops_for(g.Gx);
  if (one_block_per_grid(g, b, op))
    return op->grid_fwd(g, rows_args(b, sup, Wo, deapf, tw, 1), sup.xmask, x, grids, s);
  const uint64_t plane = (uint64_t)g.Gx * g.Gy, rows = (uint64_t)g.Nx * g.Gy;
  const int row_blocks = (int)ceil_div((uint64_t)g.Nx * g.Nz, op->rows_per_block);
  const int split = std::min(b.L, std::max(1, wanted_blocks() / std::max(1, row_blocks * b.C) + 1));
  PG_TRY(op->rows_fwd(g, rows_args(b, sup, Wo, deapf, tw, split), x, P, s));
  FftLines lx{rows, plane, (uint64_t)g.Gy, b.L, g.Nz, sup.ylist, sup.ny, sup.xmask, g.Gy / 8, tw};
  if (g.dim == 2) return op->cols_fwd(lx, b.C, P, grids, s);
  // x lines per nonzero z-slab, then z lines over the supported (x, y) columns
  float2* P2 = P + (uint64_t)B * g.Nz * rows;
  PG_TRY(op->cols_fwd(lx, (uint64_t)b.C * g.Nz, P, P2, s));
  const FftLines lz{(uint64_t)g.Nz * plane, g.ngrid(), plane, b.L, 1, sup.xylist, sup.nxy, nullptr, 0, tw + 2 * g.Gx};
  return ops_for(g.Gz)->cols_fwd(lz, b.C, P2, grids, s);
}

pg_status fftpass_clear(const NufftGeom& g, const FftBatch& b, const FftSupport& sup, float2* grids, cudaStream_t s) {
  if (sup.nxy == 0) return PG_OK;
  const unsigned bx = ceil_div((uint64_t)sup.nxy * 4, 256);
  const int zsplit = std::max(1, std::min(g.Gz, kMaxGridY / std::max(1, b.C)));
  const int zs = std::min(zsplit, 16);
  PG_LAUNCH_PDL(k_clear_groups, dim3(bx, (unsigned)(b.C * zs)), 256, 0, s, sup.xylist, sup.nxy, b.L,
                (uint64_t)g.Gx * g.Gy, g.Gz, zs, grids);
  return PG_OK;
}

static int batch_images(const FftBatch& b) {
  return b.cgroup > 0 ? (b.c0 + b.C - 1) / b.cgroup - b.c0 / b.cgroup + 1 : 1;
}

// How the grids of an image are shared out and added in the last inverse pass:
// one block (split 1), a cluster of `split` blocks, or images in memory.  A
// cluster saves the images' way through memory and a launch (64^2 x 32, 4 shots, TV
// solve 5.34 -> 5.02 ms); where 8 blocks per group of lines leave SMs idle, more
// shares with images in memory win (208^2, 12 coils, L = 10, pair: clusters of 8 378
// us, 11 shares 295 us).
struct InverseSplit {
  int split;
  bool cluster;
};
static InverseSplit inverse_split(const NufftGeom& g, const FftBatch& b, const FftOps* op) {
  const int nimages = batch_images(b);
  if (one_image_per_grid(g, b, op)) {
    const int grids = b.C / nimages * b.L;
    return {grids, grids <= 8 && (grids & (grids - 1)) == 0};
  }
  const int blocks = std::max(1, (int)ceil_div((uint64_t)g.Nx * g.Nz, op->rows_per_block) * nimages);
  const int per_image = std::max(1, b.C / nimages) * b.L;
  const int wave = op->row_blocks_per_sm * sm_count();
  if (8 * blocks < wave && per_image > 8) return {std::min(per_image, std::max(8, wave / blocks)), false};
  // the cluster size whose waves take the least time, a share's time being 1 / split
  int split = 1;
  double least = 1e30;
  for (int n = 1; n <= std::min(8, per_image); n *= 2) {
    const double t = (double)((blocks * n + wave - 1) / wave) / n;
    if (t < 0.95 * least) { least = t; split = n; }
  }
  return {split, split > 1};
}

uint64_t fftpass_scratch(const NufftGeom& g, const FftBatch& b) {
  const FftOps* op = ops_for(g.Gx);
  const InverseSplit is = inverse_split(g, b, op);
  const uint64_t images = is.split == 1 || is.cluster ? 0 : (uint64_t)is.split * batch_images(b) * g.nimg();
  return line_scratch(g, b, op) + images;
}

pg_status fftpass_adjoint(const NufftGeom& g, const FftBatch& b, const FftSupport& sup, float2* grids, int clear,
                          const float2* WoH, const float* deapf, const float2* tw, float2* scratch, int accumulate,
                          float2* x, cudaStream_t s) {
  const int B = b.C * b.L;
  if (B > kMaxGridY) return set_error(PG_INVALID_ARG, "fft passes: batch of %d grids", B);
  const uint64_t plane = (uint64_t)g.Gx * g.Gy, rows = (uint64_t)g.Nx * g.Gy, N = g.nimg();
  const int nimages = batch_images(b);
  const FftOps* op = ops_for(g.Gx);
  float2* Q = scratch;
  float2* images = scratch + line_scratch(g, b, op);
  const InverseSplit is = inverse_split(g, b, op);
  const bool kept = is.split > 1 && !is.cluster;   // images in memory, added by one more launch
  const FftRows ra = rows_args(b, sup, WoH, deapf, tw, is.split, is.cluster);
  if (one_image_per_grid(g, b, op)) {
    PG_TRY(op->grid_inv(g, ra, sup.xmask, grids, clear, accumulate, kept ? images : x, s));
  } else {
    FftLines lx{plane, rows, (uint64_t)g.Gy, b.L, g.Nz, sup.ylist, sup.ny, sup.xmask, g.Gy / 8, tw};
    if (g.dim == 2) {
      PG_TRY(op->cols_inv(lx, b.C, grids, clear, Q, s));
    } else {
      // z lines keeping the Nz cropped slabs, then x lines per slab keeping Nx rows
      float2* Q1 = Q + (uint64_t)B * g.Nz * rows;
      const FftLines lz{g.ngrid(), (uint64_t)g.Nz * plane, plane, b.L, 1, sup.xylist, sup.nxy, nullptr, 0,
                        tw + 2 * g.Gx};
      PG_TRY(ops_for(g.Gz)->cols_inv(lz, b.C, grids, clear, Q1, s));
      PG_TRY(op->cols_inv(lx, (uint64_t)b.C * g.Nz, Q1, 0, Q, s));
    }
    PG_TRY(op->rows_inv(g, ra, nimages, Q, accumulate, kept ? images : x, s));
  }
  if (!kept) return PG_OK;
  PG_LAUNCH_PDL(k_sum_images, dim3(ceil_div(N * 8, 256), (unsigned)nimages), 256, 0, s, N, is.split, images,
                b.cgroup > 0 ? b.c0 / b.cgroup : 0, b.image_stride, accumulate, b.cgroup, b.c0, x);
  return PG_OK;
}

}  // namespace pg
