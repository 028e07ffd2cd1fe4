// Kernels of the pruned oversampled FFT passes (pg_fftpass.cu), one set per
// length n = R1 * R2 = 2N.  Each translation unit pg_fft_len*.cu instantiates
// some lengths (FftOps) so that they compile in parallel.
//
// Each length-n transform is two register passes with one shared-memory
// transpose between them (the four-step form).  Forward, with m = R2 m1 + m2
// and k = k1 + R1 k2:
//   X[k] = sum_m2 W_R2^(m2 k2) * W_n^(m2 k1) * sum_m1 W_R1^(m1 k1) x[m].
// The zero padding leaves m in [n/4, 3n/4), which is m1 in [R1/4, 3 R1/4) for
// every m2: half of the first pass's inputs are literal zeros.  The inverse
// uses the split the other way round (m = R1 m1 + m2, k = k1 + R2 k2), so that
// the crop k in [n/4, 3n/4) is k2 in [R1/4, 3 R1/4): half of the second pass's
// outputs are never formed.  Both directions then store (forward) or load
// (inverse) grid rows r + R1 q, q < R2 <= 32, per thread, so the support of a
// thread's rows is one 32-bit word (pg_nufft.cuh, FftSupport).
//
// What bounds the passes is memory: in 3-D every grid line crosses HBM once
// per pass.  Rows of 8 adjacent y cells (64 bytes, the support's unit) that no
// sample of the segment touches are neither computed, stored, loaded nor
// cleared.
#pragma once

#include <algorithm>

#include <cooperative_groups.h>

#include "pg_fftdft.cuh"
#include "pg_fftpass.cuh"

namespace pg {

// Strided lines of the batch's grids: grid b = c * L + l holds `slabs` sets of
// lines (z slabs in the x pass, one set in the z pass).
struct FftLines {
  uint64_t in_stride, out_stride;   // elements between consecutive (grid, slab) sets
  uint64_t rstride;                 // elements between a line's consecutive rows
  int L, slabs;
  const uint32_t* list;             // active groups: segment << 24 | group of 8 adjacent columns
  int nlist;
  const uint32_t* rows;             // support words [segment][group][R1], or null: every row
  int ngroups;                      // groups per segment in `rows`
  const float2* tw;                 // W_n^(k1 m2): [R1][R2], then transposed [R2][R1]
};

// Image lines of the batch (rows along y).
struct FftRows {
  int L, C, c0;                     // segments, coils of the batch, their first map
  int cgroup;                       // coils per image, 0: one image
  uint64_t image_stride, phase_stride;
  const float2* S;                  // coil maps or null
  const float2* E;                  // extra image factor or null
  const float2* W;                  // Wo (forward) / WoH (inverse) or null
  const float* deapf;
  const uint32_t* rows;             // support words [segment][R1]
  const float2* tw;
  int split;                        // forward: blocks per coil; inverse: blocks per image
  int cluster;                      // inverse: the blocks of an image are a cluster
};

struct FftOps {
  int n;
  pg_status (*rows_fwd)(const NufftGeom& g, const FftRows& a, const float2* x, float2* P, cudaStream_t s);
  pg_status (*cols_fwd)(const FftLines& a, uint64_t nsets, const float2* in, float2* out, cudaStream_t s);
  pg_status (*cols_inv)(const FftLines& a, uint64_t nsets, float2* in, int clear, float2* out, cudaStream_t s);
  // out: x, or partial images (split > 1 without a cluster)
  pg_status (*rows_inv)(const NufftGeom& g, const FftRows& a, int nimages, const float2* Q, int accumulate,
                        float2* out, cudaStream_t s);
  int rows_per_block, row_blocks_per_sm;
  // both in-plane passes of a 2-D grid in one block per grid, or null
  pg_status (*grid_fwd)(const NufftGeom& g, const FftRows& a, const uint32_t* xmask, const float2* x, float2* grids,
                        cudaStream_t s);
  // split: the grids of an image; out: x, or every grid's image (split > 1 without a cluster)
  pg_status (*grid_inv)(const NufftGeom& g, const FftRows& a, const uint32_t* xmask, float2* grids, int clear,
                        int accumulate, float2* out, cudaStream_t s);
};

namespace fftk {

namespace cg = cooperative_groups;

__host__ __device__ constexpr int imax(int a, int b) { return a > b ? a : b; }
__host__ __device__ constexpr int imin(int a, int b) { return a < b ? a : b; }

// Row kernels: 16 lines per block (8, or 4 at n = 1024, where a pass has more
// than 16 threads per line), so that the 2-D sizes still give a few hundred
// blocks and the transpose fits 48 KB.
template <int R1, int R2>
struct RowGeo {
  static constexpr int n = R1 * R2;
  static constexpr int RB = n >= 1024 ? 4 : imax(R1, R2) > 16 ? 8 : 16;
  static constexpr int T = (RB * imax(R1, R2) + 31) / 32 * 32;
  // blocks per SM the registers are held to: the passes wait for memory between
  // their two barriers per grid (96^2 x 16, 8 coils, L = 6: last inverse pass with
  // its summing 94 -> 50 us; 208^2, 12 coils, L = 10: 62 -> 53 us)
  static constexpr int MINB = imax(R1, R2) <= 16 ? imin(4, 768 / T) : 2;
};
// Shared layout [row][k1 < RA][m2 < RBk]: odd m2 stride (the second pass's
// threads, one k1 each, hit distinct banks), row stride = RBk (mod 16).
template <int RA, int RBk>
struct RowSm {
  static constexpr int S2 = RBk | 1;
  static constexpr int base = RA * S2;
  static constexpr int RS = base + (((RBk - base) % 16) + 16) % 16;
};
// Line kernels: CB adjacent columns per block, shared layout [k1][m2][col];
// with 8 columns and an even R the k1 stride is padded by one row of columns
// so that the second pass's half-warps (two k1) hit distinct banks.
template <int R1, int R2>
struct ColGeo {
  static constexpr int n = R1 * R2;
  static constexpr int CB = n <= 64 ? 32 : n <= 256 ? 16 : 8;
  static constexpr int T = imin(256, (CB * imax(R1, R2) + 31) / 32 * 32);
  static constexpr int stride(int RBk) { return RBk * CB + (CB == 8 && RBk % 2 == 0 ? 8 : 0); }
  static constexpr size_t smem_fwd = (size_t)R1 * stride(R2) * sizeof(float2);
  static constexpr size_t smem_inv = (size_t)R2 * stride(R1) * sizeof(float2);
};

__device__ __forceinline__ int parity2(int a, int b) { return (a + b) & 1; }

// Image lines (ix, iz) of one coil: pre-kernel values (coil map, shot phase,
// deapodization, checkerboard sign) formed once and kept in registers, then
// per segment of the block's share the phase Wo and the FFT along y of the
// zero-padded line -> P[c * L + l][iz][ix][0..n), supported groups only.
template <int R1, int R2>
__global__ void __launch_bounds__((RowGeo<R1, R2>::T), (RowGeo<R1, R2>::MINB)) k_fft_fwd_rows(NufftGeom g, FftRows a,
                                                                      const float2* __restrict__ x,
                                                                      float2* __restrict__ P) {
  pdl_wait();
  using RG = RowGeo<R1, R2>;
  using SM = RowSm<R1, R2>;
  constexpr int n = RG::n, RB = RG::RB, H = R1 / 2;
  __shared__ float2 sh[RB * SM::RS];
  const int Nn = n / 2, nrows = g.Nx * g.Nz;
  const uint64_t N = g.nimg();
  const int cs = blockIdx.x % (a.C * a.split);   // coils fastest: they share the rows' segment phases in L2
  const int c = cs / a.split, part = cs - c * a.split;
  const int l0 = a.L * part / a.split, l1 = a.L * (part + 1) / a.split;
  const int cg = a.c0 + c;
  const int img = a.cgroup > 0 ? cg / a.cgroup : 0;
  const int r0 = blockIdx.x / (a.C * a.split) * RB;
  // first pass: thread (row, m2); second pass: thread (row, k1)
  const int m2 = threadIdx.x % R2, ra = threadIdx.x / R2;
  const int k1 = threadIdx.x % R1, rb = threadIdx.x / R1;
  const bool in_a = ra < RB && r0 + ra < nrows, in_b = rb < RB && r0 + rb < nrows;
  float2 u[H];
  uint64_t p0 = 0;
  if (in_a) {
    const int rg = r0 + ra, ix = rg % g.Nx, iz = rg / g.Nx;
    const int pxz = ix + g.pad_off[0] + iz + g.pad_off[2];
    p0 = (uint64_t)m2 + (uint64_t)Nn * rg;
#pragma unroll
    for (int h = 0; h < H; ++h) {
      const uint64_t p = p0 + R2 * h;
      float2 v = x[(uint64_t)img * a.image_stride + p];
      if (a.S) {
        const float2 sv = a.S[(uint64_t)cg * N + p];
        v = a.E ? cmul(v, cmul(sv, a.E[p])) : cmul(sv, v);
      }
      const float f = parity2(pxz, R2 * h + m2 + n / 4) ? -a.deapf[p] : a.deapf[p];
      u[h] = make_float2(v.x * f, v.y * f);
    }
  }
  const float2* W = a.W ? a.W + (uint64_t)img * a.phase_stride : nullptr;
  float2 w[H];
  if (W && in_a) {
#pragma unroll
    for (int h = 0; h < H; ++h) w[h] = W[(uint64_t)l0 * N + p0 + R2 * h];
  }
  for (int l = l0; l < l1; ++l) {
    if (in_a) {
      float2 v[R1];
#pragma unroll
      for (int m1 = 0; m1 < R1; ++m1) v[m1] = make_float2(0.f, 0.f);
#pragma unroll
      for (int h = 0; h < H; ++h) v[R1 / 4 + h] = W ? cmul(w[h], u[h]) : u[h];
      dft<R1>(v, false);
      float2* d = sh + ra * SM::RS + m2;
      d[0] = v[0];
#pragma unroll
      for (int q = 1; q < R1; ++q) d[q * SM::S2] = twiddle(v[q], a.tw[q * R2 + m2], false);
      if (W && l + 1 < l1) {               // the next segment's phases arrive during the second pass
#pragma unroll
        for (int h = 0; h < H; ++h) w[h] = W[(uint64_t)(l + 1) * N + p0 + R2 * h];
      }
    }
    __syncthreads();
    if (in_b) {
      const uint32_t sup = a.rows[l * R1 + k1];
      float2 v[R2];
      const float2* s = sh + rb * SM::RS + k1 * SM::S2;
#pragma unroll
      for (int q = 0; q < R2; ++q) v[q] = s[q];
      dft<R2>(v, false);
      float2* o = P + (((uint64_t)c * a.L + l) * nrows + r0 + rb) * n + k1;
#pragma unroll
      for (int k2 = 0; k2 < R2; ++k2)
        if (sup >> k2 & 1u) o[R1 * k2] = v[k2];
    }
    __syncthreads();
  }
}

// Strided lines forward: per active column the n/2 nonzero rows, zero padded
// to n, FFT along the line -> the output's supported rows.
template <int R1, int R2>
__global__ void __launch_bounds__((ColGeo<R1, R2>::T)) k_fft_fwd_cols(FftLines a, uint64_t set0,
                                                                      const float2* __restrict__ in,
                                                                      float2* __restrict__ out) {
  pdl_wait();
  using CG = ColGeo<R1, R2>;
  constexpr int CB = CG::CB, T = CG::T, S1 = CG::stride(R2), H = R1 / 2;
  extern __shared__ float2 sh[];
  const uint64_t y = set0 + blockIdx.y;      // coil * slabs + slab
  const uint64_t c = y / a.slabs, slab = y - c * a.slabs;
  const int e0 = blockIdx.x * (CB / 8);
#pragma unroll
  for (int it0 = 0; it0 < CB * R2; it0 += T) {
    const int it = it0 + threadIdx.x;
    if ((CB * R2) % T != 0 && it >= CB * R2) break;
    const int col = it % CB, m2 = it / CB;
    const int e = e0 + col / 8;
    if (e >= a.nlist) continue;
    const uint32_t ent = a.list[e];
    const float2* s = in + ((c * a.L + (ent >> 24)) * a.slabs + slab) * a.in_stride + (uint64_t)(ent & 0xffffffu) * 8 +
                      (col & 7) + (uint64_t)m2 * a.rstride;
    float2 v[R1];
#pragma unroll
    for (int m1 = 0; m1 < R1; ++m1) v[m1] = make_float2(0.f, 0.f);
#pragma unroll
    for (int h = 0; h < H; ++h) v[R1 / 4 + h] = s[(uint64_t)(R2 * h) * a.rstride];
    dft<R1>(v, false);
    float2* d = sh + m2 * CB + col;
    d[0] = v[0];
#pragma unroll
    for (int q = 1; q < R1; ++q) d[q * S1] = twiddle(v[q], a.tw[q * R2 + m2], false);
  }
  __syncthreads();
#pragma unroll
  for (int it0 = 0; it0 < CB * R1; it0 += T) {
    const int it = it0 + threadIdx.x;
    if ((CB * R1) % T != 0 && it >= CB * R1) break;
    const int col = it % CB, k1 = it / CB;
    const int e = e0 + col / 8;
    if (e >= a.nlist) continue;
    const uint32_t ent = a.list[e];
    const uint32_t l = ent >> 24, grp = ent & 0xffffffu;
    const uint32_t sup = a.rows ? a.rows[((uint64_t)l * a.ngroups + grp) * R1 + k1] : 0xffffffffu;
    float2 u[R2];
    const float2* s = sh + k1 * S1 + col;
#pragma unroll
    for (int q = 0; q < R2; ++q) u[q] = s[q * CB];
    dft<R2>(u, false);
    float2* o = out + ((c * a.L + l) * a.slabs + slab) * a.out_stride + (uint64_t)grp * 8 + (col & 7) +
                (uint64_t)k1 * a.rstride;
#pragma unroll
    for (int k2 = 0; k2 < R2; ++k2)
      if (sup >> k2 & 1u) o[(uint64_t)(R1 * k2) * a.rstride] = u[k2];
  }
}

// Strided lines inverse: per active column the supported rows (the others are
// zero), inverse FFT along the line, the n/2 cropped rows -> output.  Every
// supported cell is read exactly once; with CLEAR it is zeroed after that read
// (through inw, the same grids), which leaves the grids zero for the next
// adjoint spread.
template <int R1, int R2, bool CLEAR>
__global__ void __launch_bounds__((ColGeo<R1, R2>::T)) k_fft_inv_cols(FftLines a, uint64_t set0,
                                                                      const float2* __restrict__ in, float2* inw,
                                                                      float2* __restrict__ out) {
  pdl_wait();
  using CG = ColGeo<R1, R2>;
  constexpr int CB = CG::CB, T = CG::T, S1 = CG::stride(R1), H = R1 / 2;
  extern __shared__ float2 sh[];
  const uint64_t y = set0 + blockIdx.y;
  const uint64_t c = y / a.slabs, slab = y - c * a.slabs;
  const int e0 = blockIdx.x * (CB / 8);
  const float2* tw = a.tw + R1 * R2;       // transposed: [k1 < R2][m2 < R1]
#pragma unroll
  for (int it0 = 0; it0 < CB * R1; it0 += T) {
    const int it = it0 + threadIdx.x;
    if ((CB * R1) % T != 0 && it >= CB * R1) break;
    const int col = it % CB, m2 = it / CB;
    const int e = e0 + col / 8;
    if (e >= a.nlist) continue;
    const uint32_t ent = a.list[e];
    const uint32_t l = ent >> 24, grp = ent & 0xffffffu;
    const uint32_t sup = a.rows ? a.rows[((uint64_t)l * a.ngroups + grp) * R1 + m2] : 0xffffffffu;
    const uint64_t o = ((c * a.L + l) * a.slabs + slab) * a.in_stride + (uint64_t)grp * 8 + (col & 7) +
                       (uint64_t)m2 * a.rstride;
    float2 v[R2];
#pragma unroll
    for (int m1 = 0; m1 < R2; ++m1) {
      v[m1] = make_float2(0.f, 0.f);
      if (sup >> m1 & 1u) {
        if constexpr (CLEAR) v[m1] = inw[o + (uint64_t)(R1 * m1) * a.rstride];
        else v[m1] = in[o + (uint64_t)(R1 * m1) * a.rstride];
      }
    }
    dft<R2>(v, true);
    float2* d = sh + m2 * CB + col;
    d[0] = v[0];
#pragma unroll
    for (int q = 1; q < R2; ++q) d[q * S1] = twiddle(v[q], tw[q * R1 + m2], true);
    if constexpr (CLEAR) {
      // the addresses anew: kept from the loads they took up to 180 registers
      // (208^2, 12 coils, L = 10: 63 -> 45 us)
      uint64_t oc = o;
      asm volatile("" : "+l"(oc));
#pragma unroll
      for (int m1 = 0; m1 < R2; ++m1)
        if (sup >> m1 & 1u) inw[oc + (uint64_t)(R1 * m1) * a.rstride] = make_float2(0.f, 0.f);
    }
  }
  __syncthreads();
#pragma unroll
  for (int it0 = 0; it0 < CB * R2; it0 += T) {
    const int it = it0 + threadIdx.x;
    if ((CB * R2) % T != 0 && it >= CB * R2) break;
    const int col = it % CB, k1 = it / CB;
    const int e = e0 + col / 8;
    if (e >= a.nlist) continue;
    const uint32_t ent = a.list[e];
    float2 u[R1];
    const float2* s = sh + k1 * S1 + col;
#pragma unroll
    for (int q = 0; q < R1; ++q) u[q] = s[q * CB];
    dft<R1>(u, true);
    float2* o = out + ((c * a.L + (ent >> 24)) * a.slabs + slab) * a.out_stride + (uint64_t)(ent & 0xffffffu) * 8 +
                (col & 7) + (uint64_t)k1 * a.rstride;
#pragma unroll
    for (int h = 0; h < H; ++h) o[(uint64_t)(R2 * h) * a.rstride] = u[R1 / 4 + h];
  }
}

// Last inverse pass: lines (ix, iz) of the block's share of an image's grids,
// inverse FFT along y, crop, WoH, conj coil map and conj shot phase, summed
// over the share in grid order in registers; shot phase, deapodization and sign
// once at the end.  Up to 8 shares of one group of lines are the blocks of a cluster,
// which adds them in rank order through distributed shared memory; more shares
// (small images, which need them to fill the GPU) write partial images.
template <int R1, int R2>
__global__ void __launch_bounds__((RowGeo<R1, R2>::T), (RowGeo<R1, R2>::MINB)) k_fft_inv_rows(NufftGeom g, FftRows a, int nimages,
                                                                      const float2* __restrict__ Q, int accumulate,
                                                                      float2* __restrict__ out) {
  pdl_wait();
  using RG = RowGeo<R1, R2>;
  using SM = RowSm<R2, R1>;
  constexpr int n = RG::n, RB = RG::RB, H = R1 / 2;
  __shared__ float2 sh[RB * SM::RS];
  const int Nn = n / 2, nrows = g.Nx * g.Nz;
  const uint64_t N = g.nimg();
  const int is = blockIdx.x % (nimages * a.split);
  const int i = is / a.split, part = is - i * a.split;
  // the image's coils inside the batch [c0, c0 + C)
  const int img = a.cgroup > 0 ? a.c0 / a.cgroup + i : 0;
  const int ca = a.cgroup > 0 ? max(a.c0, img * a.cgroup) : a.c0;
  const int cb = a.cgroup > 0 ? min(a.c0 + a.C, (img + 1) * a.cgroup) : a.c0 + a.C;
  const int nb = (cb - ca) * a.L;
  const int b0 = (int)((int64_t)nb * part / a.split), b1 = (int)((int64_t)nb * (part + 1) / a.split);
  const int r0 = blockIdx.x / (nimages * a.split) * RB;
  // first pass: thread (row, m2 < R1); second pass: thread (row, k1 < R2)
  const int m2 = threadIdx.x % R1, ra = threadIdx.x / R1;
  const int k1 = threadIdx.x % R2, rb = threadIdx.x / R2;
  const bool in_a = ra < RB && r0 + ra < nrows, in_b = rb < RB && r0 + rb < nrows;
  const uint64_t p0 = (uint64_t)k1 + (uint64_t)Nn * (r0 + rb);
  const float2* W = a.W ? a.W + (uint64_t)img * a.phase_stride : nullptr;
  const float2* tw = a.tw + n;             // transposed: [k1 < R2][m2 < R1]
  float2 acc[H];                           // over the share
#pragma unroll
  for (int h = 0; h < H; ++h) acc[h] = make_float2(0.f, 0.f);
  for (int b = b0; b < b1; ++b) {
    const int c = ca + b / a.L, l = b % a.L;
    if (in_a) {
      const uint32_t sup = a.rows[l * R1 + m2];
      const float2* s = Q + (((uint64_t)(c - a.c0) * a.L + l) * nrows + r0 + ra) * n + m2;
      float2 v[R2];
#pragma unroll
      for (int m1 = 0; m1 < R2; ++m1) {
        v[m1] = make_float2(0.f, 0.f);
        if (sup >> m1 & 1u) v[m1] = s[R1 * m1];
      }
      dft<R2>(v, true);
      float2* d = sh + ra * SM::RS + m2;
      d[0] = v[0];
#pragma unroll
      for (int q = 1; q < R2; ++q) d[q * SM::S2] = twiddle(v[q], tw[q * R1 + m2], true);
    }
    __syncthreads();
    if (in_b) {
      float2 u[R1];
      const float2* s = sh + rb * SM::RS + k1 * SM::S2;
#pragma unroll
      for (int q = 0; q < R1; ++q) u[q] = s[q];
      dft<R1>(u, true);
#pragma unroll
      for (int h = 0; h < H; ++h) {
        const uint64_t p = p0 + R2 * h;
        float2 v = u[R1 / 4 + h];
        if (W) v = cmul(v, W[(uint64_t)l * N + p]);
        if (a.S) v = cmul(v, cconj(a.S[(uint64_t)c * N + p]));
        acc[h] = cadd(acc[h], v);
      }
    }
    __syncthreads();
  }
  const bool partial = a.split > 1 && !a.cluster;
  const bool add = !partial && (accumulate || (a.cgroup > 0 && img * a.cgroup < a.c0));
  float2* o = partial ? out + (uint64_t)is * N : out + (uint64_t)img * a.image_stride;
  auto store = [&](int row, int iy, float2 v) {
    const int rg = r0 + row, pxz = rg % g.Nx + g.crop_off[0] + rg / g.Nx + g.crop_off[2];
    const uint64_t p = (uint64_t)iy + (uint64_t)Nn * rg;
    const float f = parity2(pxz, iy + n / 4) ? -a.deapf[p] : a.deapf[p];
    if (a.S && a.E) v = cmul(cconj(a.E[p]), v);
    v = make_float2(v.x * f, v.y * f);
    o[p] = add ? cadd(o[p], v) : v;
  };
  if (a.split == 1 || partial) {
    if (in_b) {
#pragma unroll
      for (int h = 0; h < H; ++h) store(rb, k1 + R2 * h, acc[h]);
    }
    return;
  }
  // every thread of every block of the cluster reaches both barriers
  if (in_b) {
#pragma unroll
    for (int h = 0; h < H; ++h) sh[rb * Nn + k1 + R2 * h] = acc[h];
  }
  cg::cluster_group cl = cg::this_cluster();
  cl.sync();
  const int rows = min(RB, nrows - r0);
  for (int i = part * RG::T + threadIdx.x; i < rows * Nn; i += a.split * RG::T) {
    float2 v = *cl.map_shared_rank(sh + i, 0);
    for (int q = 1; q < a.split; ++q) v = cadd(v, *cl.map_shared_rank(sh + i, q));
    store(i / Nn, i % Nn, v);
  }
  cl.sync();   // no block leaves while another reads its shared memory
}

// ---------------------------------------------------------------------------
// Small 2-D grids (n <= 64): both passes of a grid in one block, the half-
// transformed rows in shared memory.  The values are those of the separate
// passes.  At these sizes a pass is a few microseconds of latency over a handful
// of blocks; one launch and one trip through L2 fewer per direction.  An operator
// pair of 32 x 32, 2 coils, L = 4: 33.4 -> 28.2 us; at n = 128 one block per grid
// was slower (a 64 x 64 solve of 3 steps 164 against 159 us).
// ---------------------------------------------------------------------------
template <int R1, int R2>
struct GridGeo {
  static constexpr int n = R1 * R2, N = n / 2;
  static constexpr int T = 256;
  static constexpr size_t held = (size_t)N * n;    // the transformed rows / the cropped columns
  static constexpr size_t work = (size_t)imax(n * n, N * imax(RowSm<R1, R2>::RS, RowSm<R2, R1>::RS));
  static constexpr size_t smem = (held + work) * sizeof(float2);
};

template <int R1, int R2>
__global__ void __launch_bounds__((GridGeo<R1, R2>::T)) k_fft2_fwd_grid(NufftGeom g, FftRows a,
                                                                       const uint32_t* __restrict__ xmask,
                                                                       const float2* __restrict__ x,
                                                                       float2* __restrict__ grids) {
  pdl_wait();
  using GG = GridGeo<R1, R2>;
  using SM = RowSm<R1, R2>;
  constexpr int n = GG::n, N = GG::N, T = GG::T, H = R1 / 2;
  extern __shared__ float2 sh[];
  float2* P = sh;                 // [row][n]
  float2* Wk = sh + GG::held;
  const int b = blockIdx.x, c = b / a.L, l = b - c * a.L, cg = a.c0 + c;
  const int img = a.cgroup > 0 ? cg / a.cgroup : 0;
  const float2* xi = x + (uint64_t)img * a.image_stride;
  const float2* S = a.S ? a.S + (uint64_t)cg * N * N : nullptr;
  const float2* W = a.W ? a.W + (uint64_t)img * a.phase_stride + (uint64_t)l * N * N : nullptr;
  for (int it = threadIdx.x; it < N * R2; it += T) {         // y transform, first pass: (row, m2)
    const int m2 = it % R2, r = it / R2;
    float2 v[R1];
#pragma unroll
    for (int m1 = 0; m1 < R1; ++m1) v[m1] = make_float2(0.f, 0.f);
#pragma unroll
    for (int h = 0; h < H; ++h) {
      const int p = R2 * h + m2 + N * r;
      float2 u = xi[p];
      if (S) u = a.E ? cmul(u, cmul(S[p], a.E[p])) : cmul(S[p], u);
      const float f = parity2(r + g.pad_off[0], R2 * h + m2 + n / 4) ? -a.deapf[p] : a.deapf[p];
      u = make_float2(u.x * f, u.y * f);
      v[R1 / 4 + h] = W ? cmul(W[p], u) : u;
    }
    dft<R1>(v, false);
    float2* d = Wk + r * SM::RS + m2;
    d[0] = v[0];
#pragma unroll
    for (int q = 1; q < R1; ++q) d[q * SM::S2] = twiddle(v[q], a.tw[q * R2 + m2], false);
  }
  __syncthreads();
  for (int it = threadIdx.x; it < N * R1; it += T) {         // second pass: (row, k1)
    const int k1 = it % R1, r = it / R1;
    float2 v[R2];
    const float2* s = Wk + r * SM::RS + k1 * SM::S2;
#pragma unroll
    for (int q = 0; q < R2; ++q) v[q] = s[q];
    dft<R2>(v, false);
#pragma unroll
    for (int k2 = 0; k2 < R2; ++k2) P[r * n + k1 + R1 * k2] = v[k2];
  }
  __syncthreads();
  const uint32_t* ym = a.rows + l * R1;                      // columns some sample reaches
  for (int it = threadIdx.x; it < n * R2; it += T) {         // x transform, first pass: (column, m2)
    const int col = it % n, m2 = it / n;
    if (!(ym[col % R1] >> (col / R1) & 1u)) continue;
    float2 v[R1];
#pragma unroll
    for (int m1 = 0; m1 < R1; ++m1) v[m1] = make_float2(0.f, 0.f);
#pragma unroll
    for (int h = 0; h < H; ++h) v[R1 / 4 + h] = P[(R2 * h + m2) * n + col];
    dft<R1>(v, false);
    float2* d = Wk + m2 * n + col;
    d[0] = v[0];
#pragma unroll
    for (int q = 1; q < R1; ++q) d[q * R2 * n] = twiddle(v[q], a.tw[q * R2 + m2], false);
  }
  __syncthreads();
  float2* out = grids + (uint64_t)b * n * n;
  for (int it = threadIdx.x; it < n * R1; it += T) {         // second pass: (column, k1)
    const int col = it % n, k1 = it / n;
    if (!(ym[col % R1] >> (col / R1) & 1u)) continue;
    const uint32_t sup = xmask[((uint64_t)l * (n / 8) + col / 8) * R1 + k1];
    float2 u[R2];
    const float2* s = Wk + k1 * R2 * n + col;
#pragma unroll
    for (int q = 0; q < R2; ++q) u[q] = s[q * n];
    dft<R2>(u, false);
#pragma unroll
    for (int k2 = 0; k2 < R2; ++k2)
      if (sup >> k2 & 1u) out[(k1 + R1 * k2) * n + col] = u[k2];
  }
}

template <int R1, int R2>
__global__ void __launch_bounds__((GridGeo<R1, R2>::T)) k_fft2_inv_grid(NufftGeom g, FftRows a,
                                                                       const uint32_t* __restrict__ xmask,
                                                                       float2* grids, int clear, int accumulate,
                                                                       float2* __restrict__ out) {
  pdl_wait();
  using GG = GridGeo<R1, R2>;
  using SM = RowSm<R2, R1>;
  constexpr int n = GG::n, N = GG::N, T = GG::T, H = R1 / 2;
  extern __shared__ float2 sh[];
  float2* Q = sh;                 // [cropped row][n]
  float2* Wk = sh + GG::held;
  const int b = blockIdx.x, c = b / a.L, l = b - c * a.L, cg = a.c0 + c;
  const int img = a.cgroup > 0 ? cg / a.cgroup : 0;
  const uint32_t* ym = a.rows + l * R1;
  const float2* tw = a.tw + n;    // transposed: [k1 < R2][m2 < R1]
  float2* in = grids + (uint64_t)b * n * n;
  for (int it = threadIdx.x; it < n * R1; it += T) {         // x transform, first pass: (column, m2)
    const int col = it % n, m2 = it / n;
    if (!(ym[col % R1] >> (col / R1) & 1u)) continue;
    const uint32_t sup = xmask[((uint64_t)l * (n / 8) + col / 8) * R1 + m2];
    float2 v[R2];
#pragma unroll
    for (int m1 = 0; m1 < R2; ++m1) v[m1] = sup >> m1 & 1u ? in[(R1 * m1 + m2) * n + col] : make_float2(0.f, 0.f);
    dft<R2>(v, true);
    float2* d = Wk + m2 * n + col;
    d[0] = v[0];
#pragma unroll
    for (int q = 1; q < R2; ++q) d[q * R1 * n] = twiddle(v[q], tw[q * R1 + m2], true);
    if (clear) {
#pragma unroll
      for (int m1 = 0; m1 < R2; ++m1)
        if (sup >> m1 & 1u) in[(R1 * m1 + m2) * n + col] = make_float2(0.f, 0.f);
    }
  }
  __syncthreads();
  for (int it = threadIdx.x; it < n * R2; it += T) {         // second pass: (column, k1 < R2)
    const int col = it % n, k1 = it / n;
    if (!(ym[col % R1] >> (col / R1) & 1u)) continue;
    float2 u[R1];
    const float2* s = Wk + k1 * R1 * n + col;
#pragma unroll
    for (int q = 0; q < R1; ++q) u[q] = s[q * n];
    dft<R1>(u, true);
#pragma unroll
    for (int h = 0; h < H; ++h) Q[(k1 + R2 * h) * n + col] = u[R1 / 4 + h];
  }
  __syncthreads();
  for (int it = threadIdx.x; it < N * R1; it += T) {         // y transform, first pass: (row, m2)
    const int m2 = it % R1, r = it / R1;
    const uint32_t sup = ym[m2];
    float2 v[R2];
#pragma unroll
    for (int m1 = 0; m1 < R2; ++m1) v[m1] = sup >> m1 & 1u ? Q[r * n + R1 * m1 + m2] : make_float2(0.f, 0.f);
    dft<R2>(v, true);
    float2* d = Wk + r * SM::RS + m2;
    d[0] = v[0];
#pragma unroll
    for (int q = 1; q < R2; ++q) d[q * SM::S2] = twiddle(v[q], tw[q * R1 + m2], true);
  }
  __syncthreads();
  const float2* S = a.S ? a.S + (uint64_t)cg * N * N : nullptr;
  const float2* W = a.W ? a.W + (uint64_t)img * a.phase_stride + (uint64_t)l * N * N : nullptr;
  // the grid's image: to x (split 1), to memory, or into shared memory, where the
  // cluster of the image's grids adds them in rank order
  const bool cluster = a.split > 1 && a.cluster;
  float2* o = cluster ? Q : a.split == 1 ? out + (uint64_t)img * a.image_stride : out + (uint64_t)b * N * N;
  const bool add = a.split == 1 && accumulate;
  for (int it = threadIdx.x; it < N * R2; it += T) {         // second pass: (row, k1 < R2)
    const int k1 = it % R2, r = it / R2;
    float2 u[R1];
    const float2* s = Wk + r * SM::RS + k1 * SM::S2;
#pragma unroll
    for (int q = 0; q < R1; ++q) u[q] = s[q];
    dft<R1>(u, true);
#pragma unroll
    for (int h = 0; h < H; ++h) {
      const int p = k1 + R2 * h + N * r;
      float2 v = u[R1 / 4 + h];
      if (W) v = cmul(v, W[p]);
      if (S) v = a.E ? cmul(cmul(cconj(S[p]), cconj(a.E[p])), v) : cmul(v, cconj(S[p]));
      const float f = parity2(r + g.crop_off[0], R2 * h + k1 + n / 4) ? -a.deapf[p] : a.deapf[p];
      v = make_float2(v.x * f, v.y * f);
      o[p] = add ? cadd(o[p], v) : v;
    }
  }
  if (!cluster) return;
  // every thread of every block of the cluster reaches both barriers
  cg::cluster_group cl = cg::this_cluster();
  cl.sync();
  float2* xi = out + (uint64_t)img * a.image_stride;
  for (int p = (int)cl.block_rank() * T + threadIdx.x; p < N * N; p += a.split * T) {
    float2 v = *cl.map_shared_rank(Q + p, 0);
    for (int q = 1; q < a.split; ++q) v = cadd(v, *cl.map_shared_rank(Q + p, q));
    xi[p] = accumulate ? cadd(xi[p], v) : v;
  }
  cl.sync();   // no block leaves while another reads its shared memory
}

template <typename K>
pg_status allow_smem(K kernel, size_t bytes) {
  if (bytes > 48 * 1024) PG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  return PG_OK;
}

constexpr uint64_t kMaxGridY = 65535;

template <int R1, int R2>
pg_status rows_fwd(const NufftGeom& g, const FftRows& a, const float2* x, float2* P, cudaStream_t s) {
  using RG = RowGeo<R1, R2>;
  PG_LAUNCH_PDL((k_fft_fwd_rows<R1, R2>), (unsigned)(a.C * a.split) * ceil_div((uint64_t)g.Nx * g.Nz, RG::RB),
                RG::T, 0, s, g, a, x, P);
  return PG_OK;
}

// Launch in clusters of `size` blocks along x, after the previous kernel (pdl_wait).
template <typename Kern, typename... Args>
pg_status launch_cluster(Kern kern, unsigned grid, int block, size_t smem, int size, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = (unsigned)size;
  at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = size > 1 ? 2 : 1;
  PG_CUDA(cudaLaunchKernelEx(&cfg, kern, args...));
  count_launch();
  return PG_OK;
}

template <int R1, int R2>
pg_status rows_inv(const NufftGeom& g, const FftRows& a, int nimages, const float2* Q, int accumulate, float2* out,
                   cudaStream_t s) {
  using RG = RowGeo<R1, R2>;
  return launch_cluster(k_fft_inv_rows<R1, R2>,
                        (unsigned)(nimages * a.split) * ceil_div((uint64_t)g.Nx * g.Nz, RG::RB), RG::T, 0,
                        a.cluster ? a.split : 1, s,
                        g, a, nimages, Q, accumulate, out);
}

template <int R1, int R2>
pg_status cols_fwd(const FftLines& a, uint64_t nsets, const float2* in, float2* out, cudaStream_t s) {
  using CG = ColGeo<R1, R2>;
  if (a.nlist == 0) return PG_OK;
  PG_TRY(allow_smem(k_fft_fwd_cols<R1, R2>, CG::smem_fwd));
  for (uint64_t s0 = 0; s0 < nsets; s0 += kMaxGridY)
    PG_LAUNCH_PDL((k_fft_fwd_cols<R1, R2>), dim3(ceil_div(a.nlist, CG::CB / 8), (unsigned)std::min(kMaxGridY, nsets - s0)),
                  CG::T, CG::smem_fwd, s, a, s0, in, out);
  return PG_OK;
}

template <int R1, int R2>
pg_status cols_inv(const FftLines& a, uint64_t nsets, float2* in, int clear, float2* out, cudaStream_t s) {
  using CG = ColGeo<R1, R2>;
  if (a.nlist == 0) return PG_OK;
  PG_TRY(clear ? allow_smem(k_fft_inv_cols<R1, R2, true>, CG::smem_inv)
               : allow_smem(k_fft_inv_cols<R1, R2, false>, CG::smem_inv));
  for (uint64_t s0 = 0; s0 < nsets; s0 += kMaxGridY) {
    const dim3 grid(ceil_div(a.nlist, CG::CB / 8), (unsigned)std::min(kMaxGridY, nsets - s0));
    if (clear)
      PG_LAUNCH_PDL((k_fft_inv_cols<R1, R2, true>), grid, CG::T, CG::smem_inv, s, a, s0, (const float2*)in, in, out);
    else
      PG_LAUNCH_PDL((k_fft_inv_cols<R1, R2, false>), grid, CG::T, CG::smem_inv, s, a, s0, (const float2*)in,
                    (float2*)nullptr, out);
  }
  return PG_OK;
}

template <int R1, int R2>
pg_status grid_fwd(const NufftGeom& g, const FftRows& a, const uint32_t* xmask, const float2* x, float2* grids,
                   cudaStream_t s) {
  using GG = GridGeo<R1, R2>;
  PG_TRY(allow_smem(k_fft2_fwd_grid<R1, R2>, GG::smem));
  PG_LAUNCH_PDL((k_fft2_fwd_grid<R1, R2>), (unsigned)(a.C * a.L), GG::T, GG::smem, s, g, a, xmask, x, grids);
  return PG_OK;
}

template <int R1, int R2>
pg_status grid_inv(const NufftGeom& g, const FftRows& a, const uint32_t* xmask, float2* grids, int clear,
                   int accumulate, float2* out, cudaStream_t s) {
  using GG = GridGeo<R1, R2>;
  PG_TRY(allow_smem(k_fft2_inv_grid<R1, R2>, GG::smem));
  return launch_cluster(k_fft2_inv_grid<R1, R2>, (unsigned)(a.C * a.L), GG::T, GG::smem, a.cluster ? a.split : 1, s, g, a,
                        xmask, grids, clear, accumulate, out);
}

}  // namespace fftk

template <int R1, int R2>
const FftOps* fft_ops() {
  static const FftOps ops = [] {
    FftOps o{R1 * R2, fftk::rows_fwd<R1, R2>, fftk::cols_fwd<R1, R2>, fftk::cols_inv<R1, R2>,
             fftk::rows_inv<R1, R2>, fftk::RowGeo<R1, R2>::RB, fftk::RowGeo<R1, R2>::MINB, nullptr, nullptr};
    if constexpr (R1 * R2 <= 64) {
      o.grid_fwd = fftk::grid_fwd<R1, R2>;
      o.grid_inv = fftk::grid_inv<R1, R2>;
    }
    return o;
  }();
  return &ops;
}

}  // namespace pg
