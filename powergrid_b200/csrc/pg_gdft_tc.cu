// The exact DFT's sums as a contraction on the 5th-generation tensor cores.
//
//   y_c[o] = sum_j e^{-/+ i phi(o, j)} v_c[j],  phi = 2 pi k . r + FM t
//
// For a tile of outputs and a run of inputs this is the real product
// D = A B with A[o][(j, cos)], A[o][(j, sin)] and B holding v_c[j]'s parts with
// the signs of the direction.  A is formed by the CUDA cores (the phase
// differs for every pair) and goes to tensor memory from registers; B is the
// coil data, staged in shared memory.  D = 2 columns per coil accumulates in
// tensor memory.  Plain FP32 needs 4 FMA per coil and pair, which at 8 coils
// was half of the instructions.
//
// 32-bit results from 16-bit operands: a = ah + al, b = bh + bl with ah, bh the
// values rounded to fp16 (11 bits) and al, bl their rests, rounded to fp16 too;
// D0 += ah bh, D1 += ah bl + al bh.  cos and sin are at most 1, so al is within
// 2^-24 of its rest; b is scaled by a power of two per coil that puts the largest
// entry into [2^14, 2^15) (undone exactly in the results), so that bl is within
// 2^-24 of it.  fp16 takes 16 rows of K per matrix instruction, tf32, of the same
// precision, 8: with two coil columns per output the instruction count is what
// the tensor core's time goes by (some 90 cycles each at N = 32).
// The tensor core's running sums round toward zero, so D is taken over after 32
// inputs (four additions) into FP32 registers, and these after 256 inputs into a
// compensated (Kahan) sum.
//
// Against 64 bits: 2.6e-7 (the plain kernels: 2.8e-7, and 4.8e-7 over sums of
// 131072 inputs).
//
// Phase: in units of turns.  q = 1.5 2^20 + kx x + ky y + kz z + (t / 2 pi) FM in
// double has its unit in the last place at 2^-32, so the low word of q is the
// fraction of a turn in two's complement: four FP64 fma, no rounding step, no
// subtraction, no FP64-to-FP32 conversion.  Holds for |phase| < 2^19 turns; plans
// are admitted below 2^18 (kTurnLimit), others use pg_gdft.cu's kernels.
//
// Split: a CTA is 8 warpgroups (4 with 16 coils) of 128 threads, each with a tile
// of 128 outputs (one thread and tensor-memory lane per output) and its share of
// the 512 tensor-memory columns: 32 of A (16 inputs x two parts, cos and sin in one
// column) and D0, D1.  The inputs' coordinates and B tile are shared by all.  A
// warpgroup's wait for its matrix product and the latency of its phase chain are
// covered by the others.
// What bounds it: the special-function unit (3 conversions or functions per
// pair at 16 a clock: 11.1 ms at 131072^2 pairs; measured 20.8 ms, from 34.8 ms on
// the plain kernels), the issue slots, and the tensor core's time per
// instruction.  With 8 warpgroups a thread has 64 registers and spills 68 bytes (100
// with gradients).  Forms measured on the way at that size: tf32 operands with 4
// warpgroups 24.5 ms, without its matrix instructions 17.7 ms; with 8 warpgroups
// and steps of 8 inputs 28.9 ms (half as many rows of K per instruction);
// polynomials in paired FP32 for sine and cosine 30.9 ms (33 instructions per pair).
#include <algorithm>

#include <cuda_fp16.h>

#include "pg_gdft_tc.cuh"

namespace pg {

namespace {

constexpr int kCh = 16;             // inputs per matrix step
constexpr int kDrain = 2;           // matrix steps per drain of D
constexpr int kFold = 2;            // tiles per compensated addition

// tcgen05 instruction descriptor: D f32, A and B f16, K-major, M = 128.
constexpr uint32_t idesc(int n) { return 1u << 4 | (uint32_t)(n >> 3) << 17 | 8u << 24; }

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory operand descriptor, K-major without swizzle: core matrices of 8
// rows x 16 bytes, `ld` bytes apart along K and 128 bytes apart along N.
__device__ __forceinline__ uint64_t bdesc(uint32_t addr, uint32_t ld) {
  return (uint64_t)(addr >> 4 & 0x3fffu) | (uint64_t)(ld >> 4) << 16 | (uint64_t)(128u >> 4) << 32 | 1ull << 46;
}

__device__ __forceinline__ void mma_f16(uint32_t d, uint32_t a, uint64_t b, uint32_t id, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(d),
      "r"(a), "l"(b), "r"(id), "r"(acc)
      : "memory");
}

#define PG_R8(r, o) "r"((r)[o]), "r"((r)[(o) + 1]), "r"((r)[(o) + 2]), "r"((r)[(o) + 3]), "r"((r)[(o) + 4]), \
                    "r"((r)[(o) + 5]), "r"((r)[(o) + 6]), "r"((r)[(o) + 7])
#define PG_W8(r, o) "=r"((r)[o]), "=r"((r)[(o) + 1]), "=r"((r)[(o) + 2]), "=r"((r)[(o) + 3]), "=r"((r)[(o) + 4]), \
                    "=r"((r)[(o) + 5]), "=r"((r)[(o) + 6]), "=r"((r)[(o) + 7])
__device__ __forceinline__ void tm_store16(uint32_t t, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15, %16};\n" ::"r"(t),
      PG_R8(r, 0), PG_R8(r, 8)
      : "memory");
}
__device__ __forceinline__ void tm_load16(uint32_t t, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
      "[%16];\n"
      : PG_W8(r, 0), PG_W8(r, 8)
      : "r"(t)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}

// Waits for a phase of an mbarrier, at most kWaitTries tries (each of which
// the hardware suspends for a while).  False when they ran out.
constexpr int kWaitTries = 1 << 16;
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  for (int i = 0; i < kWaitTries; ++i) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// Waits for the matrix products committed to `bar`.  They have then read their
// operands and written D: the fence orders this thread's next tcgen05.st (which
// overwrites A) and tcgen05.ld (which takes D) after them.
__device__ __forceinline__ bool product_wait(uint32_t bar, uint32_t parity) {
  const bool done = mbar_wait(bar, parity);
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  return done;
}

__device__ __forceinline__ void cp16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}

__device__ __forceinline__ float sinc_pg(float a) {
  return fabsf(a) < 0.0001f ? 1.0f : sinpif(a) / (3.14159265358979323846f * a);
}

// The pair's through-voxel dephasing factor (pg_gdft.cu): kn of the sample, gm of the voxel.
__device__ __forceinline__ float grad_factor(float4 kn, float4 gm) {
  return sinc_pg(kn.x + gm.x * kn.w) * sinc_pg(kn.y + gm.y * kn.w) * sinc_pg(kn.z + gm.z * kn.w);
}

template <int NC>
struct Tc {
  static constexpr int WG = NC == 8 ? 8 : 4;     // warpgroups (output tiles) per CTA
  static constexpr int TO = 128 * WG;            // outputs per CTA, threads
  static constexpr int TI = 128;                 // inputs per staged tile
  static_assert(gdft_tc_padded(1) % TI == 0, "input tables are padded to staged tiles");
  static constexpr int NT = 4 * NC;              // B columns: 2 NC heads, 2 NC rests
  static constexpr int kBlk = 8 * NT;            // words (two halves) of B per 8 inputs (16 rows of K)
  static constexpr int kTileB = TI / 8 * kBlk;   // words of B per staged tile
  static constexpr size_t tile = kTileB * sizeof(uint32_t) + TI * sizeof(double4);
  // two staged tiles, then per thread 2 NC sums and their compensations
  static constexpr size_t smem(bool grad) {
    return 2 * (tile + (grad ? TI * sizeof(float4) : 0)) + (size_t)TO * 4 * NC * sizeof(float);
  }
};

__device__ __forceinline__ float2 coil_value(const float2* S, const float2* v, uint64_t vstride, uint64_t in, int c,
                                             uint64_t j) {
  return S ? cmul(S[(uint64_t)c * in + j], v[j]) : v[(uint64_t)c * vstride + j];
}

// Largest |re| or |im| of every coil, as float bits (non-negative floats order
// like them; a NaN is the largest).
__global__ void k_tc_max(uint64_t in, const float2* __restrict__ S, const float2* __restrict__ v, uint64_t vstride,
                         unsigned* __restrict__ vmax) {
  const int c = blockIdx.y;
  unsigned m = 0u;
  for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < in; j += (uint64_t)gridDim.x * blockDim.x) {
    const float2 x = coil_value(S, v, vstride, in, c, j);
    m = max(m, max(__float_as_uint(x.x) & 0x7fffffffu, __float_as_uint(x.y) & 0x7fffffffu));
  }
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0 && m) atomicMax(&vmax[c], m);
}

// The power of two that takes a coil's largest entry into [2^14, 2^15); 1 for
// zero, infinite or NaN data.  2^127 and 2^-127 bound what can be undone.
__device__ __forceinline__ int tc_exponent(unsigned vmax) {
  if (vmax == 0u || vmax >= 0x7f800000u) return 0;
  const int e = vmax >= 0x00800000u ? (int)(vmax >> 23) - 127 : -127;
  return min(max(14 - e, -127), 127);
}

// B of the inputs [8 b, 8 b + 8): 16 K rows (cos and sin of the eight in turn) x
// NT columns as core matrices [k / 8][n / 8][n % 8][k % 8].
template <int NC>
__global__ void k_tc_pack(uint64_t in, uint64_t in_pad, int nc, int neg_i, const float2* __restrict__ S,
                          const float2* __restrict__ v, uint64_t vstride, const unsigned* __restrict__ vmax,
                          uint32_t* __restrict__ B) {
  constexpr int NT = Tc<NC>::NT;
  const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t j = t / NC;
  const int c = (int)(t - j * NC);
  if (j >= in_pad) return;
  float2 x = make_float2(0.f, 0.f);
  if (j < in && c < nc) {
    x = coil_value(S, v, vstride, in, c, j);
    const int e = tc_exponent(vmax[c]);
    x = make_float2(ldexpf(x.x, e), ldexpf(x.y, e));
  }
  // e^{-i phi} x = cos x + sin (-i x); e^{+i phi} x = cos x + sin (i x)
  const float rows[2][2] = {{x.x, x.y}, {neg_i ? x.y : -x.y, neg_i ? -x.x : x.x}};
  uint32_t* b = B + (j >> 3) * Tc<NC>::kBlk + (j & 3);
  const int kc = (int)(j >> 2) & 1;
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    const __half2 h = __floats2half2_rn(rows[0][p], rows[1][p]);
    const __half2 l = __floats2half2_rn(rows[0][p] - __low2float(h), rows[1][p] - __high2float(h));
    const int n0 = 2 * c + p, n1 = n0 + 2 * NC;
    b[((kc * (NT / 8) + n0 / 8) * 8 + n0 % 8) * 4] = *reinterpret_cast<const uint32_t*>(&h);
    b[((kc * (NT / 8) + n1 / 8) * 8 + n1 % 8) * 4] = *reinterpret_cast<const uint32_t*>(&l);
  }
}

template <int NC, bool GRAD>
__global__ void __launch_bounds__((Tc<NC>::TO), 1)
    k_tc_dft(GdftSide g, uint64_t tiles, int nsplit, const uint32_t* __restrict__ B, const unsigned* __restrict__ vmax,
             float2* __restrict__ part) {
  using T = Tc<NC>;
  constexpr int NT = T::NT, TO = T::TO, kTI = T::TI, V = 2 * NC;    // V: D0 (and D1) columns
  extern __shared__ __align__(128) unsigned char sm[];
  uint32_t* sB = reinterpret_cast<uint32_t*>(sm);                                 // [2][kTileB]
  double4* sV = reinterpret_cast<double4*>(sm + 2 * T::kTileB * sizeof(uint32_t));   // [2][kTI]
  float* sS = reinterpret_cast<float*>(sV + 2 * kTI);                             // [2 V][TO]
  float4* sG = reinterpret_cast<float4*>(sS + 2 * V * TO);                        // [2][kTI] with GRAD
  __shared__ uint64_t bars[T::WG];
  __shared__ uint32_t tmem_base;
  const int tid = threadIdx.x, warp = tid >> 5, wg = tid >> 7;
  const uint64_t o = (uint64_t)blockIdx.x * TO + tid;
  const uint64_t t0 = tiles * blockIdx.y / nsplit, t1 = tiles * (blockIdx.y + 1) / nsplit;

  auto stage = [&](uint64_t t, int buf) {
    const float4* b = reinterpret_cast<const float4*>(B + t * T::kTileB);
    const uint32_t db = smem_u32(sB + buf * T::kTileB);
    for (int q = tid; q < T::kTileB / 4; q += TO) cp16(db + q * 16, b + q);
    const uint32_t dv = smem_u32(sV + buf * kTI);
    const unsigned char* v = reinterpret_cast<const unsigned char*>(g.pi + t * kTI);
    if (tid < 2 * kTI) cp16(dv + tid * 16, v + tid * 16);
    if (GRAD && tid < kTI) cp16(smem_u32(sG + buf * kTI + tid), g.gi + t * kTI + tid);
  };

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;\n" ::"r"(smem_u32(&tmem_base))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  if (tid < T::WG) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&bars[tid])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (t0 < t1) stage(t0, 0);

  double4 k = make_double4(0, 0, 0, 0);
  float4 kn = make_float4(0.f, 0.f, 0.f, 0.f);
  if (o < g.out) {
    k = g.po[o];
    if (GRAD) kn = g.go[o];
  }
  for (int i = 0; i < 2 * V; ++i) sS[i * TO + tid] = 0.f;
  float2 sum[NC];                                      // over kFold tiles
#pragma unroll
  for (int i = 0; i < NC; ++i) sum[i] = make_float2(0.f, 0.f);

  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t tA = tmem_base + wg * (512 / T::WG), tD = tA + 32;   // A, then D0, D1
  const uint32_t lane = (uint32_t)(warp & 3) << 21;    // this warp's lanes: 32 (warp % 4) << 16
  const uint32_t bar = smem_u32(&bars[wg]);
  uint32_t parity = 0;
  bool pending = false, ok = true;

  // adds columns [0, V) at d to the sums
  auto take = [&](uint32_t d) {
#pragma unroll
    for (int h = 0; h < V / 16; ++h) {
      uint32_t r[16];
      tm_load16(d + lane + h * 16, r);
#pragma unroll
      for (int i = 0; i < 8; ++i)
        sum[h * 8 + i] = __fadd2_rn(sum[h * 8 + i], make_float2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1])));
    }
  };
  // running sums with the compensation of what each addition lost
  auto fold = [&]() {
#pragma unroll
    for (int i = 0; i < V; ++i) {
      float* ps = sS + i * TO + tid;
      float* pc = sS + (V + i) * TO + tid;
      const float s0 = *ps, v = (i & 1) ? sum[i / 2].y : sum[i / 2].x;
      const float y = __fsub_rn(v, *pc), t = __fadd_rn(s0, y);
      *pc = __fsub_rn(__fsub_rn(t, s0), y);
      *ps = t;
    }
#pragma unroll
    for (int i = 0; i < NC; ++i) sum[i] = make_float2(0.f, 0.f);
  };

  for (uint64_t t = t0; t < t1; ++t) {
    const int buf = (int)((t - t0) & 1);
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");   // the matrix unit reads what cp.async wrote
    __syncthreads();
    const double4* v4 = sV + buf * kTI;
    const float4* g4 = sG + buf * kTI;
#pragma unroll 1
    for (int ch = 0; ch < kTI / kCh; ++ch) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {                    // one K step: 8 inputs, heads, then rests
        uint32_t r[16];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int q = ch * kCh + h * 8 + j;
          const double4 v = v4[q];
          const double ph = fma(k.x, v.x, fma(k.y, v.y, fma(k.z, v.z, fma(k.w, v.w, 1572864.0))));
          float s, c;
          __sincosf((float)__double2loint(ph) * 1.4629180792671596e-9f, &s, &c);   // 2 pi / 2^32
          if (GRAD) {
            // (k / N, t) of the sample and (Gx, Gy, Gz) of the voxel, whichever side each is on
            const float4 gg = g4[q];
            const float f = g.out_is_sample ? grad_factor(kn, gg) : grad_factor(gg, kn);
            s *= f;
            c *= f;
          }
          const __half2 hd = __floats2half2_rn(c, s);
          const float2 hf = __half22float2(hd);
          const __half2 rs = __floats2half2_rn(c - hf.x, s - hf.y);
          r[j] = *reinterpret_cast<const uint32_t*>(&hd);
          r[j + 8] = *reinterpret_cast<const uint32_t*>(&rs);
        }
        if (h == 0 && pending) {
          // the previous step's product has read A and B and written D
          if (ok) ok = product_wait(bar, parity);
          parity ^= 1;
          pending = false;
          if (ch % kDrain == 0) {
            take(tD);
            take(tD + V);
          }
          if (ch == 0 && (t - t0) % kFold == 0) fold();
        }
        tm_store16(tA + lane + h * 16, r);
      }
      asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
      asm volatile("bar.sync %0, 128;\n" ::"r"(wg + 1) : "memory");
      if ((warp & 3) == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        if ((tid & 31) == 0) {
          const uint32_t b0 = smem_u32(sB + buf * T::kTileB + ch * (kCh / 8) * T::kBlk);
#pragma unroll
          for (int ks = 0; ks < kCh / 8; ++ks) {
            const uint32_t a = tA + ks * 16;
            const uint64_t bd = bdesc(b0 + ks * T::kBlk * 4, NT / 8 * 128);
            // heads x (heads | rests), then rests x heads into the rests' columns
            mma_f16(tD, a, bd, idesc(NT), (ch % kDrain > 0 || ks > 0) ? 1u : 0u);
            mma_f16(tD + V, a + 8, bd, idesc(V), 1u);
          }
          asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar)
                       : "memory");
        }
        __syncwarp();
      }
      pending = true;
      if (ch == 0 && t + 1 < t1) {
        // every warpgroup has waited for its last product of the previous
        // tile, so the other buffer is free
        __syncthreads();
        stage(t + 1, buf ^ 1);
      }
    }
  }
  if (pending) {
    // also where an earlier wait ran out: no product should be in flight when
    // tensor memory is freed
    const bool done = product_wait(bar, parity);
    ok = ok && done;
    take(tD);
    take(tD + V);
    fold();
  }
  if (o < g.out) {
    const float bad = ok ? 0.f : __int_as_float(0x7fffffff);   // a wait ran out: no silent result
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const float* ps = sS + 2 * c * TO + tid;
      const float* pc = ps + V * TO;
      const int e = -tc_exponent(vmax[c]);
      part[((uint64_t)blockIdx.y * NC + c) * g.out + o] =
          make_float2(ldexpf(ps[0] - pc[0], e) + bad, ldexpf(ps[TO] - pc[TO], e) + bad);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;\n" ::"r"(tmem_base) : "memory");
}

template <int NC>
pg_status pack_launch(const GdftSide& g, int nc, const float2* S, const float2* v, uint64_t vstride, unsigned* vmax,
                      uint32_t* B, cudaStream_t s) {
  const uint64_t ip = gdft_tc_padded(g.in);
  PG_CUDA(cudaMemsetAsync(vmax, 0, NC * sizeof(unsigned), s));
  PG_LAUNCH(k_tc_max, dim3(std::min<unsigned>(ceil_div(g.in, 1024), 4 * sm_count()), nc), 256, 0, s, g.in, S, v,
            vstride, vmax);
  PG_LAUNCH(k_tc_pack<NC>, ceil_div(ip * NC, 256), 256, 0, s, g.in, ip, nc, g.out_is_sample ? 1 : 0, S, v, vstride,
            vmax, B);
  return PG_OK;
}

template <int NC, bool GRAD>
pg_status sum_launch(const GdftSide& g, int nsplit, const uint32_t* B, const unsigned* vmax, float2* part,
                     cudaStream_t s) {
  const size_t smem = Tc<NC>::smem(GRAD);
  PG_CUDA(cudaFuncSetAttribute(k_tc_dft<NC, GRAD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  PG_LAUNCH((k_tc_dft<NC, GRAD>), dim3(ceil_div(g.out, Tc<NC>::TO), (unsigned)nsplit), Tc<NC>::TO, smem, s, g,
            gdft_tc_padded(g.in) / Tc<NC>::TI,
            nsplit, B, vmax, part);
  return PG_OK;
}

}  // namespace

int gdft_tc_coils(int C) { return C > 8 ? 16 : 8; }

uint64_t gdft_tc_operand(uint64_t in, int nc) { return gdft_tc_padded(in) / 8 * 32 * nc + 16; }

// One CTA per SM at a time: the fewest splits (of at least two tiles) whose
// last wave is at least 94 % full, else the fullest.
TcSplit gdft_tc_split(uint64_t out, uint64_t in, int ncp) {
  const uint64_t to = ncp == 8 ? Tc<8>::TO : Tc<16>::TO;
  const uint64_t blocks = (out + to - 1) / to, tiles = gdft_tc_padded(in) / 128, sms = (uint64_t)sm_count();
  const uint64_t most = std::max<uint64_t>(1, std::min<uint64_t>(tiles / 2, 64));
  TcSplit best{1, 0};
  double best_eff = 0.0;
  for (uint64_t ns = 1; ns <= most; ++ns) {
    const uint64_t waves = (blocks * ns + sms - 1) / sms;
    // tiles per split are whole: the longest split sets the wave's time
    const uint64_t longest = (tiles + ns - 1) / ns;
    const double eff = (double)(blocks * tiles) / (double)(waves * sms * longest);
    if (eff > best_eff + 1e-9) { best_eff = eff; best = {(int)ns, waves * longest}; }
    if (eff >= 0.94) break;
  }
  return best;
}

// The operand's last 16 words are the coils' largest entries.
pg_status gdft_tc_pack(const GdftSide& g, int nc, int ncp, const float2* S, const float2* v, uint64_t vstride,
                       uint32_t* B, cudaStream_t s) {
  unsigned* vmax = B + gdft_tc_operand(g.in, ncp) - 16;
  return ncp == 8 ? pack_launch<8>(g, nc, S, v, vstride, vmax, B, s) : pack_launch<16>(g, nc, S, v, vstride, vmax, B, s);
}

pg_status gdft_tc_sum(const GdftSide& g, int ncp, int nsplit, const uint32_t* B, float2* part, cudaStream_t s) {
  const bool grad = g.go != nullptr;
  const unsigned* m = B + gdft_tc_operand(g.in, ncp) - 16;
  if (ncp == 8)
    return grad ? sum_launch<8, true>(g, nsplit, B, m, part, s) : sum_launch<8, false>(g, nsplit, B, m, part, s);
  return grad ? sum_launch<16, true>(g, nsplit, B, m, part, s) : sum_launch<16, false>(g, nsplit, B, m, part, s);
}

}  // namespace pg
