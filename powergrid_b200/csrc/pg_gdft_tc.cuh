// Gdft sums on the tensor cores (pg_gdft_tc.cu).
#pragma once

#include "pg_gdft.cuh"

namespace pg {

// One direction of the DFT: `out` outputs, `in` inputs, C coils.
struct GdftSide {
  uint64_t out, in;
  const double4* po;      // per output: turn coordinates or voxel coordinates
  const double4* pi;      // per input, the other kind; gdft_tc_padded(in) entries
  const float4* go;       // GdftR2 factors of the outputs / inputs, or null
  const float4* gi;
  bool out_is_sample;     // forward: outputs are samples, sign -i; adjoint: voxels, +i
};

// Whether every |phase| of the plan stays below 2^18 turns, so that the
// fixed-point phase (pg_gdft_tc.cu) holds it.
constexpr double kTurnLimit = 262144.0;

// Entries of a table of n inputs, padded to whole staged tiles.
constexpr uint64_t gdft_tc_padded(uint64_t n) { return (n + 127) / 128 * 128; }

// Coils per tensor pass for C coils (8 or 16).
int gdft_tc_coils(int C);
// Splits of the inner sum, and the staged tiles of 128 inputs that the busiest SM
// then goes through one after another.
struct TcSplit {
  int splits;
  uint64_t steps;
};
TcSplit gdft_tc_split(uint64_t out, uint64_t in, int ncp);
// Words of the packed operand for `in` inputs and nc (8 or 16) coils.
uint64_t gdft_tc_operand(uint64_t in, int nc);
// Packs coils [0, nc) of v (S null: v_c[j]; else S_c[j] v[j], one v for all coils).
pg_status gdft_tc_pack(const GdftSide& g, int nc, int ncp, const float2* S, const float2* v, uint64_t vstride,
                       uint32_t* B, cudaStream_t s);
// part[(split * ncp + c) * out + o]
pg_status gdft_tc_sum(const GdftSide& g, int ncp, int nsplit, const uint32_t* B, float2* part, cudaStream_t s);

}  // namespace pg
