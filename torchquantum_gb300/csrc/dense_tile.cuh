// dense_tile.cuh -- dense gates on 3 to 6 wires (dense_tile.cu), launched from apply.cu.
#pragma once

#include "common.cuh"

namespace tqk {

constexpr int kTileMinWires = 3, kTileMaxWires = 6;

struct DenseTileArgs {
  const float2* in;     // state read (forward); the gate's kept input (stored reverse step)
  float2* state;        // state written (may be in); reverse in place: psi
  const float2* lam_in; // reverse: the cotangent read (may be lam)
  float2* lam;          // reverse: the cotangent written
  int64_t bsz;
  int n, k;
  const int* tbits;     // index bit of matrix-index bit j (j = 0 is the most significant)
  const float2* mat;    // [batch][2^k][2^k]
  const float2* uinv;   // reverse in place: exact inverse for psi, or null (U^H)
  int64_t mat_batch;
  double* grad;         // reverse: [batch][2^k][2^k] complex128, or null
  bool stored;          // reverse: `in` is the gate's input, nothing is uncomputed
};

int launch_dense_tile(const DenseTileArgs& a, cudaStream_t st);      // state = U in
int launch_dense_tile_adj(const DenseTileArgs& a, cudaStream_t st);  // reverse step

}  // namespace tqk
