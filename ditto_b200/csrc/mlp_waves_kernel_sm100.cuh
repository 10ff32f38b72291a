// What the wave kernel's instances (mlp_waves_kernel_sm100.cu) and the code that plans and launches them (mlp_waves_sm100.cu) share.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include "mlp_waves_sm100.cuh"

namespace ditto_b200 {
namespace waves {

constexpr int kRows = 128;                 // rows of a tile per CTA (256 per pair)
constexpr int kGroup = 8;                  // row blocks of a group of tiles, see tile_at

struct WavesParams {
  CUtensorMap map_a;        // A (K, M, batch), box 64 x 128 x 1
  CUtensorMap map_b;        // [out, in]: (K, N, batch), box 64 x BN / 2 x 1;  [in, out]: (64, K, N / 64, batch), box 64 x 64 x BN / 128 x 1,
                            // at 192 columns (N, K, batch), box 64 x 64 x 1
  void* out;                // [batch, M, N]
  const void* bias;         // [batch, N] or null
  int M, N;
  int blocks_per_batch, blocks, tiles;     // 256-row blocks; tiles of the whole result
  int per_group;            // tiles of a group of row blocks
  int steps;                // k-steps of 64
  int chunks;               // GEMM2: 256-column chunks of the hidden layer, taken in the order below (0: in order)
  int second;               // GEMM2: B is not written by the kernel ahead, its loads need not wait for that; A is, its last rows last
  int* status;
};

// The launch of an instance, tiles of 256 x bn.
template <bool BF16, int ACT, bool BIAS, bool OI>
cudaError_t launch_width(const WavesParams& p, int bn, cudaStream_t stream);

}  // namespace waves
}  // namespace ditto_b200
