// What the tile kernel's instances (mlp_tiles_kernel_sm100.cu) and the code that plans and launches them (mlp_tiles_sm100.cu) share.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include "mlp_tiles_sm100.cuh"

namespace ditto_b200 {
namespace tiles {

constexpr int kRows = 128;
constexpr int kATile = 16 * 1024;                // 128 rows x 64
constexpr int kMaxStages = 8;
constexpr int kRingLone = 192 * 1024, kRingShared = 96 * 1024;

struct TilesParams {
  CUtensorMap map_a;        // A (K, M, batch), box 64 x 128 x 1
  CUtensorMap map_b;        // [out, in]: (K, N, batch), box 64 x bn x 1;  [in, out]: (64, K, N / 64, batch), box 64 x 64 x bn / 64 x 1
  void* out;                // [batch, M, N]
  const void* bias;         // [batch, N] or null
  int M, N;
  int blocks_per_batch, blocks;         // 128-row blocks
  int steps;                // k-steps of 64
  int chunks;               // GEMM2: 256-column chunks of the hidden layer, taken in the order below (0: in order)
  int stages;
  int early_b;              // B is not written by the kernel ahead: its loads need not wait for that
  int* status;
};

// The launch of an instance with the cut g.
template <bool BF16, int ACT, bool BIAS, bool OI>
cudaError_t launch_cut(const TilesParams& p, const TilesGemm& g, int ctas, cudaStream_t stream);

}  // namespace tiles
}  // namespace ditto_b200
