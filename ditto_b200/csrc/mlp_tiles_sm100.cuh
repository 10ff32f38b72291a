// Launch interface of the tile kernel: the two GEMMs of the MLP chain as two launches (mlp_tiles_sm100.cu).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stddef.h>

namespace ditto_b200 {

// How one GEMM is cut: tiles of 128 x bn by clusters of `parts` CTAs that divide the reduction between them.
struct TilesGemm {
  int bn;              // 64, 128, 192 or 256
  int parts;           // 1, 2, 4 or 8; above 1: bn is 128 (64: at most 4; 256: 2, one CTA an SM), so that an incoming share fits the operand ring
  int per_sm;          // CTAs an SM holds: 1 (a ring of 192 KB) or 2 (96 KB)
};
struct TilesPlan {
  TilesGemm g1, g2;
};

// Whether this form is expected to be faster than the flow kernel, and its plan (with its modelled time in us, without the launches'
// fixed parts): pure functions of the shape.
bool mlp_tiles_faster(int batch, int M, int N, int K, int L);
TilesPlan mlp_tiles_plan(int batch, int M, int N, int K, int L, double* time = nullptr);
// The hidden activations [batch, M, L].
size_t mlp_tiles_workspace_bytes(int batch, int M, int L);
int launch_mlp_tiles(const void* x, const void* w1, const void* w2, void* y, int batch, int M, int N, int K, int L,
                     bool bf16, int w_layout, int act1, int act2, const void* b1, const void* b2, const TilesPlan& plan,
                     void* workspace, int* status, cudaStream_t stream);

}  // namespace ditto_b200
