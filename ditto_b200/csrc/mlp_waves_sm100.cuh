// Launch interface of the wave kernel: the two GEMMs of the MLP chain as two launches over 2-SM tiles (mlp_waves_sm100.cu).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace ditto_b200 {

// Tile widths of the two GEMMs: 256 rows by 128, 192 or 256 columns.
struct WavesPlan {
  int bn1, bn2;
};

// The plan with the shortest modelled time (us, into *time): a pure function of the shape.
WavesPlan mlp_waves_plan(int batch, int M, int N, int K, int L, double* time);
// The result and the scratch memory -- the hidden activations [batch, M, L] -- are written 32 bytes at a time.
inline bool mlp_waves_aligned(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 31) == 0; }
int launch_mlp_waves(const void* x, const void* w1, const void* w2, void* y, int batch, int M, int N, int K, int L,
                     bool bf16, int w_layout, int act1, int act2, const void* b1, const void* b2, const WavesPlan& plan,
                     void* workspace, int* status, cudaStream_t stream);

}  // namespace ditto_b200
