// Launch interface of the two-GEMM flow kernel (mlp_flow_sm100.cu).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace ditto_b200 {

// How a call is cut into work items; a pure function of the shape and the number of CTA pairs the device holds.
struct FlowPlan {
  int bn1, bn2;        // tile widths of the two GEMMs (128 or 256 columns; tiles are 256 rows high)
  int panel;           // 256-row blocks per panel
  int panels;          // panels in all
  int split;           // hidden ranges per GEMM2 tile in the last panels
  int split_from;      // first panel whose GEMM2 tiles are split
  int ring;            // row blocks of hidden activations the scratch memory holds
};

bool mlp_flow_supported(int N, int K, int L);
// CTA pairs of the kernel the current device holds at once (queried once per device).
int mlp_flow_pair_slots(bool bf16, int* slots);
FlowPlan mlp_flow_plan(int batch, int M, int N, int K, int L, int pair_slots);
size_t mlp_flow_workspace_bytes(int batch, int M, int N, int L, const FlowPlan& plan);
int launch_mlp_flow(const void* x, const void* w1, const void* w2, void* y, int batch, int M, int N, int K, int L,
                    bool bf16, int w_layout, int act1, int act2, const void* b1, const void* b2, const FlowPlan& plan,
                    void* workspace, int* status, cudaStream_t stream);

}  // namespace ditto_b200
