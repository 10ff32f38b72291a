// Plans and launches of the wave kernel (mlp_waves_kernel_sm100.cu): the MLP chain as two launches over 2-SM tiles, with the hidden layer in scratch memory.
#include <cuda.h>

#include <algorithm>
#include <cstring>

#include "../../include/ditto_b200.h"
#include "host_util.cuh"
#include "mlp_waves_kernel_sm100.cuh"

namespace ditto_b200 {

using namespace waves;

namespace {

// D [batch, M, N] = act(A [batch, M, K] * B + bias)
int launch_gemm(const void* a, const void* w, void* out, const void* bias, int batch, int M, int N, int K, bool bf16,
                int w_layout, int act, bool second, int bn, int* status, cudaStream_t stream) {
  WavesParams p;
  std::memset(&p, 0, sizeof(p));
  const uint64_t uM = M, uN = N, uK = K, ub = batch;
  auto map3 = [&](CUtensorMap* m, const void* base, uint64_t rows, uint32_t box_rows) {
    const uint64_t dims[3] = {uK, rows, ub}, strides[2] = {uK * 2, rows * uK * 2};
    const uint32_t box[3] = {64, box_rows, 1};
    return make_tensor_map(m, bf16, base, 3, dims, strides, box);
  };
  int rc = map3(&p.map_a, a, uM, kRows);
  if (rc) return rc;
  if (w_layout == 1) {
    rc = map3(&p.map_b, w, uN, static_cast<uint32_t>(bn / 2));
  } else if (bn == 192) {
    const uint64_t dims[3] = {uN, uK, ub}, strides[2] = {uN * 2, uK * uN * 2};
    const uint32_t box[3] = {64, 64, 1};
    rc = make_tensor_map(&p.map_b, bf16, w, 3, dims, strides, box);
  } else {
    // [K, N] seen as (64 columns, K, N / 64, batch): one box brings the swizzle atoms of an MN-major operand tile
    const uint64_t dims[4] = {64, uK, uN / 64, ub}, strides[3] = {uN * 2, 128, uK * uN * 2};
    const uint32_t box[4] = {64, 64, static_cast<uint32_t>(bn / 128), 1};
    rc = make_tensor_map(&p.map_b, bf16, w, 4, dims, strides, box);
  }
  if (rc) return rc;
  p.out = out;
  p.bias = bias;
  p.M = M;
  p.N = N;
  p.blocks_per_batch = (M + 255) / 256;
  p.blocks = batch * p.blocks_per_batch;
  const long long tiles = static_cast<long long>(p.blocks) * ((N + bn - 1) / bn);
  if (tiles > 0x3fffffffLL) return DITTO_ERR_UNSUPPORTED;
  p.tiles = static_cast<int>(tiles);
  p.per_group = kGroup * ((N + bn - 1) / bn);
  p.chunks = second ? (K + 255) / 256 : 0;
  p.steps = second ? 4 * p.chunks : (K + 63) / 64;      // (units past the hidden size read as zero)
  p.second = second ? 1 : 0;
  p.status = status;
  cudaError_t e = cudaErrorInvalidValue;
#define DITTO_WAVES(BF, AC, BI) \
  if (bf16 == BF && act == AC && (bias != nullptr) == BI) \
    e = w_layout == 1 ? launch_width<BF, AC, BI, true>(p, bn, stream) : launch_width<BF, AC, BI, false>(p, bn, stream);
#define DITTO_WAVES_ACTS(BF, BI) DITTO_WAVES(BF, 0, BI) DITTO_WAVES(BF, 1, BI) DITTO_WAVES(BF, 2, BI)
  DITTO_WAVES_ACTS(false, false)
  DITTO_WAVES_ACTS(false, true)
  DITTO_WAVES_ACTS(true, false)
  DITTO_WAVES_ACTS(true, true)
#undef DITTO_WAVES_ACTS
#undef DITTO_WAVES
  return e == cudaSuccess ? DITTO_OK : cuda_fail("mlp wave kernel launch", e);
}

}  // namespace

// Modelled time (us) of D [M, N] over `steps` k-steps in tiles of 256 x bn: whole rounds of 74 pairs.  Fitted to 198 shapes of the
// chain (16 to 65536 rows, all nine plans each; operands new call after call, under the power cap and in bursts): 8 % off (standard deviation); the
// plan it picks is 0.3 to 0.9 % slower than the best of the nine.
// 192 columns are for rounds that 256 would leave half empty: GEMM2 of 4096 x 768 -> 3072 -> 768 is 64 tiles of 192 columns or 48 of 256, for 74 pairs
// either way: 36.6 -> 32.8 us, under the power cap 40.5 -> 38.6; [in, out] weights, of which 128 columns are read for 96, 35.3 -> 31.9 and 38.4 -> 37.4.
// (Widths as run-time values of one kernel cost 256 columns 4 %.  The last round's tiles in halves of 128 columns, 16384 x 1024 -> 4096 -> 1024: 210 -> 210.)
static double waves_time(long long blocks, int N, int steps, int bn) {
  const long long tiles = blocks * ((N + bn - 1) / bn);
  const double step = bn == 256 ? 0.310 : bn == 192 ? 0.254 : 0.198, end = bn == 256 ? 2.3 : bn == 192 ? 1.6 : 1.1;
  return static_cast<double>((tiles + 73) / 74) * (steps * step + 1.83) + end;
}

WavesPlan mlp_waves_plan(int batch, int M, int N, int K, int L, double* time) {
  const long long blocks = static_cast<long long>(batch) * ((M + 255) / 256);
  auto best = [&](int columns, int steps) {
    int width = 256;
    double least = waves_time(blocks, columns, steps, 256);
    for (int bn : {192, 128}) {
      const double t = waves_time(blocks, columns, steps, bn);
      if (t < least) {
        least = t;
        width = bn;
      }
    }
    *time += least;
    return width;
  };
  *time = 0.0;
  WavesPlan plan;
  plan.bn1 = best(L, (K + 63) / 64);
  plan.bn2 = best(N, 4 * ((L + 255) / 256));
  return plan;
}

int launch_mlp_waves(const void* x, const void* w1, const void* w2, void* y, int batch, int M, int N, int K, int L,
                     bool bf16, int w_layout, int act1, int act2, const void* b1, const void* b2, const WavesPlan& plan,
                     void* workspace, int* status, cudaStream_t stream) {
  if (workspace == nullptr || !mlp_waves_aligned(workspace)) return DITTO_ERR_WORKSPACE;
  if (!mlp_waves_aligned(y)) return DITTO_ERR_INVALID_ARG;
  int rc = launch_gemm(x, w1, workspace, b1, batch, M, L, K, bf16, w_layout, act1, false, plan.bn1, status, stream);
  // The second launch starts when every CTA of the first is past its own dependency wait: whatever wrote the weights
  // is complete by then, and the first launch does not write them.
  return rc ? rc : launch_gemm(workspace, w2, y, b2, batch, M, N, L, bf16, w_layout, act2, true, plan.bn2, status, stream);
}

}  // namespace ditto_b200
