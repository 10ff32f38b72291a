// Plans and launches of the tile kernel (mlp_tiles_kernel_sm100.cu): the MLP chain as two launches over tiles of one SM, with the hidden layer in scratch memory.
#include <cuda.h>

#include <algorithm>
#include <cstring>

#include "../../include/ditto_b200.h"
#include "host_util.cuh"
#include "mlp_tiles_kernel_sm100.cuh"

namespace ditto_b200 {

using namespace tiles;

namespace {

// D [batch, M, N] = act(A [batch, M, K] * B + bias)
int launch_gemm(const void* a, const void* w, void* out, const void* bias, int batch, int M, int N, int K, bool bf16,
                int w_layout, int act, bool second, const TilesGemm& g, int* status, cudaStream_t stream) {
  TilesParams p;
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
    rc = map3(&p.map_b, w, uN, static_cast<uint32_t>(g.bn));
  } else {
    // [K, N] seen as (64 columns, K, N / 64, batch): one box brings the swizzle atoms of an MN-major operand tile
    const uint64_t dims[4] = {64, uK, uN / 64, ub}, strides[3] = {uN * 2, 128, uK * uN * 2};
    const uint32_t box[4] = {64, 64, static_cast<uint32_t>(g.bn / 64), 1};
    rc = make_tensor_map(&p.map_b, bf16, w, 4, dims, strides, box);
  }
  if (rc) return rc;
  p.out = out;
  p.bias = bias;
  p.M = M;
  p.N = N;
  p.blocks_per_batch = (M + kRows - 1) / kRows;
  p.blocks = batch * p.blocks_per_batch;
  p.chunks = second ? (K + 255) / 256 : 0;
  p.steps = second ? 4 * p.chunks : (K + 63) / 64;      // (units past the hidden size read as zero)
  p.stages = std::min(kMaxStages, (g.per_sm == 2 ? kRingShared : kRingLone) / (kATile + g.bn * 128));
  p.early_b = second ? 1 : 0;
  p.status = status;
  const long long ctas = static_cast<long long>(p.blocks) * ((N + g.bn - 1) / g.bn) * g.parts;
  if (ctas > 0x7fffffffLL) return DITTO_ERR_UNSUPPORTED;
  cudaError_t e = cudaErrorInvalidValue;
#define DITTO_TILES(BF, AC, BI) \
  if (bf16 == BF && act == AC && (bias != nullptr) == BI) e = w_layout == 1 ? launch_cut<BF, AC, BI, true>(p, g, static_cast<int>(ctas), stream) : launch_cut<BF, AC, BI, false>(p, g, static_cast<int>(ctas), stream);
#define DITTO_TILES_ACTS(BF, BI) DITTO_TILES(BF, 0, BI) DITTO_TILES(BF, 1, BI) DITTO_TILES(BF, 2, BI)
  DITTO_TILES_ACTS(false, false)
  DITTO_TILES_ACTS(false, true)
  DITTO_TILES_ACTS(true, false)
  DITTO_TILES_ACTS(true, true)
#undef DITTO_TILES_ACTS
#undef DITTO_TILES
  return e == cudaSuccess ? DITTO_OK : cuda_fail("mlp tile kernel launch", e);
}

}  // namespace

size_t mlp_tiles_workspace_bytes(int batch, int M, int L) { return static_cast<size_t>(batch) * M * L * 2; }

namespace {

// Modelled time (us, without a launch's fixed part) of D [M, N] over `steps` k-steps.  Waves of tiles: a step on an SM
// with a full set of CTAs, and one of a lone CTA, which is longer where too few bytes are in flight (bn = 64; a 96 KB
// ring).  The constants are fitted to 390 timings (13 shapes of 16 to 16384 rows, each with 10 to 20 ways to cut either
// GEMM) of the kernel with four epilogue warps.  With eight, whose ends are shorter, the cut it picks is on average 3 % slower than
// the best one timed (17 shapes, ReLU and GELU with biases, before 256 columns in two parts were among the cuts), at worst 12 %: 16384 x 256, first GEMM 128 wide 30.2 us, 256 wide 26.6;
// 512 x 1024, second GEMM in eight parts of 128 columns 22.4 us, four of 64 20.0.
double tiles_time(long long blocks, int N, int steps, const TilesGemm& g) {
  const double shared = 0.109 + 0.00059 * g.bn;
  const double lone = std::max(g.per_sm == 1 ? 0.382 - 0.00333 * g.bn : -0.066 + 0.00242 * g.bn, shared);
  const double own = (steps + g.parts - 1) / g.parts, ends = 1.77 + 0.0067 * g.bn;
  const long long ctas = blocks * ((N + g.bn - 1) / g.bn) * g.parts, places = 148LL * g.per_sm;
  const long long full = ctas / places, rest = ctas % places;
  double t = g.parts > 1 ? 0.975 + 0.162 * g.parts : 0.0;
  if (g.per_sm == 1) return t + static_cast<double>(full + (rest > 0)) * (own * lone + ends);
  if (full > 0) t += static_cast<double>(full) * 2.0 * own * shared + ends;
  if (rest > 0) t += own * (lone + (2.0 * shared - lone) * std::min(1.0, std::max<long long>(0, rest - 148) / 74.0)) + ends;
  return t;
}

// (A reduction over 1024 or less is not split, as in the flow kernel: the result has the bits of the cluster kernels.)
// 256 columns in two parts, alone on their SMs (an incoming share is 128 KB), keep as many SMs busy as 128 columns unsplit do, but a
// k-step of them brings 48 KB for 512 clocks of tensor work and not 32 KB for 256: 64 of those took 376 clocks each out of L2, 32 of
// these take 565.  In a graph, us, without -> with: 2048 x 1024 -> 4096 -> 1024 34.9 -> 32.9, 1120 x 560 -> 6144 -> 1536 38.0 -> 33.1,
// 1152 x 1280 -> 5120 -> 1280 39.2 -> 35.6, 2544 x 768 -> 3072 -> 768 29.3 -> 28.6; least of those that take it for GEMM2, 3072 x 768 -> 3072
// -> 768 29.4 -> 29.8.  (Four or eight parts of 256 columns are no faster than those of 128: 256 x 1536 22.4 -> 24.9.)
// GEMM1, whose operands come from memory and whose end the second launch waits for, takes them in place of 128 columns unsplit from 96
// k-steps on only.  Operands new call after call, us, without -> with: 50 k-steps, 864 x 3200 -> 2176 -> 2048 28.8 -> 30.2, 51, 2016 x 3216 ->
// 832 -> 1024 23.0 -> 24.5, 56, 2080 x 3536 -> 768 -> 256 23.3 -> 24.8, 62, 1952 x 3936 -> 960 -> 512 25.4 -> 26.2, 88, 3248 x 5584 -> 448 ->
// 512 29.3 -> 30.0; 116, 2224 x 7424 -> 768 -> 1280 37.9 -> 36.2, 125, 1376 x 8000 -> 1472 -> 512 42.7 -> 40.1.  In place of a cut that is split
// already they win with any number: 49, 736 x 3088 -> 1920 -> 1280 27.5 -> 26.0, 83, 2224 x 5264 -> 576 -> 768 32.4 -> 29.9.
TilesGemm best_gemm(long long blocks, int N, int steps, bool first, double* time) {
  TilesGemm best = {128, 1, 2};
  *time = tiles_time(blocks, N, steps, best);
  for (int bn = 64; bn <= 256; bn += 64)
    for (int parts = 1; parts <= (bn == 128 ? 8 : bn == 64 ? 4 : bn == 256 ? 2 : 1) && (parts == 1 || steps > 16); parts *= 2)
      for (int per_sm = 1; per_sm <= (bn == 256 && parts > 1 ? 1 : 2); ++per_sm) {
        const long long ctas = blocks * ((N + bn - 1) / bn) * parts;
        // all clusters at once; alone on their SMs, large ones leave part of a GPC unused
        if (parts > 1 && ctas > (per_sm == 2 ? 296 : parts == 2 ? 148 : 112)) continue;
        if (first && bn == 256 && parts > 1 && best.parts == 1 && steps < 96) continue;
        const TilesGemm g = {bn, parts, per_sm};
        const double t = tiles_time(blocks, N, steps, g);
        if (t < *time) {
          best = g;
          *time = t;
        }
      }
  return best;
}

}  // namespace

// Where two launches over these tiles are a faster form than the flow kernel (which of them then go to the wave kernel, waves_faster says).  The flow kernel's waits cost it about 10 us a call, and it is 20 % faster
// per operation once its pairs are busy: measured, flow -> tiles, 16 x 1024 -> 4096 -> 1024 25.9 -> 16.2 us, 512 x 768 23.7 ->
// 15.2, 2048 x 1024 (34 GFLOP) 42.0 -> 37.0, 4096 x 768 (39) 46.6 -> 43.3, 2560 x 1024 (43) 50.5 -> 51.5; on the other side either is
// the faster one: 6144 x 768 (58) 53.4 -> 49.0, 4096 x 1024 (69) 60.1 -> 58.5, 1024 x 2048 (69) 64.2 -> 65.7, 16384 x 512 (69) 66.9 ->
// 73.7, 3328 x 1280 (87) 70.2 -> 71.3.  The hidden layer has to stay in L2 beside the operands.
// With GEMM2 in two parts of 256 columns the tiles win between 48 and 90 GFLOP while their operands stay in L2 (a graph of the same
// call, 3072 x 1024 (52) 53.4 -> 45.9, 1024 x 2048 (69) 65.2 -> 60.8), and lose or draw with new operands call after call, under the power cap (55.8 ->
// 58.7, 71.4 -> 71.7, 2048 x 1536 (77) 78.2 -> 83.0): the line stays.
bool mlp_tiles_faster(int batch, int M, int N, int K, int L) {
  return 2.0 * batch * M * static_cast<double>(L) * (static_cast<double>(K) + N) <= 4.8e10 &&
         mlp_tiles_workspace_bytes(batch, M, L) <= (static_cast<size_t>(48) << 20);
}

TilesPlan mlp_tiles_plan(int batch, int M, int N, int K, int L, double* time) {
  const long long blocks = static_cast<long long>(batch) * ((M + kRows - 1) / kRows);
  TilesPlan plan;
  double t1, t2;
  plan.g1 = best_gemm(blocks, L, (K + 63) / 64, true, &t1);
  plan.g2 = best_gemm(blocks, N, 4 * ((L + 255) / 256), false, &t2);
  if (time != nullptr) *time = t1 + t2;
  return plan;
}

int launch_mlp_tiles(const void* x, const void* w1, const void* w2, void* y, int batch, int M, int N, int K, int L,
                     bool bf16, int w_layout, int act1, int act2, const void* b1, const void* b2, const TilesPlan& plan,
                     void* workspace, int* status, cudaStream_t stream) {
  if (workspace == nullptr || (reinterpret_cast<uintptr_t>(workspace) & 15)) return DITTO_ERR_WORKSPACE;
  int rc = launch_gemm(x, w1, workspace, b1, batch, M, L, K, bf16, w_layout, act1, false, plan.g1, status, stream);
  // The second launch starts when every CTA of the first is past its own dependency wait: whatever wrote the weights
  // is complete by then, and the first launch does not write them.
  return rc ? rc : launch_gemm(workspace, w2, y, b2, batch, M, N, L, bf16, w_layout, act2, true, plan.g2, status, stream);
}

}  // namespace ditto_b200
