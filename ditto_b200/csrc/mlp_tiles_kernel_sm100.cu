// GEMM -> activation -> GEMM for sm_100a as two launches of one tile kernel, D = act(A B + bias), with the hidden
// layer in scratch memory (up to 48 MB stay in L2: 2048 x 1024 -> 4096 -> 1024 moves 1 MB to or from memory in both launches).
//
// For calls of few tiles the flow kernel (mlp_flow_sm100.cu) is a chain of waits: its two GEMMs hand over tile by
// tile inside one launch (8 k clocks from a hidden tile to the GEMM2 tile that reads it), a split tile's partials
// make a round trip through global memory (9 k clocks and more), and a counter reset runs in front.  Two plain
// launches cost less: the second one's CTAs are set up, and have their first weights in shared memory, before the
// first one ends (programmatic dependent launch), and a reduction that would leave SMs idle is divided between the CTAs of a
// cluster, which combine through distributed shared memory.
//
// A CTA computes one tile of 128 x bn (cta_group::1 MMAs, one accumulator in tensor memory) over its share of the
// reduction.  Roles: warps 0-7 epilogue, 8 and 9 TMA producers (A and B operands), 10 MMA issuer.  Operand stages hold
// one k-step of 64; with a ring of 96 KB two CTAs share an SM, so that one's epilogue runs under the other's MMAs,
// with 192 KB a lone CTA has enough bytes in flight to be fed at the L2 rate.
//
// What bounds it: operand bytes out of L2 -- 16 KB + bn * 128 B a k-step against the 87 B/clk per SM that TMA loads
// deliver on all SMs at once: 376 clocks at bn = 128 (256 of tensor work), 565 at 256 (512) -- and, in short calls,
// two chains of launch, first load, k-steps, epilogue.
//
// Tile width, layout of B and the number of parts are template parameters: what an issuing warp works out per k-step is then known at compile time, and a launch
// fetches the code of its own width alone (all widths behind a switch in one kernel: 1 to 3 us slower than run-time values).  A k-step of a lone
// CTA at bn = 128 took 480 clocks with run-time values.  In a graph, operands new call after call, us, before -> after: 24 shapes of 16 to 8192 rows 18.6 ->
// 17.6 (geometric mean), 512 x 768 -> 3072 -> 768 with GELU 15.5 -> 14.3, 128 x 1024 -> 4096 -> 1024 14.0 -> 12.6, 1024 x 1024 23.8 -> 22.1, 432 x 1024 -> 1856 13.9 -> 12.3; the
// number of parts (and waits out of line) 17.3 -> 16.9, 512 x 768 14.3 -> 13.7.  (A CTA's own columns of a divided tile kept in tensor memory instead of going through
// its ring: no difference.)
// Two k-steps a stage, as in the wave kernel: 1 % faster with operands in L2, 1 to 8 % slower with operands from memory.  Partial sums by bulk copies
// instead of stores to the peers: 14.2 -> 16.0.  Results written from registers in 32-byte sectors: 17.6 -> 18.0 (spills at 80 registers).
//
// The instances are compiled in eight parts (DITTO_TILES_PART: type, layout and bias), a module each: a program loads those whose kernels it calls.  All 480 in
// one took the first call of a program 21.5 ms, 2.4 in parts.
#define DITTO_WAIT_OUT_OF_LINE   // see mbar_wait
#include <atomic>

#include "host_util.cuh"
#include "mlp_common.cuh"
#include "mlp_tiles_kernel_sm100.cuh"
#include "sm100_ptx.cuh"

namespace ditto_b200 {

using namespace tiles;

namespace {

// Two epilogue warps per quarter of the rows, which take a tile's columns in turn: the read-out of the accumulator (act, bias,
// turn around, store) is a chain of 32-column pieces at the end of either launch, and half as long for it.  Four warps -> eight,
// us: 512 x 768 -> 3072 -> 768 with biases and GELU 18.1 -> 16.8, 2048 x 768 32.9 -> 31.5, 4096 x 768 54.3 -> 52.3; with
// ReLU alone, whose pieces are short, no difference (2048 x 1024 41.7).
constexpr int kEpiWarps = 8;
constexpr int kWarpA = kEpiWarps, kWarpB = kEpiWarps + 1, kWarpMma = kEpiWarps + 2;
constexpr int kThreads = (kEpiWarps + 3) * 32;
constexpr uint32_t kTmemCols = 256;              // two CTAs an SM

struct alignas(16) TilesBars {
  uint64_t full[kMaxStages], empty[kMaxStages];
  uint64_t acc_full;
  uint32_t tmem_base;
  uint32_t abort_word;
};
static_assert(sizeof(TilesBars) % 16 == 0, "the biases behind the barriers are read 16 bytes at a time");

__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z, int w) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z), "r"(w)
      : "memory");
}

// First column of k-step k.  GEMM2 adds the hidden columns in the order the four-CTA kernel adds them -- 64-column units
// dealt out over four 256-column chunks: unit e of round i is quarter e / cr of chunk 4 i + e % cr (cr chunks in the
// round) -- so that a tile whose reduction is not split has the same bits in all forms of the chain.
__device__ __forceinline__ int step_col(int k, int chunks) {
  if (chunks == 0) return k * 64;
  const int i = k >> 4, e = k & 15;
  const int cr = min(4, chunks - 4 * i);
  const int qt = cr == 4 ? e >> 2 : e / cr;
  return (4 * i + (e - qt * cr)) * 256 + qt * 64;
}

// N accumulator columns + bias (in shared memory, 16-byte aligned) -> activation -> packed words.
template <bool BF16, int ACT, bool BIAS, int N>
__device__ __forceinline__ void finish(const uint32_t (&v)[N], const uint32_t* bias, uint32_t (&w)[N / 2]) {
  if constexpr (BIAS) {
    uint32_t bw[N / 2];
#pragma unroll
    for (int i = 0; i < N / 8; ++i) {
      const uint4 t = reinterpret_cast<const uint4*>(bias)[i];
      bw[4 * i] = t.x; bw[4 * i + 1] = t.y; bw[4 * i + 2] = t.z; bw[4 * i + 3] = t.w;
    }
    act_pack_words<BF16, ACT, N>(v, bw, w);
  } else {
    act_pack_fixed<BF16, ACT, false, N>(v, nullptr, w);
  }
}

}  // namespace

template <bool BF16, int ACT, bool BIAS, int BN, bool OI, int PARTS>
__global__ void __launch_bounds__(kThreads, 2) mlp_tiles_kernel(const __grid_constant__ TilesParams p) {
  constexpr int kStage = kATile + BN * 128;
  extern __shared__ uint8_t smem_raw[];
  // the CTAs of a cluster round up by the same amount: offsets match across the cluster
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  TilesBars* bar = reinterpret_cast<TilesBars*>(smem + p.stages * kStage);
  uint32_t* bias_s = reinterpret_cast<uint32_t*>(bar + 1);
  volatile uint32_t* abort_word = &bar->abort_word;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  // clusters are consecutive CTAs; row blocks innermost, so that neighbours share weights
  const int part = PARTS == 1 ? 0 : static_cast<int>(cluster_ctarank());
  const int tile = static_cast<int>(blockIdx.x) / PARTS;
  const int n = tile / p.blocks, rb = tile - n * p.blocks;
  const int b = rb / p.blocks_per_batch;
  const int row0 = (rb - b * p.blocks_per_batch) * kRows;
  const int col0 = n * BN;
  const int k0 = p.steps * part / PARTS, k1 = p.steps * (part + 1) / PARTS;   // parts <= steps: never empty

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&bar->full[s], 1);
      mbar_init(&bar->empty[s], 1);
    }
    mbar_init(&bar->acc_full, 1);
    bar->abort_word = 0;
    fence_mbar_init();
  }
  if (warp == 0) {
    tmem_alloc(&bar->tmem_base, kTmemCols);
    tmem_relinquish();
  }
  if (warp == kWarpA && lane == 0) {
    tma_prefetch_desc(&p.map_a);
    tma_prefetch_desc(&p.map_b);
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = bar->tmem_base;

  bool ok = true;
  if (warp == kWarpB) {
    // ------------------------------------------------------------ B operand (weights)
    if (p.early_b == 0) grid_dependency_wait();
    const uint32_t issuer = elect_one();
    int st = 0;
    uint32_t ph = 1;
    for (int k = k0; k < k1; ++k) {
      ok = __all_sync(0xffffffffu, mbar_wait(&bar->empty[st], ph, abort_word, 0x110));
      if (!ok) break;
      uint8_t* dst = smem + st * kStage + kATile;
      const int kc = step_col(k, p.chunks);
      if (issuer) {
        if constexpr (OI) tma_load_3d(dst, &p.map_b, &bar->full[st], kc, col0, b);
        else tma_load_4d(dst, &p.map_b, &bar->full[st], 0, kc, col0 >> 6, b);
      }
      __syncwarp();
      if (++st == p.stages) { st = 0; ph ^= 1; }
    }
    __syncwarp();
    if (p.early_b != 0) grid_dependency_wait();
    grid_launch_dependents();
  } else {
    grid_dependency_wait();
    grid_launch_dependents();
    if (warp == kWarpA) {
      // ---------------------------------------------------------- A operand; arms the stage for both
      asm volatile("fence.proxy.async.global;" ::: "memory");   // A may be the kernel ahead's ordinary stores
      const uint32_t issuer = elect_one();
      int st = 0;
      uint32_t ph = 1;
      for (int k = k0; k < k1; ++k) {
        ok = __all_sync(0xffffffffu, mbar_wait(&bar->empty[st], ph, abort_word, 0x100));
        if (!ok) break;
        const int kc = step_col(k, p.chunks);
        if (issuer) {
          mbar_arrive_expect_tx(&bar->full[st], kStage);
          tma_load_3d(smem + st * kStage, &p.map_a, &bar->full[st], kc, row0, b);
        }
        __syncwarp();
        if (++st == p.stages) { st = 0; ph ^= 1; }
      }
    } else if (warp == kWarpMma) {
      // ---------------------------------------------------------- MMA issuer (converged warp)
      const uint32_t issuer = elect_one();
      const uint32_t ring = smem_u32(smem);
      constexpr uint32_t idesc = umma_idesc_f16(BF16, kRows, BN, false, !OI);
      constexpr uint32_t step_b = (OI ? 32 : 2048) >> 4;
      int st = 0;
      uint32_t ph = 0;
      for (int k = k0; k < k1; ++k) {
        ok = __all_sync(0xffffffffu, mbar_wait(&bar->full[st], ph, abort_word, 0x200));
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t sa = ring + st * kStage, sb = sa + kATile;
        const uint64_t da = umma_desc_sw128(sa, 16, 1024);
        const uint64_t db = OI ? umma_desc_sw128(sb, 16, 1024) : umma_desc_sw128(sb, 8192, 1024);
#pragma unroll
        for (int i = 0; i < 4; ++i)
          umma_ss_elected(tmem_base, da + ((i * 32) >> 4), db + i * step_b, idesc, (k > k0 || i > 0) ? 1u : 0u, issuer);
        umma_commit_elected(&bar->empty[st], issuer);
        if (++st == p.stages) { st = 0; ph ^= 1; }
      }
      if (ok) umma_commit_elected(&bar->acc_full, issuer);
    } else {
      // ---------------------------------------------------------- epilogue
      // The tile's biases come into shared memory while the MMAs run: read where they are added, every 32 columns were a
      // trip to L2 in the middle of the read-out.  With the packed GELU (act_apply_pair), in a graph, us, biases and GELU: 512 x 768 -> 3072
      // -> 768 16.5 -> 15.7, 2048 x 1024 -> 4096 -> 1024 37.5 -> 35.4, 4096 x 768 43.7 -> 41.6, 256 x 1536 -> 6144 -> 1536 22.7 -> 21.7.
      if constexpr (BIAS) {
        const int i = static_cast<int>(threadIdx.x);
        if (2 * i < BN)
          bias_s[i] = col0 + 2 * i < p.N ? __ldg(reinterpret_cast<const uint32_t*>(p.bias) + (static_cast<size_t>(b) * p.N + col0) / 2 + i) : 0u;
        asm volatile("bar.sync 1, %0;" ::"n"(kEpiWarps * 32) : "memory");
      }
      ok = mbar_wait(&bar->acc_full, 0, abort_word, 0x300);
      ok = __all_sync(0xffffffffu, ok);
      tc_fence_after_sync();
      if (ok && PARTS == 1) {
        // 32 columns at a time, turned around in 2 KB of the (now idle) ring per warp -- 64-byte rows of four 16-byte
        // pieces, swizzled: no bank conflicts -- so that a store instruction writes 64 contiguous bytes of eight rows
        const uint32_t acc = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16);
        uint8_t* stage = smem + warp * 2048;
        const int row = row0 + (warp & 3) * 32;
        uint8_t* to = static_cast<uint8_t*>(p.out) + (static_cast<size_t>(b) * p.M + row + (lane >> 2)) * p.N * 2 + (lane & 3) * 16;
        const int cols = min(BN, p.N - col0);          // N is a multiple of 64
#pragma unroll 1
        for (int c = (warp >> 2) * 32; c < cols; c += 64) {
          uint32_t v[32], w[16];
          tmem_ld_x32_wait(acc + c, v);
          finish<BF16, ACT, BIAS>(v, bias_s + c / 2, w);
#pragma unroll
          for (int i = 0; i < 4; ++i)
            *reinterpret_cast<uint4*>(stage + lane * 64 + ((i ^ ((lane >> 1) & 3)) << 4)) =
                make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int rr = 8 * i + (lane >> 2);
            const uint4 t = *reinterpret_cast<const uint4*>(stage + rr * 64 + (((lane & 3) ^ ((rr >> 1) & 3)) << 4));
            if (row + rr < p.M) *reinterpret_cast<uint4*>(to + static_cast<size_t>(8 * i) * p.N * 2 + (col0 + c) * 2) = t;
          }
          __syncwarp();
        }
      }
    }
  }

  if constexpr (PARTS > 1) {
    // The CTAs of the cluster hold partial sums of the same tile.  Each hands bn / parts columns of its own to every
    // CTA (into its ring, idle since the last MMA: first barrier), adds what it was given in rank order and finishes
    // those columns.  Laid out [source][four columns][row], a warp's store or load covers 512 contiguous bytes.  Every
    // thread reaches both barriers whether its waits expired or not.
    __syncwarp();
    cluster_sync_all();
    constexpr int cols = BN / PARTS;                   // 16, 32, 64 or 128
    const int row = (warp & 3) * 32 + lane;
    if (warp < kEpiWarps) {
      constexpr int cols_log2 = cols == 16 ? 4 : cols == 32 ? 5 : cols == 64 ? 6 : 7;
      const uint32_t in0 = smem_u32(smem) + (part * (cols / 4) * kRows + row) * 16;
      const uint32_t acc = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16);
#pragma unroll 1
      for (int h = (warp >> 2) * 32; h < BN; h += 64) {
        uint32_t v[32];
        tmem_ld_x32_wait(acc + h, v);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const int col = h + 4 * q;
          st_cluster_v4(map_to_cta(in0 + (col & (cols - 1)) * (kRows * 4), col >> cols_log2), __uint_as_float(v[4 * q]),
                        __uint_as_float(v[4 * q + 1]), __uint_as_float(v[4 * q + 2]), __uint_as_float(v[4 * q + 3]));
        }
      }
    }
    __syncwarp();
    cluster_sync_all();
    if (warp < kEpiWarps && row0 + row < p.M) {
      const float4* in = reinterpret_cast<const float4*>(smem) + row;
      uint8_t* to = static_cast<uint8_t*>(p.out) + (static_cast<size_t>(b) * p.M + row0 + row) * p.N * 2;
#pragma unroll 1
      for (int c = (warp >> 2) * 16; c < cols; c += 32) {
        const int col = col0 + part * cols + c;
        if (col >= p.N) break;
        float sum[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) sum[j] = 0.f;
#pragma unroll
        for (int r = 0; r < PARTS; ++r) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float4 t = in[(r * (cols / 4) + c / 4 + q) * kRows];
            sum[4 * q] += t.x; sum[4 * q + 1] += t.y; sum[4 * q + 2] += t.z; sum[4 * q + 3] += t.w;
          }
        }
        uint32_t v[16], w[8];
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = __float_as_uint(sum[j]);
        finish<BF16, ACT, BIAS>(v, bias_s + (col - col0) / 2, w);
        *reinterpret_cast<uint4*>(to + col * 2) = make_uint4(w[0], w[1], w[2], w[3]);
        *reinterpret_cast<uint4*>(to + col * 2 + 16) = make_uint4(w[4], w[5], w[6], w[7]);
      }
    }
  }

  // After a wait has given up, copies this CTA issued may still be in flight; they complete within microseconds.
  if (*abort_word != 0u) {
    for (int t = 0; t < 64; ++t) __nanosleep(1000);
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    tmem_dealloc(tmem_base, kTmemCols);
    if (lane == 0 && bar->abort_word != 0 && p.status != nullptr) atomicCAS(p.status, 0, static_cast<int>(bar->abort_word));
  }
}

// ------------------------------------------------------------------ host side
namespace {

constexpr int kBarBytes = sizeof(TilesBars) + 512, kSlack = 1024;    // (barriers, and the biases of 256 columns)

template <bool BF16, int ACT, bool BIAS, int BN, bool OI, int PARTS>
cudaError_t launch_one(const TilesParams& p, int ctas, cudaStream_t stream) {
  auto kern = mlp_tiles_kernel<BF16, ACT, BIAS, BN, OI, PARTS>;
  static std::atomic<unsigned long long> configured{0};
  int dev = 0;
  cudaError_t e = current_device_checked(&dev);
  if (e != cudaSuccess) return e;
  if (!device_configured(configured, dev)) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kRingLone + kBarBytes + kSlack);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    mark_device_configured(configured, dev);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(ctas), 1, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = static_cast<size_t>(p.stages) * (kATile + BN * 128) + kBarBytes + kSlack;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = PARTS;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = PARTS > 1 ? 2 : 1;
  return launch_kernel(cfg, kern, p);
}

}  // namespace

template <bool BF16, int ACT, bool BIAS, bool OI>
cudaError_t tiles::launch_cut(const TilesParams& p, const TilesGemm& g, int ctas, cudaStream_t stream) {
#define DITTO_CUT(BN, PARTS) \
  if (g.bn == BN && g.parts == PARTS) return launch_one<BF16, ACT, BIAS, BN, OI, PARTS>(p, ctas, stream);
  DITTO_CUT(64, 1)
  DITTO_CUT(64, 2)
  DITTO_CUT(64, 4)
  DITTO_CUT(128, 1)
  DITTO_CUT(128, 2)
  DITTO_CUT(128, 4)
  DITTO_CUT(128, 8)
  DITTO_CUT(192, 1)
  DITTO_CUT(256, 1)
  DITTO_CUT(256, 2)
#undef DITTO_CUT
  return cudaErrorInvalidValue;
}

#define DITTO_TILES(ACT) \
  template cudaError_t tiles::launch_cut<(DITTO_TILES_PART & 1) != 0, ACT, (DITTO_TILES_PART & 2) != 0, (DITTO_TILES_PART & 4) != 0>( \
      const TilesParams&, const TilesGemm&, int, cudaStream_t);
DITTO_TILES(0)
DITTO_TILES(1)
DITTO_TILES(2)
#undef DITTO_TILES

}  // namespace ditto_b200
