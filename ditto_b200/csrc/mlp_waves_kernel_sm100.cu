// GEMM -> activation -> GEMM for sm_100a as two launches of one persistent kernel over 2-SM tiles, D = act(A B + bias), with
// the hidden layer in scratch memory.
//
// The form of calls with enough tiles to fill the device.  A pair of CTAs computes tiles of 256 x BN (BN 256, 192 or 128), tile t of
// pair q is q + t * pairs: nothing is drawn, counted or waited for inside a launch, so that the operands of a pair's next tile are on
// their way while the last k-steps of this one are multiplied.  (The flow kernel, mlp_flow_sm100.cu, hands tiles out by a ticket and lets
// GEMM2 tiles wait for hidden ones: for 16384 x 1024 -> 4096 -> 1024 its pairs stood still 0.8 us a GEMM1 tile of 6 us, and 5 us a GEMM2
// tile of 20.)  Two accumulators of BN columns: one tile is written out while the next is multiplied.
//
// Main loop.  Everything that an issuing warp works out per k-step is known at compile time (layout, tile width, stage size):
// measured alone, loads and MMAs on all SMs, 257 clocks a k-step of 128 columns and 514 of 256, which is what the tensor
// pipe takes; with those as run-time values the same loop took 338 at 128.  At 128 columns a stage holds two k-steps
// (with one it is 340-360, a stage's wait and commit take as long as its MMAs), at 256 one: seven stages in flight
// instead of three of twice the size, 16384 rows 260 -> 238 us where operands come from memory.
//
// Epilogue: every lane owns a row and writes it in whole sectors of 32 bytes, the next 32 columns on their way out of tensor memory
// meanwhile.  Against turning 32 x 64 blocks around in shared memory for 128-byte rows: 4096 x 768 -> 3072 -> 768 with GELU 39.3 -> 37.5 us, 16384
// x 1024 214 -> 200, and the 32 KB are two more stages.  (Sixteen epilogue warps: 2 % slower.)
//
// What bounds it: the tensor pipe under the power cap -- 490 to 550 clocks a k-step at 1.55 to 1.7 GHz -- and, in calls of few tiles, the
// ends of the two launches (set-up 1.0, first load 1.2, write-out of the last tile 0.7 to 3.4, teardown 0.8, hand-over 1.2 us)
// and a last wave that is not full.
//
// The instances are compiled in eight parts (DITTO_WAVES_PART: type, layout and bias), a module each: a program loads those whose kernels it calls.
#define DITTO_WAIT_OUT_OF_LINE   // see mbar_wait
#include <algorithm>
#include <atomic>

#include "host_util.cuh"
#include "mlp_common.cuh"
#include "mlp_waves_kernel_sm100.cuh"
#include "sm100_ptx.cuh"

namespace ditto_b200 {

using namespace waves;

namespace {

constexpr int kATile = 16 * 1024;          // A operand of one 64-wide k-step: 128 rows x 64
constexpr int kEpiWarps = 8;
constexpr int kWarpA = kEpiWarps, kWarpB = kEpiWarps + 1, kWarpMma = kEpiWarps + 2;
constexpr int kThreads = (kEpiWarps + 4) * 32;
constexpr int kRingBytes = 224 * 1024;
template <int BN, bool OI> struct Ring {
  static constexpr int steps = BN == 128 ? 2 : 1;                         // k-steps a stage
  // this CTA's half of the B tile of one k-step; 96 columns of an [in, out] layout come in two boxes of 64
  static constexpr int b_tile = BN == 192 && !OI ? 128 * 128 : BN * 64;
  static constexpr int stage = steps * (kATile + b_tile);
  static constexpr int stages = kRingBytes / stage;
};
constexpr int kMaxStages = 8;
constexpr int kOffBar = kRingBytes;

struct alignas(16) WavesBars {
  uint64_t full[kMaxStages], empty[kMaxStages];
  uint64_t acc_full[2], acc_empty[2];
  uint32_t tmem_base;
  uint32_t abort_word;
};
constexpr int kSmemBytes = kOffBar + sizeof(WavesBars) + 2 * 512 + 1024;
static_assert(kSmemBytes <= 227 * 1024, "shared memory budget");

__device__ __forceinline__ void tma_load_3d_pair(void* dst, const CUtensorMap* map, uint32_t bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void tma_load_4d_pair(void* dst, const CUtensorMap* map, uint32_t bar, int x, int y, int z, int w) {
  asm volatile(
      "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z), "r"(w)
      : "memory");
}
__device__ __forceinline__ void arrive_leader_relaxed(uint64_t* bar) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(map_to_cta(smem_u32(bar), 0)) : "memory");
}
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
template <int STAGES>
struct RingPos {
  int st = 0;
  uint32_t ph;                  // parity that the stage's barrier is waited for
  bool ready = false;           // the test made one step ahead has succeeded
  __device__ __forceinline__ explicit RingPos(uint32_t first) : ph(first) {}
  __device__ __forceinline__ bool take(uint64_t* bars, volatile uint32_t* abort_word, uint32_t code, int* st_now) {
    bool ok = ready || mbar_wait(&bars[st], ph, abort_word, code);
    ok = __all_sync(0xffffffffu, ok);
    *st_now = st;
    if (++st == STAGES) { st = 0; ph ^= 1; }
    ready = mbar_test(&bars[st], ph);
    return ok;
  }
};

__device__ __forceinline__ int step_col(int k, int chunks) {
  if (chunks == 0) return k * 64;
  const int i = k >> 4, e = k & 15;
  const int cr = min(4, chunks - 4 * i);
  const int qt = cr == 4 ? e >> 2 : e / cr;
  return (4 * i + (e - qt * cr)) * 256 + qt * 64;
}

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

// 32 bytes, 32-byte aligned
__device__ __forceinline__ void st_global_32(void* to, const uint32_t* w) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"l"(to), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
               : "memory");
}
// Tile t: row blocks innermost, in groups of kGroup, so that the tiles in flight share both operands (74 tiles: 8 row blocks x 9).
// GEMM2 takes the row blocks from the end, where the hidden layer was written last: of 134 MB for 16384 x 4096 what is
// still in L2 is read from there.  All row blocks innermost, from the start -> groups of 8 from the end, us: 16384 x 1024 -> 4096 -> 1024 249 -> 221,
// 2048 x 1024 35.5 -> 33.7; groups of 4 and 16 are within 1 % of 8.
struct Tile { int rb, n, b, row; };      // row block, column of tiles, batch entry, first row in it
__device__ __forceinline__ Tile tile_at(const WavesParams& p, int t) {
  const int per = p.per_group, g = t / per, r = t - g * per;
  const int gs = max(1, min(kGroup, p.blocks - g * kGroup));    // (the loops work out one tile past the end, in a group that may be empty)
  Tile x;
  x.n = r / gs;
  x.rb = g * kGroup + r - x.n * gs;
  if (p.second) x.rb = p.blocks - 1 - x.rb;
  x.b = x.rb / p.blocks_per_batch;
  x.row = (x.rb - x.b * p.blocks_per_batch) * 256;
  return x;
}

}  // namespace

template <bool BF16, int ACT, bool BIAS, int BN, bool OI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
    mlp_waves_kernel(const __grid_constant__ WavesParams p) {
  using R = Ring<BN, OI>;
  constexpr int kStageSteps = R::steps;
  extern __shared__ uint8_t smem_raw[];
  // both CTAs of a pair round up by the same amount: offsets match across the pair
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  WavesBars* bar = reinterpret_cast<WavesBars*>(smem + kOffBar);
  uint32_t* bias_s = reinterpret_cast<uint32_t*>(bar + 1);
  volatile uint32_t* abort_word = &bar->abort_word;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();        // rows [128 rank, 128 rank + 128) of every tile; rank 0 leads
  const int first_tile = static_cast<int>(blockIdx.x >> 1), tile_step = static_cast<int>(gridDim.x >> 1);

  // (barriers and tensor memory by two warps: one after the other they are 0.2 us of a launch that nothing hides)
  if (warp == kWarpMma && lane == 0) {
    for (int s = 0; s < R::stages; ++s) {
      mbar_init(&bar->full[s], 1);
      mbar_init(&bar->empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&bar->acc_full[a], 1);
      mbar_init(&bar->acc_empty[a], 2 * kEpiWarps);
    }
    bar->abort_word = 0;
    fence_mbar_init();
  }
  if (warp == 0) {
    tmem_alloc_pair(&bar->tmem_base, 512);
    tmem_relinquish_pair();
  }
  if (warp == kWarpA && lane == 0) {
    tma_prefetch_desc(&p.map_a);
    tma_prefetch_desc(&p.map_b);
  }
  const Tile first = tile_at(p, first_tile);
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();                     // both CTAs' barriers exist before anyone signals them
  tc_fence_after_sync();
  const uint32_t tmem_base = bar->tmem_base;

  if (warp == kWarpB) {
    // ------------------------------------------------------------ B operand (weights), each CTA its half of the columns
    if (p.second == 0) grid_dependency_wait();
    const uint32_t issuer = elect_one();
    const uint32_t full0 = map_to_cta(smem_u32(&bar->full[0]), 0);      // the leader's barriers
    RingPos<R::stages> pos(1);            // (the first pass over the ring waits for nothing)
    bool ok = true;
    Tile x = first;
    for (int t = first_tile; t < p.tiles && ok; t += tile_step, x = tile_at(p, t)) {
      const int b = x.b, col = x.n * BN + static_cast<int>(rank) * (BN / 2);
      for (int k = 0; k < p.steps; k += kStageSteps) {
        int st;
        ok = pos.take(bar->empty, abort_word, 0x110, &st);
        if (!ok) break;
        uint8_t* dst = smem + st * R::stage + kStageSteps * kATile;
        if (issuer) {
#pragma unroll
          for (int j = 0; j < kStageSteps; ++j) {
            if (j == 0 || k + j < p.steps) {
              const int row = step_col(k + j, p.chunks);
              if constexpr (OI) {
                tma_load_3d_pair(dst + j * R::b_tile, &p.map_b, full0 + st * 8, row, col, b);
              } else if constexpr (BN == 192) {
                tma_load_3d_pair(dst, &p.map_b, full0 + st * 8, col, row, b);
                tma_load_3d_pair(dst + 64 * 128, &p.map_b, full0 + st * 8, col + 64, row, b);
              } else {
                tma_load_4d_pair(dst + j * R::b_tile, &p.map_b, full0 + st * 8, 0, row, col >> 6, b);
              }
            }
          }
        }
        __syncwarp();
      }
    }
    if (p.second != 0) grid_dependency_wait();
    grid_launch_dependents();
  } else {
    grid_dependency_wait();
    grid_launch_dependents();
    if (warp == kWarpA) {
      // ---------------------------------------------------------- A operand, each CTA its rows; the leader arms the stage for both
      asm volatile("fence.proxy.async.global;" ::: "memory");   // A may be the kernel ahead's ordinary stores
      const uint32_t issuer = elect_one();
      const uint32_t full0 = map_to_cta(smem_u32(&bar->full[0]), 0);
      RingPos<R::stages> pos(1);
      bool ok = true;
      Tile x = first;
      for (int t = first_tile; t < p.tiles && ok; t += tile_step, x = tile_at(p, t)) {
        const int b = x.b, row = x.row + static_cast<int>(rank) * kRows;
        for (int k = 0; k < p.steps; k += kStageSteps) {
          int st;
          ok = pos.take(bar->empty, abort_word, 0x100, &st);
          if (!ok) break;
          uint8_t* dst = smem + st * R::stage;
          const uint32_t bytes = 2u * (kATile + R::b_tile) * static_cast<uint32_t>(min(kStageSteps, p.steps - k));
          if (issuer) {
            if (rank == 0) mbar_arrive_expect_tx(&bar->full[st], bytes);
#pragma unroll
            for (int j = 0; j < kStageSteps; ++j)
              if (j == 0 || k + j < p.steps) tma_load_3d_pair(dst + j * kATile, &p.map_a, full0 + st * 8, step_col(k + j, p.chunks), row, b);
          }
          __syncwarp();
        }
      }
    } else if (warp == kWarpMma) {
      // ---------------------------------------------------------- MMA issuer (leader, converged warp)
      if (rank == 0) {
        const uint32_t issuer = elect_one();
        const uint32_t ring = smem_u32(smem);
        const uint32_t idesc = umma_idesc_f16(BF16, 256, BN, false, !OI);
        constexpr uint32_t step_b = (OI ? 32 : 2048) >> 4;
        RingPos<R::stages> pos(0);
        bool ok = true;
        int i = 0;
        for (int t = first_tile; t < p.tiles && ok; t += tile_step, ++i) {
          const int a = i & 1;
          const uint32_t acc = tmem_base + a * 256;
          if (i >= 2) {                   // both CTAs' epilogue warps have read the accumulator's previous tile out
            ok = mbar_wait(&bar->acc_empty[a], ((i >> 1) & 1) ^ 1, abort_word, 0x200);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after_sync();
          }
          for (int k = 0; k < p.steps; k += kStageSteps) {
            int st;
            ok = pos.take(bar->full, abort_word, 0x210, &st);
            if (!ok) break;
            tc_fence_after_sync();
            const uint32_t sa = ring + st * R::stage, sb = sa + kStageSteps * kATile;
            const uint64_t da = umma_desc_sw128(sa, 16, 1024);
            const uint64_t db = OI ? umma_desc_sw128(sb, 16, 1024) : umma_desc_sw128(sb, 8192, 1024);
#pragma unroll
            for (int s4 = 0; s4 < 4 * kStageSteps; ++s4) {
              const uint32_t on = s4 < 4 || k + s4 / 4 < p.steps ? issuer : 0u;       // (the last stage may be half full)
              umma_ss_pair_elected(acc, da + (((s4 / 4) * kATile + (s4 % 4) * 32) >> 4), db + (((s4 / 4) * R::b_tile) >> 4) + (s4 % 4) * step_b,
                                   idesc, (k | s4) ? 1u : 0u, on);
            }
            umma_commit_pair_elected(&bar->empty[st], 3u, issuer);
          }
          if (!ok) break;
          umma_commit_pair_elected(&bar->acc_full[a], 3u, issuer);
        }
      }
    } else if (warp < kEpiWarps) {
      // ---------------------------------------------------------- epilogue (both CTAs, eight warps each)
      // Warp w: rows 32 (w % 4) ... + 31 (its TMEM lanes), columns [w / 4 * kCols, + kCols) of the tile.
      constexpr int kCols = BN / (kEpiWarps / 4);
      const int part = (warp >> 2) * kCols;
      const int wrow = (warp & 3) * 32;
      int i = 0;
      Tile x = first;
      for (int t = first_tile; t < p.tiles; t += tile_step, x = tile_at(p, t), ++i) {
        const int a = i & 1;
        const int n = x.n, b = x.b, row = x.row + static_cast<int>(rank) * kRows + wrow;
        uint32_t* bias = bias_s + a * 128;
        if constexpr (BIAS) {
          const int c = static_cast<int>(threadIdx.x), col = n * BN + 2 * c;
          if (2 * c < BN) bias[c] = col < p.N ? __ldg(reinterpret_cast<const uint32_t*>(p.bias) + (static_cast<size_t>(b) * p.N + col) / 2) : 0u;
          asm volatile("bar.sync 1, %0;" ::"n"(kEpiWarps * 32) : "memory");
        }
        bool ok = mbar_wait(&bar->acc_full[a], (i >> 1) & 1, abort_word, 0x300);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok && !BIAS) break;          // (with biases the warps meet at a barrier: all of them go on, and store nothing)
        tc_fence_after_sync();
        const uint32_t acc = tmem_base + a * 256 + (static_cast<uint32_t>(wrow) << 16) + part;
        const bool stores = ok && row + lane < p.M;           // rows past M are computed on zero-filled A and not stored
        uint8_t* out_row = static_cast<uint8_t*>(p.out) + (static_cast<size_t>(b) * p.M + row + lane) * p.N * 2;
        // 32 columns at a time, the next 32 on their way out of tensor memory meanwhile
        uint32_t v[2][32];
        tmem_ld_x32(acc, v[0]);
#pragma unroll
        for (int c = 0; c < kCols; c += 32) {
          uint32_t (&u)[32] = v[(c / 32) & 1];
          uint32_t w[16];
          tmem_wait_ld(u);
          if (c + 32 < kCols) {
            tmem_ld_x32(acc + c + 32, v[(c / 32 + 1) & 1]);
          } else {
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) arrive_leader_relaxed(&bar->acc_empty[a]);
          }
          finish<BF16, ACT, BIAS>(u, bias + (part + c) / 2, w);
          const int col = n * BN + part + c;      // (N is a multiple of 64)
          if (stores && col < p.N) {
            uint8_t* to = out_row + static_cast<size_t>(col) * 2;
            st_global_32(to, w);
            st_global_32(to + 32, w + 8);
          }
        }
      }
    }
  }

  // After a wait has given up, copies this CTA issued may still be in flight; they complete within microseconds.
  if (*abort_word != 0u) {
    for (int t = 0; t < 64; ++t) __nanosleep(1000);
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();                     // no CTA leaves while the other may still signal it
  if (warp == 0) {
    tmem_dealloc_pair(tmem_base, 512);
    if (lane == 0 && bar->abort_word != 0 && p.status != nullptr) atomicCAS(p.status, 0, static_cast<int>(bar->abort_word));
  }
}

// ------------------------------------------------------------------ launcher
namespace {

template <bool BF16, int ACT, bool BIAS, int BN, bool OI>
cudaError_t launch_one(const WavesParams& p, cudaStream_t stream) {
  auto kern = mlp_waves_kernel<BF16, ACT, BIAS, BN, OI>;
  static std::atomic<unsigned long long> configured{0};
  static std::atomic<int> pair_slots[kMaxDevices];
  int dev = 0;
  cudaError_t e = current_device_checked(&dev);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(256, 1, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = kSmemBytes;
  cfg.stream = stream;
  if (!device_configured(configured, dev)) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
    if (e != cudaSuccess) return e;
    int n = 0;
    e = cudaOccupancyMaxActiveClusters(&n, kern, &cfg);
    if (e != cudaSuccess) return e;
    pair_slots[dev].store(n > 0 ? n : 1, std::memory_order_relaxed);
    mark_device_configured(configured, dev);
  }
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cfg.gridDim = dim3(static_cast<unsigned>(2 * std::min(p.tiles, pair_slots[dev].load(std::memory_order_relaxed))), 1, 1);
  return launch_kernel(cfg, kern, p);
}

}  // namespace

template <bool BF16, int ACT, bool BIAS, bool OI>
cudaError_t waves::launch_width(const WavesParams& p, int bn, cudaStream_t stream) {
  return bn == 256 ? launch_one<BF16, ACT, BIAS, 256, OI>(p, stream) : bn == 192 ? launch_one<BF16, ACT, BIAS, 192, OI>(p, stream) : launch_one<BF16, ACT, BIAS, 128, OI>(p, stream);
}

#define DITTO_WAVES(ACT) \
  template cudaError_t waves::launch_width<(DITTO_WAVES_PART & 1) != 0, ACT, (DITTO_WAVES_PART & 2) != 0, (DITTO_WAVES_PART & 4) != 0>( \
      const WavesParams&, int, cudaStream_t);
DITTO_WAVES(0)
DITTO_WAVES(1)
DITTO_WAVES(2)
#undef DITTO_WAVES

}  // namespace ditto_b200
