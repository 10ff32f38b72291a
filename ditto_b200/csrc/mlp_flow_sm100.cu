// GEMM -> activation -> GEMM for sm_100a as one persistent launch over the tiles of both GEMMs:
//   Y = act2(act1(X W1 + b1) W2 + b2)
//
// The cluster kernels (mlp_wide_sm100.cu and its relatives) keep the hidden layer inside a cluster of four SMs.
// That costs them the operand reuse of a plain GEMM -- every CTA brings 48 KB per 128 x 256 x 64 step, the hidden
// tiles travel through distributed shared memory, and a result wider than 1024 columns recomputes GEMM1 -- and
// they end at 0.6 of the tensor peak.  Here the hidden layer passes through a ring of scratch memory, as long as the
// row blocks that are on their way at a time (50 MB of the 134 MB hidden layer for 16384 x 4096), and both GEMMs run on
// tiles of 256 x 256 (or 256 x 128) by CTA pairs: 2-SM MMAs with 32 KB of operands per CTA and 512 clocks of
// tensor work, against the 87 B/clk per SM that TMA loads from L2 were measured to deliver on all SMs at once.
//
// Work items, in the order they are handed out (a ticket counter in the scratch memory):
//   panel = a few 256-row blocks.  G1(0); then for each panel p: G1(p + 1), G2(p).
//   G1 item: one hidden tile, 256 rows x bn1 columns.   G2 item: one tile of Y, 256 rows x bn2 columns, over the
//   whole hidden dimension or, in the last panels, over one of `split` ranges of it (fp32 partials through
//   scratch memory, added in range order by the last range's item: deterministic).
// An item depends on items with smaller tickets only, and a ticket is drawn by a pair that is already running:
// the pairs never wait for work that cannot make progress, whatever else shares the device.  GEMM2's loads wait
// for the hidden tiles they read (a counter per row block and 1024 hidden columns), GEMM1's stores for the row
// block that used the ring slot before.  Putting a panel of GEMM1 between a hidden tile and its use keeps both
// waits short and every pair busy across the two GEMMs -- there is no tail between them.
//
// Roles per CTA (12 warps): 0-7 epilogue, 8 and 9 TMA producers (A and B operands), 10 MMA issuer (leader CTA),
// 11 ticket drawer (leader).
// Three operand stages of 64 KB (two k-steps each); two accumulators of up to 256 columns, so that one tile is written out while the
// next is multiplied.  Every epilogue warp turns 32 rows x 64 columns around in 4 KB of shared memory of its own, so
// that a store instruction writes whole 128-byte rows.
//
// Two launches over tiles (mlp_tiles_sm100.cu, mlp_waves_sm100.cu) are the faster form wherever they are possible; this one serves hidden layers
// of 512 MB and more, first GEMMs over fewer than 128 columns, results or scratch memory not aligned to 32 bytes, calls without memory for their hidden layer, and
// callers who ask for it.
//
// What bounds it: the tensor pipe under the power cap for large inputs; the chain first load -> GEMM1 tile -> hidden
// tile announced -> GEMM2 tile (about 13 us) and tile quantisation for short ones.  Measured, cluster kernel -> this one (two launches: 214 and 203, 33, 13 and 72):
//   16384 x 1024 -> 4096 -> 1024        290 -> 238 us sustained (260 -> 204 us for twenty launches)
//   2048 x 1024 -> 4096 -> 1024         59.7 -> 43 us      512 x 768 -> 3072 -> 768   53.5 -> 28 us (host-bound)
//   3328 x 1280 -> 5120 -> 1280         216 -> 87 us (no GEMM1 recomputed for a second column group)
//
// GEMM2 adds the hidden columns in the order the four-CTA kernel adds them (64-column units dealt out over four
// 256-column chunks), so an unsplit tile has the same bits in both kernels.
#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <cstring>

#include "../../include/ditto_b200.h"
#include "host_util.cuh"
#include "mlp_common.cuh"
#include "mlp_flow_sm100.cuh"
#include "sm100_ptx.cuh"

namespace ditto_b200 {

namespace {

constexpr int kRows = 128;                 // rows of a tile per CTA (256 per pair)
constexpr int kATile = 16 * 1024;          // A operand of one 64-wide k-step: 128 rows x 64
constexpr int kBTile = 16 * 1024;          // this CTA's half of the B tile of one k-step: 64 x (128 or 64)
// A stage holds two k-steps: waiting for a stage, arming it and committing it cost an issuing thread about as much
// as the four MMAs of one k-step take to execute.
constexpr int kStageSteps = 2;
constexpr int kStageBytes = kStageSteps * (kATile + kBTile);
constexpr int kStages = 6 / kStageSteps;
constexpr int kEpiWarps = 8;
constexpr int kWarpProducerA = 8, kWarpProducerB = 9, kWarpMma = 10, kWarpTicket = 11;
constexpr int kThreads = 12 * 32;
constexpr int kOffStage = kStages * kStageBytes;            // 4 KB per epilogue warp
constexpr int kOffBar = kOffStage + kEpiWarps * 4096;
constexpr int kSmemBytes = kOffBar + 512 + 1024;
static_assert(kSmemBytes <= 227 * 1024, "shared memory budget");
constexpr int kItemSlots = 4;              // items between the producer and the epilogue
constexpr int kDrawAhead = 6;              // k-steps of loads left when the next ticket is drawn (its latency: about 1.5 k clocks)
constexpr int kItemReaders = 4 + 1 + 2 * kEpiWarps;   // producers, MMA issuer, epilogue warps of the pair
constexpr int kRoundCols = 1024;           // hidden columns per readiness counter: four chunks of 256
constexpr int kRoundSteps = kRoundCols / 64;

struct FlowParams {
  CUtensorMap map_x;        // X (K, M, batch), box 64 x 128 x 1
  CUtensorMap map_w1;       // [in, out]: (64, K, L/64, batch), box 64 x 64 x bn1/128 x 1;  [out, in]: (K, L, batch), box 64 x bn1/2 x 1
  CUtensorMap map_h;        // hidden ring (L, ring * 256), box 64 x 128
  CUtensorMap map_w2;       // like map_w1 with (N, L) for (L, K)
  void* y;                  // Y [batch, M, N]
  void* hidden;             // the ring [ring * 256, L]
  const void* b1;
  const void* b2;
  float* slabs;             // fp32 partials of split tiles
  int* ticket;              // next item
  int* h_count;             // per (row block, CTA rank, round): warps that have stored their part of a hidden tile
  int* g2_done;             // per row block: GEMM2 items that have read it
  int* split_count;         // per (split tile, CTA rank, epilogue warp): partials written
  int M, N, K, L;
  int bn1, bn2, tn1, tn2;   // tile widths and tiles per row block
  int blocks_per_batch, blocks;   // 256-row blocks
  int panel, panels, split, split_from, ring;
  int rounds, steps1, steps2, chunks;
  int w_oi, act1, act2;
  int* status;
};

struct FlowBars {
  uint64_t full[kStages], empty[kStages];
  uint64_t acc_full[2], acc_empty[2];
  uint64_t item_full[kItemSlots], item_empty[kItemSlots];
  uint64_t draw;             // the leader's producer is about to run out of loads: time for the next ticket
  int item[kItemSlots];
  uint32_t tmem_base;
  uint32_t abort_word;
};
static_assert(sizeof(FlowBars) <= 512, "barrier block too large");

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
// Orders global memory accesses of the two proxies: hidden tiles are written by ordinary stores and
// read by TMA.
__device__ __forceinline__ void fence_proxy_async_global() { asm volatile("fence.proxy.async.global;" ::: "memory"); }
__device__ __forceinline__ int load_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void add_release(int* p, int v) {
  asm volatile("red.release.gpu.global.add.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// Arrival at a barrier of the pair's leader without release semantics.  What it says -- tensor memory has been read
// (tcgen05.wait::ld), a ticket has been read -- involves no memory that the leader looks at; a releasing arrival
// at cluster scope also waits for the warp's global stores (measured: 1 k clocks of the epilogue's 2.8 k per 64 columns).
__device__ __forceinline__ void arrive_leader_relaxed(uint64_t* bar) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(map_to_cta(smem_u32(bar), 0)) : "memory");
}
// One look at a barrier.  (mbarrier.try_wait may suspend the thread until the phase completes or a time limit runs out.)
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
// Position in a ring of stages whose next barrier is tested one step ahead: a ready barrier still takes an issuing
// warp 60-200 clocks to see, which this hides behind the issue of the step before.
struct RingPos {
  int st = 0;
  uint32_t ph;                  // parity that the stage's barrier is waited for
  bool ready = false;           // the test made one step ahead has succeeded
  __device__ __forceinline__ explicit RingPos(uint32_t first) : ph(first) {}
  // waits for the stage (warp-uniform), moves on and tests the next one; `st_now`: the stage to use
  __device__ __forceinline__ bool take(uint64_t* bars, volatile uint32_t* abort_word, uint32_t code, int* st_now) {
    bool ok = ready || mbar_wait(&bars[st], ph, abort_word, code);
    ok = __all_sync(0xffffffffu, ok);
    *st_now = st;
    if (++st == kStages) { st = 0; ph ^= 1; }
    ready = mbar_test(&bars[st], ph);
    return ok;
  }
};
// Bounded wait for a counter in global memory (about a second, like the barrier waits).
__device__ __forceinline__ bool wait_count(const int* p, int target, volatile uint32_t* abort_word, uint32_t code) {
  for (uint32_t spin = 0; spin < (1u << 20); ++spin) {
    if (load_acquire(p) >= target) return true;
    if (*abort_word != 0u) return false;
    if (spin > 64u) __nanosleep(64);
  }
  atomicCAS(const_cast<uint32_t*>(abort_word), 0u, code);
  return false;
}

// One work item.
struct Item {
  int gemm;        // 1, 2, or 0 past the end
  int rb;          // row block, over all batch entries
  int n;           // tile along the result's columns
  int s;           // hidden range of a split GEMM2 tile
  int split;       // ranges of this tile
};

// Turns ticket numbers (increasing) into items; keeps its place in the sequence of panels.
struct Decoder {
  int phase = -1;   // -1: G1(0); p >= 0: G1(p + 1) then G2(p)
  int base = 0;     // ticket of the phase's first item
  __device__ __forceinline__ int blocks_in(const FlowParams& p, int panel) const {
    return min(p.panel, p.blocks - panel * p.panel);
  }
  __device__ __forceinline__ Item next(const FlowParams& p, int ticket) {
    Item it;
    for (;;) {
      if (phase >= p.panels) {
        it.gemm = 0;
        it.rb = it.n = it.s = 0;
        it.split = 1;
        return it;
      }
      const int g1_panel = phase + 1;
      const int b1 = g1_panel < p.panels ? blocks_in(p, g1_panel) : 0;
      const int n1 = b1 * p.tn1;
      const int split = phase >= p.split_from ? p.split : 1;
      const int b2 = phase >= 0 ? blocks_in(p, phase) : 0;
      const int n2 = b2 * p.tn2 * split;
      int i = ticket - base;
      if (i < n1) {
        it.gemm = 1;
        it.n = i / b1;
        it.rb = g1_panel * p.panel + (i - it.n * b1);
        it.s = 0;
        it.split = 1;
        return it;
      }
      i -= n1;
      if (i < n2) {
        it.gemm = 2;
        const int j = i / b2;                       // (range, tile), row blocks innermost
        it.rb = phase * p.panel + (i - j * b2);
        it.s = j / p.tn2;
        it.n = j - it.s * p.tn2;
        it.split = split;
        return it;
      }
      base += n1 + n2;
      ++phase;
    }
  }
};

// First and last + 1 hidden unit (64 columns) of range s.
// (even: a stage holds two)
__device__ __forceinline__ int range_begin(int steps, int s, int split) { return steps / 2 * s / split * 2; }

}  // namespace

// Clears the ticket and the counters in front of the main kernel.  Launched with programmatic serialization, like
// the main kernel: that one's set-up runs under this one.
__global__ void __launch_bounds__(256) mlp_flow_reset_kernel(int* counters, int n) {
  grid_launch_dependents();
  grid_dependency_wait();                 // the scratch memory may still be in use by the kernel ahead
  for (int i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) counters[i] = 0;
}

// The epilogues known at compile time, as in mlp_wide_sm100.cu; form 0 picks them at run time.
template <int EPI> struct FlowEpilogues;
template <> struct FlowEpilogues<0> { static constexpr int act1 = 0, act2 = 0; static constexpr bool bias = false; };
template <> struct FlowEpilogues<1> { static constexpr int act1 = 1, act2 = 0; static constexpr bool bias = false; };
template <> struct FlowEpilogues<2> { static constexpr int act1 = 1, act2 = 1; static constexpr bool bias = true; };
template <> struct FlowEpilogues<3> { static constexpr int act1 = 2, act2 = 0; static constexpr bool bias = true; };
template <> struct FlowEpilogues<4> { static constexpr int act1 = 0, act2 = 0; static constexpr bool bias = false; };
template <> struct FlowEpilogues<5> { static constexpr int act1 = 1, act2 = 0; static constexpr bool bias = true; };

template <bool BF16, int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
    mlp_flow_kernel(const __grid_constant__ FlowParams p) {
  extern __shared__ uint8_t smem_raw[];
  // both CTAs of a pair round up by the same amount: offsets match across the pair
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  FlowBars* bar = reinterpret_cast<FlowBars*>(smem + kOffBar);
  volatile uint32_t* abort_word = &bar->abort_word;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();        // rows [128 rank, 128 rank + 128) of every tile; rank 0 leads

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&bar->full[s], 1);
      mbar_init(&bar->empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&bar->acc_full[a], 1);
      mbar_init(&bar->acc_empty[a], 2 * kEpiWarps);
    }
    for (int i = 0; i < kItemSlots; ++i) {
      mbar_init(&bar->item_full[i], 1);
      mbar_init(&bar->item_empty[i], kItemReaders);
    }
    mbar_init(&bar->draw, 1);
    bar->abort_word = 0;
    fence_mbar_init();
  }
  if (warp == 0) {
    tmem_alloc_pair(&bar->tmem_base, 512);
    tmem_relinquish_pair();
  }
  if (warp == kWarpProducerA && lane == 0) {
    tma_prefetch_desc(&p.map_x);
    tma_prefetch_desc(&p.map_w1);
    tma_prefetch_desc(&p.map_h);
    tma_prefetch_desc(&p.map_w2);
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();                     // both CTAs' barriers exist before anyone signals them
  tc_fence_after_sync();
  const uint32_t tmem_base = bar->tmem_base;
  // (fetch the parameters and the decoder's code before there is anything to wait for)
  {
    Decoder warm;
    const Item w = warm.next(p, warp);
    asm volatile("" ::"r"(w.rb), "r"(w.n), "r"(w.gemm));
  }
  // Programmatic dependent launch: the set-up above touches no global memory.
  grid_dependency_wait();
  grid_launch_dependents();

  // Readers of the item ring: the ticket drawn by the leader arrives in both CTAs' shared memory.
  int item_slot = 0;
  uint32_t item_par = 0;
  auto next_ticket = [&](bool* ok) -> int {      // warp-uniform
    bool r = mbar_wait_cluster(&bar->item_full[item_slot], item_par, abort_word, 0x10);
    r = __all_sync(0xffffffffu, r);
    const int t = *reinterpret_cast<volatile int*>(&bar->item[item_slot]);
    __syncwarp();
    if (r && lane == 0 && t >= 0) arrive_leader_relaxed(&bar->item_empty[item_slot]);   // (t >= 0 always: the value is here)
    if (++item_slot == kItemSlots) { item_slot = 0; item_par ^= 1; }
    *ok = r;
    return t;
  };

  if (warp == kWarpTicket) {
    // ------------------------------------------------------------ ticket drawer (leader, one thread)
    if (rank == 0 && lane == 0) {
      Decoder dec;
      uint32_t par = 1;                           // the first pass over the ring waits for nothing
      int slot = 0;
      for (int n = 0;; ++n) {
        // A ticket is drawn when the loads of the item before are nearly all issued: drawn earlier, its item would
        // sit in this pair's queue -- behind up to 30 k clocks of work -- while other pairs wait for its result.
        if (n > 0 && !mbar_wait(&bar->draw, (n - 1) & 1, abort_word, 0x21)) break;
        if (!mbar_wait_cluster(&bar->item_empty[slot], par, abort_word, 0x20)) break;
        const int t = atomicAdd(p.ticket, 1);
        for (uint32_t c = 0; c < 2; ++c) {
          const uint32_t dst = map_to_cta(smem_u32(&bar->item[slot]), c);
          asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(dst), "r"(t) : "memory");
          mbar_arrive_cluster(&bar->item_full[slot], c);
        }
        if (dec.next(p, t).gemm == 0) break;      // past the end: the readers see it and stop as well
        if (++slot == kItemSlots) { slot = 0; par ^= 1; }
      }
    }
  } else if (warp == kWarpProducerA || warp == kWarpProducerB) {
    // ------------------------------------------------------------ TMA producers (each CTA for itself)
    // One warp brings the A operand (rows of X or of the hidden ring), one the B operand (weights): a k-step costs
    // one issuing thread 670 clocks with both boxes -- more than the 512 of its MMAs -- and the weights of a GEMM2
    // item are on their way while its hidden tiles are still awaited.
    const bool is_a = warp == kWarpProducerA;
    Decoder dec;
    RingPos pos(1);                     // (the first pass over the ring waits for nothing)
    bool ok = true;
    const uint32_t full0 = map_to_cta(smem_u32(&bar->full[0]), 0);      // the leader's barriers
    const uint32_t issuer = elect_one();
    for (;;) {
      const int t = next_ticket(&ok);
      if (!ok) break;
      const Item it = dec.next(p, t);
      if (it.gemm == 0) break;
      const int b = it.rb / p.blocks_per_batch;
      const int k0 = it.gemm == 1 ? 0 : range_begin(p.steps2, it.s, it.split);
      const int k1 = it.gemm == 1 ? p.steps1 : range_begin(p.steps2, it.s + 1, it.split);
      if (is_a && it.gemm == 2) {
        // the hidden tiles this item reads must have been stored: one counter per round, polled side by side
        const int r0 = k0 / kRoundSteps, r1 = (k1 - 1) / kRoundSteps;
        const int per_round = kRoundCols / p.bn1;
        const int* count = p.h_count + (static_cast<size_t>(it.rb) * 2 + rank) * p.rounds;
        bool good = true;
        for (int r = r0 + lane; r <= r1 && good; r += 32)
          good = wait_count(count + r, min(per_round, p.tn1 - r * per_round) * kEpiWarps, abort_word, 0x30);
        ok = __all_sync(0xffffffffu, good);
        if (!ok) break;
        __syncwarp();                                      // (a vote orders no memory: the lane that polled is not the one that loads)
        fence_proxy_async_global();
      }
      // 64-column unit k of the hidden dimension in summation order: unit e of round i is quarter e / cr of chunk
      // 4 i + e % cr (cr chunks in the round)
      auto hidden_col = [&](int k) {
        const int i = k >> 4, e = k & 15;
        const int cr = min(4, p.chunks - 4 * i);
        const int qt = cr == 4 ? e >> 2 : e / cr;
        return (4 * i + (e - qt * cr)) * 256 + qt * 64;
      };
      const bool g1 = it.gemm == 1;
      const int bn = g1 ? p.bn1 : p.bn2;
      if (is_a) {
        const uint32_t bytes = 2u * (kATile + 64 * bn);      // a k-step of both CTAs: 128 x 64 of A, bn / 2 x 64 of B, 16 bits each
        const CUtensorMap* map = g1 ? &p.map_x : &p.map_h;
        const int row = (g1 ? it.rb - b * p.blocks_per_batch : it.rb % p.ring) * 256 + static_cast<int>(rank) * kRows;
        const int z = g1 ? b : 0;
        int k_draw = max(k0, k1 - kDrawAhead);
        for (int k = k0; k < k1; k += kStageSteps) {
          const bool two = kStageSteps == 2 && k + 1 < k1;
          const int col = g1 ? k * 64 : hidden_col(k), col2 = g1 ? col + 64 : hidden_col(k + 1);
          int st;
          ok = pos.take(bar->empty, abort_word, 0x100, &st);
          if (!ok) break;
          uint8_t* dst = smem + st * kStageBytes;
          if (issuer) {
            if (rank == 0) mbar_arrive_expect_tx(&bar->full[st], two ? 2 * bytes : bytes);
            tma_load_3d_pair(dst, map, full0 + st * 8, col, row, z);
            if (two) tma_load_3d_pair(dst + kATile, map, full0 + st * 8, col2, row, z);
            if (rank == 0 && k >= k_draw) mbar_arrive(&bar->draw);
          }
          if (k >= k_draw) k_draw = k1;
          __syncwarp();
        }
      } else {
        const CUtensorMap* map = g1 ? &p.map_w1 : &p.map_w2;
        const int bcol = it.n * bn + static_cast<int>(rank) * (bn / 2);      // this CTA's half of the B tile
        const bool oi = p.w_oi != 0;
        for (int k = k0; k < k1; k += kStageSteps) {
          const bool two = kStageSteps == 2 && k + 1 < k1;
          const int row = g1 ? k * 64 : hidden_col(k), row2 = g1 ? row + 64 : hidden_col(k + 1);
          int st;
          ok = pos.take(bar->empty, abort_word, 0x110, &st);
          if (!ok) break;
          uint8_t* dst = smem + st * kStageBytes + kStageSteps * kATile;
          if (issuer) {
            if (oi) {
              tma_load_3d_pair(dst, map, full0 + st * 8, row, bcol, b);
              if (two) tma_load_3d_pair(dst + kBTile, map, full0 + st * 8, row2, bcol, b);
            } else {
              tma_load_4d_pair(dst, map, full0 + st * 8, 0, row, bcol >> 6, b);
              if (two) tma_load_4d_pair(dst + kBTile, map, full0 + st * 8, 0, row2, bcol >> 6, b);
            }
          }
          __syncwarp();
        }
      }
      if (!ok) break;
    }
  } else if (warp == kWarpMma) {
    // ------------------------------------------------------------ MMA issuer (leader, converged warp)
    if (rank == 0) {
      const uint32_t issuer = elect_one();
      const uint32_t ring = smem_u32(smem);
      auto wait = [&](uint64_t* bp, uint32_t parity, uint32_t code) {
        bool r = mbar_wait(bp, parity, abort_word, code);
        r = __all_sync(0xffffffffu, r);
        tc_fence_after_sync();
        return r;
      };
      Decoder dec;
      RingPos pos(0);
      int n_item = 0;
      bool ok = true;
      for (;; ++n_item) {
        const int t = next_ticket(&ok);
        if (!ok) break;
        const Item it = dec.next(p, t);
        if (it.gemm == 0) break;
        const int bn = it.gemm == 1 ? p.bn1 : p.bn2;
        const int steps = it.gemm == 1 ? p.steps1
                                       : range_begin(p.steps2, it.s + 1, it.split) - range_begin(p.steps2, it.s, it.split);
        const uint32_t idesc = umma_idesc_f16(BF16, 256, bn, false, p.w_oi == 0);
        const int a = n_item & 1;
        const uint32_t acc = tmem_base + a * 256;
        // both CTAs' epilogue warps have read the accumulator's previous tile out
        if (n_item >= 2) {
          ok = wait(&bar->acc_empty[a], ((n_item >> 1) & 1) ^ 1, 0x200);
          if (!ok) break;
        }
        for (int k = 0; k < steps; k += kStageSteps) {
          int st;
          ok = pos.take(bar->full, abort_word, 0x210, &st);
          if (!ok) break;
          tc_fence_after_sync();
          const uint32_t sa = ring + st * kStageBytes, sb = sa + kStageSteps * kATile;
          const uint64_t da = umma_desc_sw128(sa, 16, 1024);
          const uint64_t db = p.w_oi ? umma_desc_sw128(sb, 16, 1024) : umma_desc_sw128(sb, 8192, 1024);
          const uint32_t second = k + 1 < steps ? issuer : 0u;       // (the last stage of an odd number of k-steps is half full)
#pragma unroll
          for (int s4 = 0; s4 < 4 * kStageSteps; ++s4) {
            const uint32_t offa = ((s4 / 4) * kATile + (s4 % 4) * 32) >> 4;
            const uint32_t offb = ((s4 / 4) * kBTile + (p.w_oi ? (s4 % 4) * 32 : (s4 % 4) * 2048)) >> 4;
            umma_ss_pair_elected(acc, da + offa, db + offb, idesc, (k | s4) ? 1u : 0u, s4 < 4 ? issuer : second);
          }
          umma_commit_pair_elected(&bar->empty[st], 3u, issuer);
        }
        if (!ok) break;
        umma_commit_pair_elected(&bar->acc_full[a], 3u, issuer);
      }
    }
  } else if (warp < kEpiWarps) {
    // ------------------------------------------------------------ epilogue (both CTAs, eight warps each)
    // Warp w: rows 32 (w % 4) ... + 31 (its TMEM lanes), columns [w / 4 * bn / 2, + bn / 2) of the tile.
    using E = FlowEpilogues<EPI>;
    const int half = warp >> 2;
    const int wrow = (warp & 3) * 32;
    uint8_t* stage = smem + kOffStage + warp * 4096;
    Decoder dec;
    int n_item = 0;
    bool ok = true;
    // 32 accumulator columns -> bias, activation, rounding -> 16 words
    auto finish32 = [&](const uint32_t (&v)[32], const uint32_t* bias, bool first, uint32_t (&w)[16]) __attribute__((always_inline)) {
      if constexpr (EPI == 0) {
        act_pack<BF16>(v, bias, first ? p.act1 : p.act2, w);
      } else if (first) {
        if (E::bias && bias != nullptr) act_pack_fixed<BF16, E::act1, true, 32, true>(v, bias, w);
        else act_pack_fixed<BF16, E::act1, false>(v, nullptr, w);
      } else {
        if (E::bias) act_pack_fixed<BF16, E::act2, true, 32, true>(v, bias, w);
        else act_pack_fixed<BF16, E::act2, false>(v, nullptr, w);
      }
    };
    // Announcing a hidden tile waits for its stores to complete: the warp does that behind the conversion of the next
    // tile's first columns -- or at once, when there is nothing else to do.
    int* announce = nullptr;                             // counter of the hidden tile that is not announced yet
    auto announce_now = [&]() __attribute__((always_inline)) {
      fence_proxy_async_global();                        // the hidden values are read by TMA
      __syncwarp();
      if (lane == 0) add_release(announce, 1);           // (with the warp's stores in front of it: they were ordered by __syncwarp)
      announce = nullptr;
    };
    for (;; ++n_item) {
      const int t = next_ticket(&ok);
      if (!ok) break;
      const Item it = dec.next(p, t);
      if (announce != nullptr && (it.gemm == 0 || !__all_sync(0xffffffffu, mbar_try_wait(&bar->acc_full[n_item & 1], (n_item >> 1) & 1))))
        announce_now();
      if (it.gemm == 0) break;
      const bool first = it.gemm == 1;
      const int b = it.rb / p.blocks_per_batch;
      const int bn = first ? p.bn1 : p.bn2;
      const int a = n_item & 1;
      const uint32_t acc = tmem_base + a * 256 + (static_cast<uint32_t>(wrow) << 16) + half * (bn / 2);
      const int col0 = it.n * bn + half * (bn / 2);
      const int pieces = bn / 64;                        // of 32 columns, this warp's share of the tile
      const int row = (first ? it.rb % p.ring : it.rb - b * p.blocks_per_batch) * 256 + static_cast<int>(rank) * kRows + wrow;
      ok = mbar_wait(&bar->acc_full[a], (n_item >> 1) & 1, abort_word, 0x300);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after_sync();
      if (!first && warp == 0 && rank == 0 && lane == 0) add_release(p.g2_done + it.rb, 1);
      auto release = [&]() __attribute__((always_inline)) {
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) arrive_leader_relaxed(&bar->acc_empty[a]);
      };
      // A split tile: the ranges but the last leave their fp32 partial in a slab, the last range's item -- it has the
      // largest ticket, the others are running -- waits for them and adds them in range order, its own last.  A
      // warp's share of the tile is combined by itself.
      const int others = it.split - 1;
      const size_t tile = static_cast<size_t>(it.rb - p.split_from * p.panel) * p.tn2 + it.n;
      const size_t share4 = 32 * (p.bn2 / 2) / 4;        // 16-byte pieces of a share; 16 shares in a slab
      float4* part = reinterpret_cast<float4*>(p.slabs) + (tile * others * 16 + rank * 8 + warp) * share4 + lane;
      int* count = p.split_count + (tile * 2 + rank) * 8 + warp;
      if (it.s < others) {
        float4* mine = part + it.s * 16 * share4;
#pragma unroll 1
        for (int c = 0; c < pieces; ++c) {
          uint32_t v[32];
          tmem_ld_x32_wait(acc + c * 32, v);
#pragma unroll
          for (int j = 0; j < 8; ++j)                    // one coalesced 512-byte store per four columns
            __stcg(mine + (c * 8 + j) * 32, make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]),
                                                        __uint_as_float(v[4 * j + 2]), __uint_as_float(v[4 * j + 3])));
        }
        release();
        __threadfence();
        __syncwarp();
        if (lane == 0) add_release(count, 1);
        if (announce != nullptr) announce_now();
        continue;
      }
      if (announce != nullptr && (others > 0 || (first && it.rb >= p.ring))) announce_now();   // never wait with news untold
      if (others > 0 || (first && it.rb >= p.ring)) {
        // a split tile's last range: the partials of the others; a hidden tile: the GEMM2 items that read the ring
        // slot's previous row block
        const int old = it.rb - p.ring;
        const int* what = first ? p.g2_done + old : count;
        const int target = first ? p.tn2 * (old / p.panel >= p.split_from ? p.split : 1) : others;
        if (lane == 0) ok = wait_count(what, target, abort_word, 0x310);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        __syncwarp();                                      // (as above: one lane polled, all of them load or store)
        if (first) fence_proxy_async_global();
        else __threadfence();
      }
      // 64 packed columns (two halves of 16 words) into the staging area, and from there to memory in whole 128-byte
      // rows, four per instruction.  (Not by TMA: a store queues behind the operand loads in the TMA unit and the
      // staging area came free 2 k clocks later.)
      auto stage32 = [&](int h, const uint32_t (&w)[16]) __attribute__((always_inline)) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          *reinterpret_cast<uint4*>(stage + lane * 128 + (((h * 4 + i) ^ (lane & 7)) << 4)) =
              make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
      };
      uint8_t* out_base = first ? static_cast<uint8_t*>(p.hidden) + static_cast<size_t>(row) * p.L * 2
                                : static_cast<uint8_t*>(p.y) + (static_cast<size_t>(b) * p.M + row) * p.N * 2;
      const size_t pitch = static_cast<size_t>(first ? p.L : p.N) * 2;
      const int rows = first ? 32 : min(32, p.M - row);  // rows past M are computed on zero-filled X and not stored
      auto send = [&](int col) __attribute__((always_inline)) {
        __syncwarp();
        uint8_t* to = out_base + (lane >> 3) * pitch + col * 2 + (lane & 7) * 16;
        if (!first || col < p.L) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int rr = 4 * i + (lane >> 3);
            const uint4 v = *reinterpret_cast<const uint4*>(stage + rr * 128 + (((lane & 7) ^ (rr & 7)) << 4));
            if (rr < rows) *reinterpret_cast<uint4*>(to + i * 4 * pitch) = v;
          }
        }
        __syncwarp();
      };
      if (others == 0) {
#pragma unroll 1
        for (int c = 0; c < pieces; c += 2) {
          uint32_t v[64], w0[16], w1[16];
          tmem_ld_x64_wait(acc + c * 32, v);
          if (c + 2 == pieces) release();
          const int col = col0 + c * 32;
          const uint32_t(&lo)[32] = *reinterpret_cast<const uint32_t(*)[32]>(&v[0]);
          const uint32_t(&hi)[32] = *reinterpret_cast<const uint32_t(*)[32]>(&v[32]);
          if (first) {
            // (columns past L: the bias is not read, the store is clipped)
            const uint32_t* bias = p.b1 == nullptr || col >= p.L ? nullptr
                                                                 : reinterpret_cast<const uint32_t*>(p.b1) + (static_cast<size_t>(b) * p.L + col) / 2;
            finish32(lo, bias, true, w0);
            finish32(hi, bias == nullptr ? nullptr : bias + 16, true, w1);
          } else {
            const uint32_t* bias = p.b2 == nullptr ? nullptr : reinterpret_cast<const uint32_t*>(p.b2) + (static_cast<size_t>(b) * p.N + col) / 2;
            finish32(lo, bias, false, w0);
            finish32(hi, bias == nullptr ? nullptr : bias + 16, false, w1);
          }
          stage32(0, w0);
          stage32(1, w1);
          if (announce != nullptr) announce_now();
          send(col);
        }
        if (first) announce = p.h_count + (static_cast<size_t>(it.rb) * 2 + rank) * p.rounds + it.n * p.bn1 / kRoundCols;
        continue;
      }
      // The combining item: 32 columns at a time, the loads of the next two (range, 32 columns) steps in flight.  One
      // compact loop: in a short launch these instructions run once, and fetching them is most of their cost.
      const int steps = pieces * others;
      int loaded = 0, lpiece = 0, ls = 0;
      float4 f1[8], f2[8];
      auto load = [&](float4 (&f)[8]) __attribute__((always_inline)) {
        const float4* from = part + ls * 16 * share4 + lpiece * 256;
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = __ldcg(from + j * 32);
        ++loaded;
        if (++ls == others) { ls = 0; ++lpiece; }
      };
      load(f1);
      load(f2);                                          // (pieces is even: there are at least two steps)
#pragma unroll 1
      for (int c = 0; c < pieces; ++c) {
        uint32_t v[32], w[16];
        float sum[32];
#pragma unroll
        for (int j = 0; j < 8; ++j) { sum[4 * j] = f1[j].x; sum[4 * j + 1] = f1[j].y; sum[4 * j + 2] = f1[j].z; sum[4 * j + 3] = f1[j].w; }
#pragma unroll 1
        for (int s = 1;; ++s) {
#pragma unroll
          for (int j = 0; j < 8; ++j) f1[j] = f2[j];
          if (loaded < steps) load(f2);
          if (s == others) break;                        // f1 belongs to the next piece
#pragma unroll
          for (int j = 0; j < 8; ++j) { sum[4 * j] += f1[j].x; sum[4 * j + 1] += f1[j].y; sum[4 * j + 2] += f1[j].z; sum[4 * j + 3] += f1[j].w; }
        }
        tmem_ld_x32_wait(acc + c * 32, v);
        if (c + 1 == pieces) release();
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(sum[j] + __uint_as_float(v[j]));
        const int col = col0 + c * 32;
        finish32(v, p.b2 == nullptr ? nullptr : reinterpret_cast<const uint32_t*>(p.b2) + (static_cast<size_t>(b) * p.N + col) / 2, false, w);
        stage32(c & 1, w);
        if (c & 1) send(col - 32);
      }
      if (announce != nullptr) announce_now();
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

// ------------------------------------------------------------------ host side
bool mlp_flow_supported(int N, int K, int L) { return N % 256 == 0 && L % 64 == 0 && K % 16 == 0; }

namespace {

template <bool BF16, int EPI>
cudaError_t flow_attributes() {
  return cudaFuncSetAttribute(mlp_flow_kernel<BF16, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
}

template <bool BF16>
cudaError_t flow_configure(int* slots_out) {
  static std::atomic<unsigned long long> configured{0};
  static std::atomic<int> pair_slots[kMaxDevices];
  int dev = 0;
  cudaError_t e = current_device_checked(&dev);
  if (e != cudaSuccess) return e;
  if (!device_configured(configured, dev)) {
    for (cudaError_t r : {flow_attributes<BF16, 0>(), flow_attributes<BF16, 1>(), flow_attributes<BF16, 2>(),
                          flow_attributes<BF16, 3>(), flow_attributes<BF16, 4>(), flow_attributes<BF16, 5>()})
      if (r != cudaSuccess) return r;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(256, 1, 1);
    cfg.blockDim = dim3(kThreads, 1, 1);
    cfg.dynamicSmemBytes = kSmemBytes;
    int n = 0;
    e = cudaOccupancyMaxActiveClusters(&n, mlp_flow_kernel<BF16, 0>, &cfg);
    if (e != cudaSuccess) return e;
    pair_slots[dev].store(n > 0 ? n : 1, std::memory_order_relaxed);
    mark_device_configured(configured, dev);
  }
  *slots_out = pair_slots[dev].load(std::memory_order_relaxed);
  return cudaSuccess;
}

struct FlowSizes {
  int blocks, tn1, tn2, rounds, split_blocks;
  size_t ring_bytes, slab_bytes, counters;   // counters: ints, the ticket among them
};
FlowSizes flow_sizes(int batch, int M, int N, int L, const FlowPlan& plan) {
  FlowSizes z;
  z.blocks = batch * ((M + 255) / 256);
  z.tn1 = (L + plan.bn1 - 1) / plan.bn1;
  z.tn2 = N / plan.bn2;
  z.rounds = (L + kRoundCols - 1) / kRoundCols;
  z.split_blocks = plan.split > 1 ? std::max(0, z.blocks - plan.split_from * plan.panel) : 0;
  z.ring_bytes = static_cast<size_t>(plan.ring) * 256 * L * 2;
  const size_t tiles = static_cast<size_t>(z.split_blocks) * z.tn2;
  z.slab_bytes = tiles * (plan.split - 1) * 256 * plan.bn2 * sizeof(float);   // the last range keeps its own
  z.counters = 4 + static_cast<size_t>(z.blocks) * (2 * z.rounds + 1) + tiles * 16;
  return z;
}

}  // namespace

int mlp_flow_pair_slots(bool bf16, int* slots) {
  cudaError_t e = bf16 ? flow_configure<true>(slots) : flow_configure<false>(slots);
  return e == cudaSuccess ? DITTO_OK : cuda_fail("mlp flow kernel set-up", e);
}

size_t mlp_flow_workspace_bytes(int batch, int M, int N, int L, const FlowPlan& plan) {
  const FlowSizes z = flow_sizes(batch, M, N, L, plan);
  return z.ring_bytes + z.slab_bytes + z.counters * sizeof(int);
}

namespace {

// The times at which a launch's pairs come free, in order.
constexpr int kMaxSlots = 128;
struct SlotTimes {
  double t[kMaxSlots];
  int n;
  explicit SlotTimes(int slots) : n(slots) { std::fill(t, t + n, 0.0); }
  // Hands out `count` items that take `dur` each and start at `ready` or later; returns when the last one ends.
  double place(long long count, double ready, double dur) {
    double last = 0.0;
    while (count > 0) {
      // the first c pairs come free before any of them has finished another item: one item each
      const double first = std::max(t[0], ready);
      int c = 1;
      while (c < n && c < count && t[c] <= first + dur) ++c;
      const long long rounds = c == n ? count / n : 1;
      double done[kMaxSlots];
      for (int i = 0; i < c; ++i) done[i] = std::max(t[i], ready) + static_cast<double>(rounds) * dur;
      last = std::max(last, done[c - 1]);
      count -= rounds * c;
      for (int i = 0, j = 0, k = c; i < n; ++i) t[i] = k == n || (j < c && done[j] <= t[k]) ? done[j++] : t[k++];
    }
    return last;
  }
};

// The launch's run time under a plan, in clocks: items go in ticket order to whichever pair is free first; a GEMM2
// item also waits for its panel's GEMM1.  Constants fitted to a sweep of tile widths, splits and panel sizes over
// fourteen shapes (16 to 16384 rows): the plan it picks is on average 1.6 % slower than the best of the sweep.
// A user pays for the search with the first call of a shape, so items of a kind are handed out a round at a time: 48 us a search over
// 1500 shapes (item by item 0.85 ms, up to 90 ms for long calls, with the same plan for all but two of them).
double flow_makespan(int blocks, int tn1, int tn2, int steps1, int steps2, const FlowPlan& plan, int slots) {
  auto step = [](int bn) { return bn == 256 ? 640.0 : 514.0; };
  const double fixed = 300.0, hand_over = 8000.0, end = 5000.0;
  const double partial = plan.split > 1 ? 9000.0 + 2500.0 * (plan.split - 1) * plan.bn2 / 128 : 0.0;
  SlotTimes free_at(std::min(slots, kMaxSlots));
  const double dur1 = steps1 * step(plan.bn1) + fixed, dur2 = steps2 * step(plan.bn2) + fixed;
  // the panels in the middle of a long call are all alike: the first kPanels and the last two are played through
  constexpr int kPanels = 48;
  const int panels = std::min(plan.panels, kPanels), skipped = plan.panels - panels;
  double ready = 0.0, next = 0.0, last = 0.0, half = 0.0, most = 0.0;
  for (int ph = -1; ph < panels; ++ph) {
    auto in_panel = [&](int i) { return i + 1 < panels ? plan.panel : blocks - (i + skipped) * plan.panel; };
    if (ph + 1 < panels) next = free_at.place(static_cast<long long>(in_panel(ph + 1)) * tn1, 0.0, dur1);
    if (ph >= 0) {
      const int split = ph + skipped >= plan.split_from ? plan.split : 1;
      const double dur = split > 1 ? static_cast<double>(steps2) / split * step(plan.bn2) + fixed + 2600.0 : dur2;
      last = std::max(last, free_at.place(static_cast<long long>(in_panel(ph)) * tn2 * split, ready + hand_over, dur));
      if (ph == kPanels / 3 - 1) half = last;
      if (ph == kPanels / 3 * 2 - 1) most = last;
    }
    ready = next;
  }
  return last + skipped * (most - half) / (kPanels / 3) + end + partial;
}

}  // namespace

FlowPlan mlp_flow_plan(int batch, int M, int N, int K, int L, int pair_slots) {
  struct Memo {
    int batch, M, N, K, L, slots;
    FlowPlan plan;
    bool valid;
  };
  constexpr uint32_t kMemo = 256;                         // a place by the sizes: a newer shape takes an older one's
  thread_local Memo memo[kMemo] = {};
  uint32_t h = static_cast<uint32_t>(batch);
  for (int v : {M, N, K, L, pair_slots}) h = (h ^ (h >> 15)) * 0x9E3779B1u + static_cast<uint32_t>(v);
  Memo& m = memo[(h ^ (h >> 16)) % kMemo];
  if (m.valid && m.batch == batch && m.M == M && m.N == N && m.K == K && m.L == L && m.slots == pair_slots) return m.plan;
  const int blocks = batch * ((M + 255) / 256);
  const int steps1 = (K + 63) / 64, steps2 = 4 * ((L + 255) / 256);
  FlowPlan best = {};
  double best_t = 0.0;
  // Panels are the unit of the hand-out order: small ones keep few hidden tiles alive, large ones make GEMM2 wait less.
  // The ring should stay in L2 beside the weights: half of it at most, or what panels of four blocks need.  Those are not cut:
  // with 64 MB at most GEMM1 would wait for GEMM2 tiles that take longer than the ring (measured, as it is -> cut, us:
  // 16384 x 128 -> 8192 -> 256 167 -> 341, 16384 x 256 -> 16384 -> 256 358 -> 1261, 4096 x 2048 -> 65536 -> 2048 1510 -> 1714).
  constexpr size_t kRingBytes = static_cast<size_t>(64) << 20;
  const long long wide_tiles = static_cast<long long>(blocks) * ((L + 255) / 256 + N / 256);
  // A range of a split tile is at least eight 64-column units, and a hidden size of 1024 or less is not split.
  for (int split : {1, 2, 3, 4, 6, 8}) {
    if (split > 1 && (steps2 <= kRoundSteps || steps2 / split < 8)) break;
    if (split > 3 && wide_tiles > 600) break;             // many tiles: finer ranges of the last panels change nothing
    for (int c = 0; c < 4; ++c) {
      if (c != 0 && wide_tiles > 600) break;              // ... nor do narrower tiles
      for (int panel = 4; panel <= 16; panel *= 2) {
        if (panel > 4 && panel / 2 >= blocks) break;
        FlowPlan plan = {};
        plan.bn1 = c & 2 ? 128 : 256;
        plan.bn2 = c & 1 ? 128 : 256;
        plan.panel = panel;
        plan.panels = (blocks + panel - 1) / panel;
        plan.split = split;
        plan.split_from = std::max(0, plan.panels - 2);
        // A row block's hidden tiles live from the start of its panel's GEMM1 to the end of its GEMM2: about four
        // panels of hand-out order and the time one GEMM2 tile takes, in panels.
        const int tn1 = (L + plan.bn1 - 1) / plan.bn1, tn2 = N / plan.bn2;
        const double per_panel = static_cast<double>(panel) * (static_cast<double>(tn1) * steps1 * plan.bn1 + static_cast<double>(tn2) * steps2 * plan.bn2) / pair_slots;
        plan.ring = std::min(blocks, panel * (4 + static_cast<int>(steps2 * static_cast<double>(plan.bn2) / per_panel)));
        if (panel > 4 && static_cast<size_t>(plan.ring) * 256 * L * 2 > kRingBytes) break;
        const double t = flow_makespan(blocks, tn1, tn2, steps1, steps2, plan, pair_slots);
        if (best.split == 0 || t < best_t * (split > best.split ? 0.98 : 0.99)) {
          best = plan;
          best_t = t;
        }
      }
    }
  }
  m = {batch, M, N, K, L, pair_slots, best, true};
  return best;
}

int launch_mlp_flow(const void* x, const void* w1, const void* w2, void* y, int batch, int M, int N, int K, int L,
                    bool bf16, int w_layout, int act1, int act2, const void* b1, const void* b2, const FlowPlan& plan,
                    void* workspace, int* status, cudaStream_t stream) {
  if (!mlp_flow_supported(N, K, L)) return DITTO_ERR_UNSUPPORTED;
  if (workspace == nullptr || (reinterpret_cast<uintptr_t>(workspace) & 15)) return DITTO_ERR_WORKSPACE;
  int slots = 0;
  int rc = mlp_flow_pair_slots(bf16, &slots);
  if (rc) return rc;
  const FlowSizes z = flow_sizes(batch, M, N, L, plan);
  FlowParams p;
  std::memset(&p, 0, sizeof(p));
  const uint64_t uM = M, uN = N, uK = K, uL = L, ub = batch, ur = static_cast<uint64_t>(plan.ring) * 256;
  auto map3 = [&](CUtensorMap* m, const void* base, uint64_t cols, uint64_t rows, uint64_t slices, uint32_t box_rows) {
    const uint64_t dims[3] = {cols, rows, slices}, strides[2] = {cols * 2, rows * cols * 2};
    const uint32_t box[3] = {64, box_rows, 1};
    return make_tensor_map(m, bf16, base, 3, dims, strides, box);
  };
  // [rows, cols] weights seen as (64 columns, rows, cols / 64, batch): one box brings the swizzle atoms of an
  // MN-major operand tile
  auto map4 = [&](CUtensorMap* m, const void* base, uint64_t cols, uint64_t rows, uint32_t atoms) {
    const uint64_t dims[4] = {64, rows, cols / 64, ub}, strides[3] = {cols * 2, 128, rows * cols * 2};
    const uint32_t box[4] = {64, 64, atoms, 1};
    return make_tensor_map(m, bf16, base, 4, dims, strides, box);
  };
  if ((rc = map3(&p.map_x, x, uK, uM, ub, kRows)) != DITTO_OK) return rc;
  if (w_layout == 1) {
    if ((rc = map3(&p.map_w1, w1, uK, uL, ub, plan.bn1 / 2)) != DITTO_OK) return rc;
    if ((rc = map3(&p.map_w2, w2, uL, uN, ub, plan.bn2 / 2)) != DITTO_OK) return rc;
  } else {
    if ((rc = map4(&p.map_w1, w1, uL, uK, plan.bn1 / 128)) != DITTO_OK) return rc;
    if ((rc = map4(&p.map_w2, w2, uN, uL, plan.bn2 / 128)) != DITTO_OK) return rc;
  }
  if ((rc = map3(&p.map_h, workspace, uL, ur, 1, kRows)) != DITTO_OK) return rc;
  p.y = y;
  p.hidden = workspace;
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  p.slabs = reinterpret_cast<float*>(ws + z.ring_bytes);
  p.ticket = reinterpret_cast<int*>(ws + z.ring_bytes + z.slab_bytes);
  p.g2_done = p.ticket + 4;
  p.h_count = p.g2_done + z.blocks;
  p.split_count = p.h_count + static_cast<size_t>(z.blocks) * 2 * z.rounds;
  p.M = M;
  p.N = N;
  p.K = K;
  p.L = L;
  p.bn1 = plan.bn1;
  p.bn2 = plan.bn2;
  p.tn1 = z.tn1;
  p.tn2 = z.tn2;
  p.blocks_per_batch = (M + 255) / 256;
  p.blocks = z.blocks;
  p.panel = plan.panel;
  p.panels = plan.panels;
  p.split = plan.split;
  p.split_from = plan.split > 1 ? plan.split_from : plan.panels;
  p.ring = plan.ring;
  p.rounds = z.rounds;
  p.steps1 = (K + 63) / 64;
  p.chunks = (L + 255) / 256;
  p.steps2 = 4 * p.chunks;
  p.w_oi = w_layout == 1;
  p.act1 = act1;
  p.act2 = act2;
  p.b1 = b1;
  p.b2 = b2;
  p.status = status;

  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const int counters = static_cast<int>(z.counters);
  cfg.gridDim = dim3(static_cast<unsigned>(std::min(32, (counters + 1023) / 1024)), 1, 1);
  cfg.blockDim = dim3(256, 1, 1);
  cudaError_t e = launch_kernel(cfg, mlp_flow_reset_kernel, p.ticket, counters);
  if (e != cudaSuccess) return cuda_fail("mlp flow reset launch", e);
  const long long items = static_cast<long long>(z.blocks) * (z.tn1 + static_cast<long long>(z.tn2) * plan.split);
  cfg.gridDim = dim3(static_cast<unsigned>(2 * std::min<long long>(items, slots)), 1, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = kSmemBytes;
  // the named forms read their biases 16 bytes at a time
  const bool both = b1 != nullptr && b2 != nullptr && ((reinterpret_cast<uintptr_t>(b1) | reinterpret_cast<uintptr_t>(b2)) & 15) == 0;
  const bool none = b1 == nullptr && b2 == nullptr;
  const int epi = none && act2 == 0 && act1 == 1 ? 1 : none && act2 == 0 && act1 == 0 ? 4
                  : both && act1 == 1 && act2 == 1 ? 2 : both && act1 == 2 && act2 == 0 ? 3 : both && act1 == 1 && act2 == 0 ? 5 : 0;
#define DITTO_FLOW_LAUNCH(E) \
  case E: e = bf16 ? launch_kernel(cfg, mlp_flow_kernel<true, E>, p) : launch_kernel(cfg, mlp_flow_kernel<false, E>, p); break;
  switch (epi) {
    DITTO_FLOW_LAUNCH(1)
    DITTO_FLOW_LAUNCH(2)
    DITTO_FLOW_LAUNCH(3)
    DITTO_FLOW_LAUNCH(4)
    DITTO_FLOW_LAUNCH(5)
    default: e = bf16 ? launch_kernel(cfg, mlp_flow_kernel<true, 0>, p) : launch_kernel(cfg, mlp_flow_kernel<false, 0>, p);
  }
#undef DITTO_FLOW_LAUNCH
  return e == cudaSuccess ? DITTO_OK : cuda_fail("mlp flow kernel launch", e);
}

}  // namespace ditto_b200
