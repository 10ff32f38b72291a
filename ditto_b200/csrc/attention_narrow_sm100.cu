// Fused bmm -> softmax -> bmm for head dimensions up to 64 and many short items: 64-key blocks, one small CTA an item.
//
// A short item spends most of its life outside its blocks: launch and set-up, first loads, write-out.  The work loop of
// attention_persistent_sm100.cu hides some of that, with two CTAs of six warps, 80 KB and 256 tensor-memory columns an SM and
// 128-key blocks.  Here a CTA needs 128 columns (S 64, overwritten by P; O 64), 50 KB of shared memory and five warps of
// at most 96 registers, so that the next CTA is set up while others work, a padded last block wastes at most 48 keys
// and not 112, and the first P*V starts after 64 exponentials a row.  The price is twice the hand-overs per key, which is why
// long items, and few ones, stay on the other kernels (see attention_narrow_pays).
//
// Roles: warps 0-3 softmax and write-out (thread r <-> query row r <-> TMEM lane r), warp 4 loads and MMAs.  One control
// warp suffices because the order of events is fixed: S(g) complete frees K's stage and (S(g) is issued behind
// P*V(g-1), and a commit covers all earlier MMAs) V's stage of block g - 1, so the loads need no "empty" barriers.
#define DITTO_WAIT_OUT_OF_LINE   // see mbar_wait
#include "attention_sm100.cuh"

#include <atomic>

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "host_util.cuh"
#include "mlp_common.cuh"
#include "sm100_ptx.cuh"
#include "softmax_step.cuh"

namespace ditto_b200 {

namespace {

constexpr int kBM = 128, kBN = 64, kD = 64;
constexpr int kTileQ = kBM * kD * 2;      // 16 KB
constexpr int kTileKV = kBN * kD * 2;     // 8 KB
constexpr int kOffQ = 0;
constexpr int kOffK = kOffQ + kTileQ;     // two stages each
constexpr int kOffV = kOffK + 2 * kTileKV;
constexpr int kOffBar = kOffV + 2 * kTileKV;
constexpr int kSmemBytes = kOffBar + 128 + 1024;
// For as many items as three CTAs an SM take (an SM's 228 KB hold one KB more a CTA), see launch_n.
constexpr int kSmemBytesThree = 75 * 1024;
constexpr int kThreads = 160;
constexpr uint32_t kTmemCols = 128;
constexpr uint32_t kColO = 64;
// What the close references (softmax_step.cuh) do here: with blocks half as long as in the other kernels a reference is stale more
// often.  Error against float64, other kernels / this one with 8 throughout / this one: 2.88e-4 / 2.90e-4 / 2.88e-4 for fp16 rows of
// 512 keys at scale d^-0.5, 2.19e-4 / 2.28e-4 / 2.15e-4 unscaled; 144 keys at 0.35, simulated, 2.33e-4 / 2.60e-4 / 2.29e-4.
// The price is about one rescale an item, 56.4 -> 58.2 us for 2048 items of 512 keys, 7.5 -> 8.0 for one wave of 304; all
// of O in one piece, or the rescale behind P, spill or delay every item (65.6 and 59.0 us).

// Some weights are computed on the multiply-add pipe (weights_on_fma).  Four softmax warps on a scheduler keep the special-function unit
// 63 % busy over a long launch and issue in half of the slots; a tenth of the exponentials elsewhere is what pays, beyond that the
// longer instruction stream, and the clock under the power it takes, cost more.  Scalar arithmetic / packed with 1 / 2 / 3 / 4 of 32
// pairs there, us, at the power cap: 16 slices of 8192 x 8192 405 / 391.6 / 389.5 / 388.9 / 389.7, 64 of 2048 x 2048 107.0 / 104.4 / 103.6 /
// 103.4 / 103.4, 512 of 512 x 512 66.4 / 64.5 / 64.5 / 65.1 / 65.5, 1024 of 208 x 208 41.6 / 40.3 / 40.3 / 40.8 / 41.0.
constexpr int kModeSoftmax = 0, kModeRelu = 1;

struct NBars {
  uint64_t q_full, k_full[2], v_full[2], s_full, p_full, o_done;
  uint32_t tmem_base;
  uint32_t abort_word;
};
static_assert(sizeof(NBars) <= 128, "barrier block too large");

}  // namespace

template <bool BF16, int MODE>
__global__ void __launch_bounds__(kThreads, 4) attention_narrow_kernel(const __grid_constant__ AttnParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  NBars* bar = reinterpret_cast<NBars*>(smem + kOffBar);
  volatile uint32_t* abort_word = &bar->abort_word;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int tiles = (p.M + kBM - 1) / kBM;
  const int nkv = (p.L + kBN - 1) / kBN;
  // tile index fastest: the tiles of a slice run together and share its K/V in L2
  const int slice = static_cast<int>(blockIdx.x) / tiles;
  const int m0 = (static_cast<int>(blockIdx.x) - slice * tiles) * kBM;
  const int seq = slice / p.heads;
  const int head_col = (slice - seq * p.heads) * p.d;

  if (threadIdx.x == 0) {
    mbar_init(&bar->q_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bar->k_full[s], 1);
      mbar_init(&bar->v_full[s], 1);
    }
    mbar_init(&bar->s_full, 1);
    mbar_init(&bar->p_full, kBM);
    mbar_init(&bar->o_done, 1);
    bar->abort_word = 0;
    fence_mbar_init();
  }
  if (warp == 0) {
    tmem_alloc(&bar->tmem_base, kTmemCols);
    tmem_relinquish();
  }
  if (warp == 4 && lane == 0) {
    tma_prefetch_desc(&p.map_q);
    tma_prefetch_desc(&p.map_k);
    tma_prefetch_desc(&p.map_v);
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = bar->tmem_base;
  // Programmatic dependent launch: nothing above touches global memory.
  grid_dependency_wait();
  grid_launch_dependents();

  if (warp == 4) {
    // ------------------------------------------------------------ loads and MMAs (converged warp, elected lane issues)
    const uint32_t issuer = elect_one();
    const bool kt = p.k_transposed != 0, vt = p.v_transposed != 0;
    const int ksteps_d = p.d / 16;
    const uint32_t idesc_s = umma_idesc_f16(BF16, kBM, kBN, false, kt);
    const uint32_t idesc_o = umma_idesc_f16(BF16, kBM, kD, false, !vt);
    const uint64_t dq = umma_desc_sw128(smem_u32(smem + kOffQ), 16, 1024);
    // one 64-wide atom in either direction: MN-major operands have no second atom to lead to
    const uint64_t dk0 = kt ? umma_desc_sw128(smem_u32(smem + kOffK), kTileKV, 1024) : umma_desc_sw128(smem_u32(smem + kOffK), 16, 1024);
    const uint64_t dv0 = vt ? umma_desc_sw128(smem_u32(smem + kOffV), 16, 1024) : umma_desc_sw128(smem_u32(smem + kOffV), kTileKV, 1024);
    const uint32_t step_k = kt ? 2048u >> 4 : 32u >> 4, step_v = vt ? 32u >> 4 : 2048u >> 4;
    auto load_k = [&](int g) {
      if (issuer) {
        uint8_t* dst = smem + kOffK + (g & 1) * kTileKV;
        mbar_arrive_expect_tx(&bar->k_full[g & 1], kTileKV);
        if (kt) tma_load_3d(dst, &p.map_k, &bar->k_full[g & 1], g * kBN, 0, slice);
        else tma_load_3d(dst, &p.map_k, &bar->k_full[g & 1], p.k_col0 + head_col, g * kBN, seq);
      }
      __syncwarp();
    };
    auto load_v = [&](int g) {
      if (issuer) {
        uint8_t* dst = smem + kOffV + (g & 1) * kTileKV;
        mbar_arrive_expect_tx(&bar->v_full[g & 1], kTileKV);
        if (vt) tma_load_3d(dst, &p.map_v, &bar->v_full[g & 1], g * kBN, 0, slice);
        else tma_load_3d(dst, &p.map_v, &bar->v_full[g & 1], p.v_col0 + head_col, g * kBN, seq);
      }
      __syncwarp();
    };
    auto wait = [&](uint64_t* b, uint32_t parity, uint32_t code) {
      bool r = mbar_wait(b, parity, abort_word, code);
      r = __all_sync(0xffffffffu, r);
      tc_fence_after_sync();
      return r;
    };
    auto issue_s = [&](int g) {
      const uint64_t db = dk0 + (((g & 1) * kTileKV) >> 4);
#pragma unroll
      for (int i = 0; i < kD / 16; ++i)
        if (i < ksteps_d) umma_ss_elected(tmem_base, dq + ((i * 32) >> 4), db + i * step_k, idesc_s, i > 0 ? 1u : 0u, issuer);
      umma_commit_elected(&bar->s_full, issuer);
    };
    if (issuer) {
      mbar_arrive_expect_tx(&bar->q_full, kTileQ);
      tma_load_3d(smem + kOffQ, &p.map_q, &bar->q_full, p.q_col0 + head_col, m0, seq);
    }
    __syncwarp();
    load_k(0);
    load_v(0);
    if (nkv > 1) {
      load_k(1);
      load_v(1);
    }
    bool ok = wait(&bar->q_full, 0, 0x100) && wait(&bar->k_full[0], 0, 0x110);
    if (ok) issue_s(0);
    for (int g = 0; g < nkv && ok; ++g) {
      const bool more = g + 1 < nkv;
      // S(g), and with it P*V(g - 1), complete: K's stage of block g and V's of block g - 1 may be refilled
      ok = wait(&bar->s_full, g & 1, 0x120);
      if (!ok) break;
      if (g + 2 < nkv) load_k(g + 2);
      if (g > 0 && more) load_v(g + 1);
      ok = wait(&bar->v_full[g & 1], (g >> 1) & 1, 0x130) && (!more || wait(&bar->k_full[(g + 1) & 1], ((g + 1) >> 1) & 1, 0x140)) &&
           wait(&bar->p_full, g & 1, 0x150);
      if (!ok) break;
      const uint64_t db = dv0 + (((g & 1) * kTileKV) >> 4);
#pragma unroll
      for (int i = 0; i < kBN / 16; ++i)
        umma_ts_elected(tmem_base + kColO, tmem_base + i * 8, db + i * step_v, idesc_o, (g > 0 || i > 0) ? 1u : 0u, issuer);
      // same thread, in-order pipe: S(g + 1) overwrites P(g) only after P*V(g) has read it
      if (more) issue_s(g + 1);
      else umma_commit_elected(&bar->o_done, issuer);
    }
  } else {
    // ------------------------------------------------------------ softmax and write-out
    const uint32_t s_col = tmem_base + (static_cast<uint32_t>(warp * 32) << 16), o_col = s_col + kColO;
    const float c = p.scale_log2;
    RowReference ref(c);
    float l = 0.f;
    bool ok = true;
    for (int g = 0; g < nkv; ++g) {
      ok = mbar_wait(&bar->s_full, g & 1, abort_word, 0x800);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after_sync();
      uint32_t sv[kBN];
      tmem_ld_x64_wait(s_col, sv);
      if constexpr (MODE == kModeSoftmax) {
        if (g == nkv - 1 && (p.L % kBN) != 0) {
          const int valid = p.L % kBN;             // partial last block: zero-filled K rows must not count
#pragma unroll
          for (int i = 0; i < kBN; ++i)
            if (i >= valid) sv[i] = __float_as_uint(-INFINITY);
        }
        float mx[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) mx[u] = __uint_as_float(sv[u]);
#pragma unroll
        for (int i = 8; i < kBN; i += 8) {
#pragma unroll
          for (int u = 0; u < 8; ++u) mx[u] = fmaxf(mx[u], __uint_as_float(sv[i + u]));
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) mx[u] = fmaxf(mx[u], mx[u + 4]);
        const float m_new = fmaxf(fmaxf(ref.m, mx[0]), fmaxf(fmaxf(mx[1], mx[2]), mx[3]));
        // lazy rescale, as in attention_sm100.cu; s_full(g) implies that P*V(g - 1) is done, so O is quiescent
        if (__any_sync(0xffffffffu, ref.asks(m_new, c, g == 1 ? kCloseSecondBlock : kCloseRescale))) {
          const float f = ref.move(m_new, c);
          if (g > 0) {
#pragma unroll 1
            for (int cc = 0; cc < kD; cc += 16) {
              uint32_t o[16];
              tmem_ld_x16_wait(o_col + cc, o);
#pragma unroll
              for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * f);
              tmem_st_x16(o_col + cc, o);
            }
            tmem_wait_st();
          }
          l *= f;
          ref.subtract(sv);
        }
      }
      const float mc = ref.offset(c);
      const uint64_t c2 = pack_f32x2(c, c), nmc2 = pack_f32x2(-mc, -mc);
      uint64_t sum[2] = {0, 0};
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t pk[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          float p0 = __uint_as_float(sv[32 * h + 2 * i]), p1 = __uint_as_float(sv[32 * h + 2 * i + 1]);
          if constexpr (MODE == kModeSoftmax) {
            const uint64_t w = softmax_weights(sv[32 * h + 2 * i], sv[32 * h + 2 * i + 1], c2, nmc2, weights_on_fma(16 * h + i));
            sum[i & 1] = add_f32x2(sum[i & 1], w);
            unpack_f32x2(w, p0, p1);
          } else if constexpr (MODE == kModeRelu) {
            p0 = p0 > 0.f ? p0 : 0.f;
            p1 = p1 > 0.f ? p1 : 0.f;
          }
          pk[i] = pack2<BF16>(p0, p1);
        }
        tmem_st_x16(s_col + 16 * h, pk);           // (every lane's scores are in registers: the load is warp-collective)
      }
      float sum0, sum1;
      unpack_f32x2(add_f32x2(sum[0], sum[1]), sum0, sum1);
      l += sum0 + sum1;
      tmem_wait_st();
      tc_fence_before_sync();
      mbar_arrive(&bar->p_full);
    }
    if (ok) {
      ok = mbar_wait(&bar->o_done, 0, abort_word, 0xA00);
      ok = __all_sync(0xffffffffu, ok);
    }
    if (ok) {
      tc_fence_after_sync();
      uint32_t o[kD];
      tmem_ld_x64_wait(o_col, o);
      const float inv = MODE == kModeSoftmax ? 1.0f / l : 1.0f;
      // The warp's 32 rows x 128 bytes turned around in its 4 KB of the Q buffer (every MMA has retired), 16-byte
      // pieces swizzled by row: a store instruction writes 4 rows x 128 contiguous bytes.
      uint8_t* stage = smem + kOffQ + warp * 4096;
#pragma unroll
      for (int i = 0; i < kD / 8; ++i) {
        uint32_t w[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          w[u] = pack2<BF16>(__uint_as_float(o[8 * i + 2 * u]) * inv, __uint_as_float(o[8 * i + 2 * u + 1]) * inv);
        *reinterpret_cast<uint4*>(stage + lane * 128 + ((i ^ (lane & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
      }
      __syncwarp();
      const size_t out_row0 = static_cast<size_t>(seq) * p.M + m0 + warp * 32;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int rr = 4 * i + (lane >> 3), piece = lane & 7;
        const uint4 v = *reinterpret_cast<const uint4*>(stage + rr * 128 + ((piece ^ (rr & 7)) << 4));
        if (m0 + warp * 32 + rr < p.M && piece * 8 < p.dv)
          *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(p.out) + ((out_row0 + rr) * p.out_ld + head_col + piece * 8) * 2) = v;
      }
    }
  }

  // After a wait has given up, TMA loads this CTA has armed may still be in flight; they complete within microseconds.
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

// ------------------------------------------------------------------ launcher
template <bool BF16, int MODE>
static cudaError_t launch_n(const AttnParams& p, long long items, cudaStream_t stream) {
  auto kern = attention_narrow_kernel<BF16, MODE>;
  static std::atomic<unsigned long long> configured{0};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  if (!((configured.load(std::memory_order_acquire) >> dev) & 1ull)) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytesThree);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    configured.fetch_or(1ull << dev, std::memory_order_release);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(items), 1, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  // Up to three items an SM: no place for a fourth.  The CTAs of a call go to the places that the call before it leaves free, while that one still runs (the
  // launch is programmatic): with four an SM they end up four on some SMs and two on others, and the call lasts as long as one of 592
  // items.  us, four places -> three, calls one after another: 300 items of 128 / 512 / 1024 keys 7.0 -> 6.3, 16.6 -> 14.3, 29.1 -> 25.1, 384 of 512 17.5 -> 14.4,
  // 444 of 512 17.0 -> 14.7; behind another kernel the placing is even and nothing changes (17.1 -> 17.0).  Items of one 64-key block are over so soon that the fourth place, where
  // the next call's CTAs are set up, is worth more once the three are nearly full (in a graph, both builds in turn, chains 365 0.87 to 0.95, 395 0.92 to 1.05, 444 4.16 -> 4.54; softmax
  // 425 0.90 to 0.95, 444 5.18 -> 5.34).
  const int three = p.L > 64 ? 444 : MODE == kModeSoftmax ? 425 : 370;
  cfg.dynamicSmemBytes = items > 296 && items <= three ? kSmemBytesThree : kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // see grid_dependency_wait in the kernel
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return launch_kernel(cfg, kern, p);
}

cudaError_t launch_attention_narrow(const AttnParams& p, int batch, bool bf16, int mode, cudaStream_t stream) {
  const long long items = static_cast<long long>((p.M + kBM - 1) / kBM) * batch;
  if (items > 0x7fffffffLL) return cudaErrorInvalidValue;
  if (mode == 0) return bf16 ? launch_n<true, 0>(p, items, stream) : launch_n<false, 0>(p, items, stream);
  if (mode == 1) return bf16 ? launch_n<true, 1>(p, items, stream) : launch_n<false, 1>(p, items, stream);
  return bf16 ? launch_n<true, 2>(p, items, stream) : launch_n<false, 2>(p, items, stream);
}

// Where the lines lie: calls of up to 296 items have other forms (attention_few: of up to four 128-key blocks, and of any number up to 148 items;
// those between are not long enough for this one, 200 x 5 blocks 13.8 -> 14.0, 200 x 8 18.6 -> 19.9).  With three items an SM and no place for a fourth this is the
// faster form for all numbers of blocks, with a softmax and without; us, others -> this kernel: softmax, 300 items of 5, 8, 16, 64 blocks 19.0 -> 17.2, 27.5 -> 25.5, 49.1 -> 46.7,
// 173.7 -> 171.1, 384 22.8 -> 17.6, 31.9 -> 26.3, 50.4 -> 46.9, 175.5 -> 170.8, 444 25.1 -> 18.8, 34.7 -> 26.2, 51.3 -> 46.8, 200 -> 194; chains, 300 items of 1, 4, 8, 32 blocks
// 6.4 -> 5.0, 12.2 -> 10.3, 20.1 -> 17.8, 62.0 -> 60.4, 444 7.5 -> 5.6, 14.0 -> 11.2, 23.5 -> 18.9, 71.1 -> 66.9.  (With a fourth place, 300 x 16 53.8 and 384 x 32 106.7 against
// 91.4 of the others.)  Above, it is ahead up to 24 blocks: 450 x 16 64.5 -> 59.4, 520 x 16 58.9 -> 56.0, 592 x 24 96.4 -> 92.2, 700 x 16 82.4 -> 80.2, 640 x 24
// 111.9 -> 112.1, 2048 x 4 83.8 -> 69.2, 1200 of 208 keys 30.6 -> 27.0, 640 of 64 13.0 -> 8.2; for longer items the other
// kernels' 128-key blocks cost less (1.6 us for two a SM against 2 x 1.0; 640 x 64 291 -> 301), and it pays again once a launch is three waves of those
// or more: 1024 x 64 398 -> 384.  A chain without a softmax has less between the hand-overs: there
// it gains with one or two blocks only (600 x 208 rows and keys 19.4 -> 18.0, 640 of 64 9.4 -> 7.4; 640 of 1024 would go 40 -> 43).
bool attention_narrow_pays(int batch, int M, int L, int mode) {
  const long long items = static_cast<long long>((M + kBM - 1) / kBM) * batch;
  const int blocks = (L + 127) / 128;
  if (items <= 444) return items > 296;
  return mode != kModeSoftmax ? blocks <= 2 : blocks <= 24 || items > 887;
}

}  // namespace ditto_b200
