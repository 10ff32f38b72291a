// Fused bmm -> softmax -> bmm for calls of few items: one 128-row tile per CTA, or per cluster of CTAs that divide its keys
// between them, and two softmax warps on every quarter of the rows.
//
// Such a call lasts as long as one CTA: set-up, first loads, its blocks of 128 keys one after another, write-out.  Little else
// runs on the SM meanwhile, so a block should take as little time as the chain
//   scores in tensor memory -> registers -> row maximum -> exponentials -> P in tensor memory -> P*V
// allows.  With one thread a row (the other kernels) each of the four warps has its sub-partition's units to itself and
// leaves them idle whenever it waits; here two warps share a row's 128 scores -- 32-key groups 0 and 2, and 1 and 3 -- and
// tell each other their maxima through shared memory.  S, O and P have tensor-memory columns of their own, so the next
// block's scores are ready by then, and a last block ends with its keys.
//
// Roles: warps 0-7 softmax and write-out (warps w and w + 4: rows 32 w .. 32 w + 31, TMEM lanes alike), 8 loads, 9 MMAs.
// With `parts` CTAs in the cluster each takes a contiguous part of the tile's blocks; they combine (max, sum, O) through
// distributed shared memory at the end.
//
// Two CTAs fit an SM at head dimension 64 (84 KB, 112 with four parts; 256 tensor-memory columns, 94 registers): the next call's are set up under this
// one's.  At head dimension 128 (TWO) they do with one stage of K and of V and with P in the place of S (100 KB, 256 columns): a CTA by itself
// is a chain then -- scores, softmax, P*V, next scores -- and two of them fill each other's gaps; for more items than SMs.  What it measured
// stands at attention_few.
#define DITTO_WAIT_OUT_OF_LINE   // see mbar_wait
#include "attention_sm100.cuh"

#include <algorithm>
#include <atomic>

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "host_util.cuh"
#include "mlp_common.cuh"
#include "sm100_ptx.cuh"
#include "softmax_step.cuh"

namespace ditto_b200 {

namespace {

constexpr int kBM = 128, kBN = 128;
constexpr int kSoftmaxWarps = 8, kWarpLoad = 8, kWarpMma = 9;
constexpr int kThreads = 10 * 32;
constexpr int kFirstKeys = 64;            // of a block, in the first part of P (groups 0 and 1); the rest follows by itself
constexpr int kModeSoftmax = 0, kModeRelu = 1;

// TWO: the form of which two CTAs fit an SM at head dimension 128
template <int D, bool TWO>
struct Layout {
  static constexpr int kStages = TWO ? 1 : 2;
  static constexpr int kTileQ = kBM * D * 2;
  static constexpr int kTileKV = kBN * D * 2;
  static constexpr int kOffQ = 0;
  static constexpr int kOffK = kOffQ + kTileQ;
  static constexpr int kOffV = kOffK + kStages * kTileKV;
  static constexpr int kOffPair = kOffV + kStages * kTileKV;      // float [2][2][128]: maxima, by parity of the block and half
  static constexpr int kOffRows = kOffPair + 2 * 2 * kBM * 4;     // float2 [128]: (max, sum) for the cluster, eight parts
  static constexpr int kOffBar = kOffRows + kBM * 8;
  // the other parts' (max, sum), float2 [parts - 1][128], and columns, float4 [parts - 1][D / parts / 4][128]
  static constexpr int kOffMl = kOffBar + 256;
  static __host__ __device__ constexpr bool own_memory(int parts) { return parts == 2 || parts == 4; }
  static __host__ __device__ constexpr int off_in(int parts) { return kOffMl + (parts - 1) * kBM * 8; }
  static __host__ __device__ constexpr int bytes(int parts) {
    return (own_memory(parts) ? off_in(parts) + (parts - 1) * (D / parts) * kBM * 4 : kOffMl) + 1024;
  }
  static constexpr uint32_t kColS = 0, kColO = 128, kColP = TWO ? 0 : 128 + D;
  static constexpr uint32_t kTmemCols = D == 64 || TWO ? 256 : 512;
};

struct SBars {
  uint64_t q_full, k_full[2], k_empty[2], v_full[2], v_empty[2];
  uint64_t s_full, s_taken, p_part[2], o_done;
  uint64_t pair[4];                       // the two warps of a quarter have written what the other one reads
  uint32_t tmem_base;
  uint32_t abort_word;
};
static_assert(sizeof(SBars) <= 256, "barrier block too large");
static_assert(2 * (Layout<64, false>::bytes(4) + 1024) <= 228 * 1024 && Layout<128, false>::bytes(4) <= 227 * 1024, "shared memory budget");

// The largest of 32 scores and m.
__device__ __forceinline__ float max_with(float m, const uint32_t* s) {
  auto v = [&](int i) { return __uint_as_float(s[i]); };
  float a[4] = {m, v(0), v(1), v(2)};
  // 29 scores left, two at a time on four chains
#pragma unroll
  for (int i = 3; i < 27; i += 8) {
#pragma unroll
    for (int u = 0; u < 4; ++u) a[u] = max3(a[u], v(i + 2 * u), v(i + 2 * u + 1));
  }
  a[0] = max3(a[0], v(27), v(28));
  a[1] = max3(a[1], v(29), v(30));
  a[2] = max3(a[2], a[3], v(31));
  return max3(a[0], a[1], a[2]);
}

// The 32 scores of a row's group g -> their weights 2^(s c - mc), rounded to the operand type and packed; the sums take them before rounding.
// A block is a chain of one warp's steps here, and the exponentials its longest: some are computed on the multiply-add pipe
// (weights_on_fma).  Scalar arithmetic / packed with 2 / 3 / 4 of 32 pairs there, us: head dimension 64, 12 slices of 512 rows and keys 7.66 /
// 7.58 / 7.58 / 7.62, 40 of them 11.67 / 11.67 / 11.55 / 11.47, 16 of 1024 14.50 / 14.30 / 14.21 / 14.42; 128, 140 tiles of 1024 keys 16.71 / 16.34 /
// 16.34 / 16.30, 4 slices of 1024 x 4096 18.96 / 18.39 / 18.47 / 18.60.
template <bool BF16>
__device__ __forceinline__ void row_weights(int g, const uint32_t* s, float c, float mc, uint64_t& sum, uint32_t (&w)[16]) {
  const uint64_t c2 = pack_f32x2(c, c), nmc2 = pack_f32x2(-mc, -mc);
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const uint64_t p = softmax_weights(s[2 * i], s[2 * i + 1], c2, nmc2, weights_on_fma(16 * g + i));
    sum = add_f32x2(sum, p);
    float a, b;
    unpack_f32x2(p, a, b);
    w[i] = pack2<BF16>(a, b);
  }
}

// The same place of the chains without a softmax.
template <bool BF16, bool RELU>
__device__ __forceinline__ void pass_on(const uint32_t* s, uint32_t (&w)[16]) {
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    float a = __uint_as_float(s[2 * i]), b = __uint_as_float(s[2 * i + 1]);
    if constexpr (RELU) {                              // if_then_else(D > 0, D, 0) as in the reference
      a = a > 0.f ? a : 0.f;
      b = b > 0.f ? b : 0.f;
    }
    w[i] = pack2<BF16>(a, b);
  }
}

}  // namespace

// PARTS: CTAs that share an item's keys
template <bool BF16, int D, int MODE, int PARTS, bool TWO>
__global__ void __launch_bounds__(kThreads, 2) attention_short_kernel(const __grid_constant__ AttnParams p) {
  using SM = Layout<D, TWO>;
  constexpr int kAtoms = D / 64, kStages = SM::kStages;
  extern __shared__ uint8_t smem_raw[];
  // the CTAs of a cluster round up by the same amount: offsets match across the cluster
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  SBars* bar = reinterpret_cast<SBars*>(smem + SM::kOffBar);
  volatile uint32_t* abort_word = &bar->abort_word;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int tiles = (p.M + kBM - 1) / kBM;
  // the CTAs of a cluster are consecutive: rank r of `parts` takes K/V blocks [r * n / parts, (r + 1) * n / parts)
  constexpr int parts = PARTS;
  const int part = PARTS == 1 ? 0 : static_cast<int>(cluster_ctarank());
  const int id = static_cast<int>(blockIdx.x) / parts;
  const int slice = id / tiles, seq = slice / p.heads;
  const int head_col = (slice - seq * p.heads) * p.d;
  const int m0 = (id - slice * tiles) * kBM;
  const int blocks = (p.L + kBN - 1) / kBN;
  const int j0 = part * blocks / parts, nkv = (part + 1) * blocks / parts - j0;
  // keys of this CTA's last block, a multiple of 16
  const int last_keys = part == parts - 1 ? p.L - (blocks - 1) * kBN : kBN;

  if (threadIdx.x == 0) {
    mbar_init(&bar->q_full, 1);
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&bar->k_full[s], 1);
      mbar_init(&bar->k_empty[s], 1);
      mbar_init(&bar->v_full[s], 1);
      mbar_init(&bar->v_empty[s], 1);
    }
    mbar_init(&bar->s_full, 1);
    mbar_init(&bar->s_taken, kSoftmaxWarps);
    mbar_init(&bar->p_part[0], kSoftmaxWarps);
    mbar_init(&bar->p_part[1], kSoftmaxWarps);
    mbar_init(&bar->o_done, 1);
    for (int q = 0; q < 4; ++q) mbar_init(&bar->pair[q], 2);
    bar->abort_word = 0;
    fence_mbar_init();
  }
  if (warp == 0) {
    tmem_alloc(&bar->tmem_base, SM::kTmemCols);
    tmem_relinquish();
  }
  if (warp == kWarpLoad && lane == 0) {
    tma_prefetch_desc(&p.map_q);
    tma_prefetch_desc(&p.map_k);
    tma_prefetch_desc(&p.map_v);
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  // (a peer's shared memory may be written once the peer has started)
  if (SM::own_memory(PARTS)) cluster_arrive();
  const uint32_t tmem_base = bar->tmem_base;
  // Programmatic dependent launch: nothing above touches global memory.
  grid_dependency_wait();
  grid_launch_dependents();

  bool ok = true;
  float row_m = 0.f, row_l = 0.f;          // this CTA's maximum and sum of the thread's row
  const int quarter = warp & 3, half = (warp >> 2) & 1;
  const int row = quarter * 32 + lane;
  const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);

  if (warp == kWarpLoad) {
    // ------------------------------------------------------------ TMA producer (one thread)
    if (lane == 0) {
      mbar_arrive_expect_tx(&bar->q_full, SM::kTileQ);
      for (int a = 0; a < kAtoms; ++a)
        tma_load_3d(smem + SM::kOffQ + a * (kBM * 128), &p.map_q, &bar->q_full, p.q_col0 + head_col + a * 64, m0, seq);
      for (int j = 0; j < nkv; ++j) {
        const int s = j % kStages;
        const uint32_t ph = (j / kStages) & 1;
        ok = mbar_wait(&bar->k_empty[s], ph ^ 1, abort_word, 0x100 + j);
        if (!ok) break;
        uint8_t* k = smem + SM::kOffK + s * SM::kTileKV;
        mbar_arrive_expect_tx(&bar->k_full[s], SM::kTileKV);
        if (p.k_transposed) {
          for (int a = 0; a < kBN / 64; ++a)
            tma_load_3d(k + a * (D * 128), &p.map_k, &bar->k_full[s], (j0 + j) * kBN + a * 64, 0, slice);
        } else {
          for (int a = 0; a < kAtoms; ++a)
            tma_load_3d(k + a * (kBN * 128), &p.map_k, &bar->k_full[s], p.k_col0 + head_col + a * 64, (j0 + j) * kBN, seq);
        }
        ok = mbar_wait(&bar->v_empty[s], ph ^ 1, abort_word, 0x200 + j);
        if (!ok) break;
        uint8_t* v = smem + SM::kOffV + s * SM::kTileKV;
        mbar_arrive_expect_tx(&bar->v_full[s], SM::kTileKV);
        if (p.v_transposed) {
          for (int a = 0; a < kBN / 64; ++a)
            tma_load_3d(v + a * (D * 128), &p.map_v, &bar->v_full[s], (j0 + j) * kBN + a * 64, 0, slice);
        } else {
          for (int a = 0; a < kAtoms; ++a)
            tma_load_3d(v + a * (kBN * 128), &p.map_v, &bar->v_full[s], p.v_col0 + head_col + a * 64, (j0 + j) * kBN, seq);
        }
      }
    }
    __syncwarp();
  } else if (warp == kWarpMma) {
    // ------------------------------------------------------------ MMA issuer (converged warp, elected lane issues)
    const uint32_t issuer = elect_one();
    const bool kt = p.k_transposed != 0, vt = p.v_transposed != 0;
    const int ksteps_d = p.d / 16;
    const uint32_t idesc_s = umma_idesc_f16(BF16, kBM, kBN, false, kt);
    const uint32_t idesc_o = umma_idesc_f16(BF16, kBM, p.dv, false, !vt);   // (columns past dv are not stored)
    const uint64_t dq = umma_desc_sw128(smem_u32(smem + SM::kOffQ), 16, 1024);
    const uint64_t dk0 = kt ? umma_desc_sw128(smem_u32(smem + SM::kOffK), D * 128, 1024) : umma_desc_sw128(smem_u32(smem + SM::kOffK), 16, 1024);
    const uint64_t dv0 = vt ? umma_desc_sw128(smem_u32(smem + SM::kOffV), 16, 1024) : umma_desc_sw128(smem_u32(smem + SM::kOffV), kBN * 128, 1024);
    auto wait = [&](uint64_t* b, uint32_t parity, uint32_t code) {
      bool r = mbar_wait(b, parity, abort_word, code);
      r = __all_sync(0xffffffffu, r);
      tc_fence_after_sync();
      return r;
    };
    auto issue_s = [&](int stage) {
      const uint64_t db = dk0 + ((stage * SM::kTileKV) >> 4);
#pragma unroll
      for (int i = 0; i < D / 16; ++i) {
        const uint32_t off = ((i / 4) * (kBM * 128) + (i % 4) * 32) >> 4;
        if (i < ksteps_d)
          umma_ss_elected(tmem_base + SM::kColS, dq + off, db + (kt ? static_cast<uint32_t>((i * 2048) >> 4) : off), idesc_s,
                          i > 0 ? 1u : 0u, issuer);
      }
      umma_commit_elected(&bar->s_full, issuer);
      umma_commit_elected(&bar->k_empty[stage], issuer);
    };
    auto issue_pv = [&](int stage, int from, int to, bool first) {
      const uint64_t db = dv0 + ((stage * SM::kTileKV) >> 4);
#pragma unroll
      for (int i = 0; i < kFirstKeys / 16; ++i) {
        const int step = from / 16 + i;
        if (step * 16 < to) {
          const uint32_t off = vt ? static_cast<uint32_t>(((step / 4) * (D * 128) + (step % 4) * 32) >> 4) : static_cast<uint32_t>((step * 2048) >> 4);
          umma_ts_elected(tmem_base + SM::kColO, tmem_base + SM::kColP + step * 8, db + off, idesc_o, first && i == 0 ? 0u : 1u, issuer);
        }
      }
    };
    ok = wait(&bar->k_full[0], 0, 0x300) && wait(&bar->q_full, 0, 0x301);
    if (ok) issue_s(0);
    for (int j = 0; j < nkv && ok; ++j) {
      const int st = j % kStages, sn = (j + 1) % kStages;
      const bool more = j + 1 < nkv;
      const int keys = more ? kBN : last_keys;
      if (!TWO && more) {
        // the softmax warps must have taken S(j) out of tensor memory before S(j + 1) lands there
        ok = wait(&bar->k_full[sn], ((j + 1) / kStages) & 1, 0x310) && wait(&bar->s_taken, j & 1, 0x320);
        if (!ok) break;
        issue_s(sn);
      }
      ok = wait(&bar->v_full[st], (j / kStages) & 1, 0x330) && wait(&bar->p_part[0], j & 1, 0x340);
      if (!ok) break;
      issue_pv(st, 0, min(keys, kFirstKeys), j == 0);
      ok = wait(&bar->p_part[1], j & 1, 0x350);
      if (!ok) break;
      issue_pv(st, kFirstKeys, keys, false);
      umma_commit_elected(&bar->v_empty[st], issuer);     // also tells the softmax warps that P*V(j) is done
      if (!more) umma_commit_elected(&bar->o_done, issuer);
      if (TWO && more) {
        // P lies where S was: the next scores follow its last use in the order of issue
        ok = wait(&bar->k_full[0], (j + 1) & 1, 0x310);
        if (ok) issue_s(0);
      }
    }
  } else {
    // ------------------------------------------------------------ softmax (warps 0-7)
    const uint32_t s_col = lane_base + SM::kColS, o_col = lane_base + SM::kColO + half * (D / 2), p_col = lane_base + SM::kColP;
    const float c = p.scale_log2;
    float* told = reinterpret_cast<float*>(smem + SM::kOffPair) + row;     // [parity][half][row]
    RowReference ref(c);
    float l = 0.f;
    for (int j = 0; j < nkv; ++j) {
      const uint32_t par = j & 1;
      ok = mbar_wait(&bar->s_full, par, abort_word, 0x800);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after_sync();
      uint32_t sv[64];                                     // groups `half` and 2 + `half` of 32 keys
      tmem_ld_2x32_wait(s_col + 32 * half, s_col + 64 + 32 * half, sv);
      tc_fence_before_sync();
      if (!TWO) mbar_arrive_warp(&bar->s_taken, lane);
      const int keys = j == nkv - 1 ? last_keys : kBN;
      if constexpr (MODE == kModeSoftmax) {
        if (keys != kBN) {
          // a partial last block brings zero-filled rows, whose scores must not count
#pragma unroll
          for (int i = 0; i < 64; ++i)
            if (64 * (i / 32) + 32 * half + i % 32 >= keys) sv[i] = __float_as_uint(-INFINITY);
        }
        float m_new = max_with(max_with(ref.m, sv), sv + 32);
        told[(par * 2 + half) * kBM] = m_new;
        mbar_arrive_warp(&bar->pair[quarter], lane);
        ok = mbar_wait(&bar->pair[quarter], par, abort_word, 0x880);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        m_new = fmaxf(m_new, told[(par * 2 + (half ^ 1)) * kBM]);
        if (TWO) tc_fence_after_sync();                    // (the other warp has its scores too: P may take their place)
        if (!TWO && j > 0) {
          // P*V(j-1) must have finished before P is overwritten or O is rescaled (S(j) was issued ahead of it)
          ok = mbar_wait(&bar->v_empty[(j - 1) % kStages], ((j - 1) / kStages) & 1, abort_word, 0x900);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tc_fence_after_sync();
        }
        // lazy rescale, as in attention_sm100.cu; both warps of a quarter see the same maxima and decide alike
        if (__any_sync(0xffffffffu, ref.asks(m_new, c, j == 1 ? kCloseSecondBlock : kCloseRescale))) {
          const float f = ref.move(m_new, c);
          if (j > 0) {
#pragma unroll 1
            for (int h = 0; h < D / 2; h += 16) {
              uint32_t o[16];
              tmem_ld_x16_wait(o_col + h, o);
#pragma unroll
              for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * f);
              tmem_st_x16(o_col + h, o);
            }
            tmem_wait_st();
          }
          l *= f;
          ref.subtract(sv);
        }
      } else if (TWO) {
        // P takes the place of the scores once both warps of the quarter have theirs
        mbar_arrive_warp(&bar->pair[quarter], lane);
        ok = mbar_wait(&bar->pair[quarter], par, abort_word, 0x880);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after_sync();
      } else if (j > 0) {
        ok = mbar_wait(&bar->v_empty[(j - 1) % kStages], ((j - 1) / kStages) & 1, abort_word, 0x900);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after_sync();
      }
      const float mc = ref.offset(c);
      uint64_t sum = 0;
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        if (64 * g + 32 * half < keys) {                   // (P*V reads no others)
          uint32_t w[16];
          if constexpr (MODE == kModeSoftmax) row_weights<BF16>(g, sv + 32 * g, c, mc, sum, w);
          else pass_on<BF16, MODE == kModeRelu>(sv + 32 * g, w);
          tmem_st_x16(p_col + 32 * g + 16 * half, w);
        }
        tmem_wait_st();
        tc_fence_before_sync();
        mbar_arrive_warp(&bar->p_part[g], lane);
      }
      float sum0, sum1;
      unpack_f32x2(sum, sum0, sum1);
      l += sum0 + sum1;
    }
    if (ok && MODE == kModeSoftmax) {
      // the row's sum, in the same order in both warps
      told[((nkv & 1) * 2 + half) * kBM] = l;
      mbar_arrive_warp(&bar->pair[quarter], lane);
      ok = mbar_wait(&bar->pair[quarter], nkv & 1, abort_word, 0x890);
      ok = __all_sync(0xffffffffu, ok);
      if (ok) l = told[(nkv & 1) * 2 * kBM] + told[((nkv & 1) * 2 + 1) * kBM];
    }
    if (ok) {
      ok = mbar_wait(&bar->o_done, 0, abort_word, 0xA00);
      ok = __all_sync(0xffffffffu, ok);
      tc_fence_after_sync();
    }
    row_m = ref.m;
    row_l = l;
    if (ok && PARTS == 1) {
      const float inv = MODE == kModeSoftmax ? 1.0f / l : 1.0f;
      // Turned around in 2 or 4 KB of the K ring per warp (every MMA has retired), 16-byte pieces swizzled by row, so that a
      // store instruction writes rows of 64 or 128 contiguous bytes.
      constexpr int kPieces = D / 16;                      // 16-byte pieces of a row's half
      uint8_t* stage = smem + SM::kOffK + warp * (kPieces * 512);
      uint32_t o[D / 2];
      if constexpr (D == 128) tmem_ld_x64_wait(o_col, o); else tmem_ld_x32_wait(o_col, o);
#pragma unroll
      for (int i = 0; i < kPieces; ++i) {
        uint32_t w[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          w[u] = pack2<BF16>(__uint_as_float(o[8 * i + 2 * u]) * inv, __uint_as_float(o[8 * i + 2 * u + 1]) * inv);
        const int at = D == 128 ? i ^ (lane & 7) : i ^ ((lane >> 1) & 3);
        *reinterpret_cast<uint4*>(stage + lane * (kPieces * 16) + at * 16) = make_uint4(w[0], w[1], w[2], w[3]);
      }
      __syncwarp();
      const size_t out_row0 = static_cast<size_t>(seq) * p.M + m0 + quarter * 32;
      constexpr int kRowsAtOnce = 32 / kPieces;
#pragma unroll
      for (int i = 0; i < kPieces; ++i) {
        const int rr = kRowsAtOnce * i + lane / kPieces, piece = lane % kPieces;
        const int at = D == 128 ? piece ^ (rr & 7) : piece ^ ((rr >> 1) & 3);
        const uint4 v = *reinterpret_cast<const uint4*>(stage + rr * (kPieces * 16) + at * 16);
        const int col = half * (D / 2) + piece * 8;        // widths are multiples of 16: whole 16-byte pieces
        if (m0 + quarter * 32 + rr < p.M && col < p.dv)
          *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(p.out) + ((out_row0 + rr) * p.out_ld + head_col + col) * 2) = v;
      }
    }
  }

  if constexpr (SM::own_memory(PARTS)) {
    // Combine the parts.  Every CTA hands each of the others D / PARTS columns of its O and its rows' (max, sum), into memory of their own; once it has
    // theirs it scales what it was given and its own columns, which are still in tensor memory, by 2^(max - overall max) / overall sum, adds them in
    // rank order and writes those columns of the result: a reduce-scatter, so the exchange and the write-out are spread over the cluster.
    // Laid out [source][16-byte piece][row], a warp's store or load covers 512 contiguous bytes.  Both barriers are reached by every thread
    // whether its waits expired or not.
    // One barrier between the last P*V and the result (the first one has long been passed: it says that the peers have started), the number of parts
    // known at compile time.  Against (max, sum) read from the peers behind a barrier, columns through the K ring and a number of parts known at
    // run time: 0.88 to 0.92 of the time of a call in two parts (one ViT-Base image 5.9 -> 5.3 us), and unsplit calls, which bring none of this code, 0.98 to 0.99.
    __syncwarp();
    cluster_wait();
    constexpr int kCols = D / PARTS, kPiece = kCols >= 32 ? 16 : kCols / 2;
    const uint32_t o_base = lane_base + SM::kColO;
    float2* ml = reinterpret_cast<float2*>(smem + SM::kOffMl) + row;       // [PARTS - 1][row]
    float4* in = reinterpret_cast<float4*>(smem + SM::off_in(PARTS)) + row;  // [PARTS - 1][kCols / 4][row]
    if (warp < kSoftmaxWarps) {
      if (MODE == kModeSoftmax && half == 0) {
#pragma unroll
        for (int i = 0; i < PARTS - 1; ++i) {
          const int to = i + (i >= part);
          st_cluster_v2(map_to_cta(smem_u32(ml + (part - (part > to)) * kBM), to), row_m, row_l);
        }
      }
#pragma unroll 1
      for (int c = half; c < (PARTS - 1) * kCols / 16; c += 2) {
        const int i = c / (kCols / 16), sub = c - i * (kCols / 16), to = i + (i >= part);
        uint32_t o[16];
        tmem_ld_x16_wait(o_base + to * kCols + sub * 16, o);
        const uint32_t at = map_to_cta(smem_u32(in + ((part - (part > to)) * (kCols / 4) + sub * 4) * kBM), to);
#pragma unroll
        for (int q = 0; q < 4; ++q)
          st_cluster_v4(at + q * (kBM * 16), __uint_as_float(o[4 * q]), __uint_as_float(o[4 * q + 1]), __uint_as_float(o[4 * q + 2]), __uint_as_float(o[4 * q + 3]));
      }
    }
    __syncwarp();
    cluster_sync_all();
    if (warp < kSoftmaxWarps) {
      float f[PARTS];                                    // factors of the parts
      if constexpr (MODE == kModeSoftmax) {
        float2 t[PARTS];
        float top = -INFINITY, total = 0.f;
#pragma unroll
        for (int r = 0; r < PARTS; ++r) {
          t[r] = r == part ? make_float2(row_m, row_l) : ml[(r - (r > part)) * kBM];
          top = fmaxf(top, t[r].x);
        }
#pragma unroll
        for (int r = 0; r < PARTS; ++r) {
          f[r] = ex2_approx((t[r].x - top) * p.scale_log2);
          total = fmaf(t[r].y, f[r], total);
        }
#pragma unroll
        for (int r = 0; r < PARTS; ++r) f[r] = f[r] / total;
      }
      uint8_t* dst = reinterpret_cast<uint8_t*>(p.out) + ((static_cast<size_t>(seq) * p.M + m0 + row) * p.out_ld + head_col) * 2;
#pragma unroll 1
      for (int c = half * kPiece; c < kCols; c += 2 * kPiece) {
        const int col = part * kCols + c;                // widths are multiples of 16
        if (col >= p.dv) break;
        uint32_t own[kPiece];
        if constexpr (kPiece == 16) tmem_ld_x16_wait(o_base + col, own); else tmem_ld_x8_wait(o_base + col, own);
        float sum[kPiece];
        if constexpr (PARTS == 2 && MODE == kModeSoftmax) {          // (two terms: either order is the same sum)
          const float mine = part == 0 ? f[0] : f[1], theirs = part == 0 ? f[1] : f[0];
#pragma unroll
          for (int q = 0; q < kPiece / 4; ++q) {
            const float4 g = in[(c / 4 + q) * kBM];
            sum[4 * q] = __fadd_rn(__fmul_rn(__uint_as_float(own[4 * q]), mine), __fmul_rn(g.x, theirs));
            sum[4 * q + 1] = __fadd_rn(__fmul_rn(__uint_as_float(own[4 * q + 1]), mine), __fmul_rn(g.y, theirs));
            sum[4 * q + 2] = __fadd_rn(__fmul_rn(__uint_as_float(own[4 * q + 2]), mine), __fmul_rn(g.z, theirs));
            sum[4 * q + 3] = __fadd_rn(__fmul_rn(__uint_as_float(own[4 * q + 3]), mine), __fmul_rn(g.w, theirs));
          }
        } else {
#pragma unroll
          for (int r = 0; r < PARTS; ++r) {
            const float4* from = in + ((r - (r > part)) * (kCols / 4) + c / 4) * kBM;
#pragma unroll
            for (int q = 0; q < kPiece / 4; ++q) {
              float4 g = make_float4(__uint_as_float(own[4 * q]), __uint_as_float(own[4 * q + 1]), __uint_as_float(own[4 * q + 2]), __uint_as_float(own[4 * q + 3]));
              if (r != part) g = from[q * kBM];
              if constexpr (MODE == kModeSoftmax) g = make_float4(__fmul_rn(g.x, f[r]), __fmul_rn(g.y, f[r]), __fmul_rn(g.z, f[r]), __fmul_rn(g.w, f[r]));
              sum[4 * q] = r == 0 ? g.x : sum[4 * q] + g.x;
              sum[4 * q + 1] = r == 0 ? g.y : sum[4 * q + 1] + g.y;
              sum[4 * q + 2] = r == 0 ? g.z : sum[4 * q + 2] + g.z;
              sum[4 * q + 3] = r == 0 ? g.w : sum[4 * q + 3] + g.w;
            }
          }
        }
        if (m0 + row < p.M) {
#pragma unroll
          for (int q = 0; q < kPiece / 8; ++q)
            *reinterpret_cast<uint4*>(dst + col * 2 + 16 * q) = make_uint4(pack2<BF16>(sum[8 * q], sum[8 * q + 1]), pack2<BF16>(sum[8 * q + 2], sum[8 * q + 3]),
                                                                           pack2<BF16>(sum[8 * q + 4], sum[8 * q + 5]), pack2<BF16>(sum[8 * q + 6], sum[8 * q + 7]));
        }
      }
    }
  }

  if constexpr (PARTS > 1 && !SM::own_memory(PARTS)) {
    // (Eight parts: their columns in memory of their own leave room for one CTA an SM at head dimension 64, and take 0 to 4 % longer at 128.)
    // Combine the parts.  Every CTA publishes its rows' (max, sum), scales its O by
    // 2^(max - overall max) / overall sum and hands D / parts columns of it to each CTA of the cluster, which adds
    // what it was given and writes those columns of the result: a reduce-scatter, so the exchange (D * 512 bytes in
    // and out of every CTA) and the write-out are spread over the cluster.  Parts are added in rank order.
    // The incoming pieces go to the K ring, idle since the last P*V of this CTA (first cluster barrier); laid out
    // [source][16-byte piece][row], a warp's store or load covers 512 contiguous bytes.  Both barriers are reached
    // by every thread whether its waits expired or not.
    float2* ml = reinterpret_cast<float2*>(smem + SM::kOffRows) + row;
    if (warp < 4 && MODE == kModeSoftmax) *ml = make_float2(row_m, row_l);
    __syncwarp();
    cluster_sync_all();
    const int cols = D / parts;                        // columns of the result that one CTA adds up: 8 to 64
    const int cols_log2 = 31 - __clz(cols);
    if (warp < kSoftmaxWarps) {
      float f = 1.f;
      if constexpr (MODE == kModeSoftmax) {
        const uint32_t at = smem_u32(ml);
        float mv[8], lv[8], top = -INFINITY;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          if (r < parts) {
            ld_cluster_v2(map_to_cta(at, r), mv[r], lv[r]);
            top = fmaxf(top, mv[r]);
          }
        }
        float total = 0.f;
#pragma unroll
        for (int r = 0; r < 8; ++r)
          if (r < parts) total = fmaf(lv[r], ex2_approx((mv[r] - top) * p.scale_log2), total);
        f = ex2_approx((row_m - top) * p.scale_log2) / total;
      }
      const uint32_t in0 = smem_u32(smem + SM::kOffK) + (part * (cols / 4) * kBM + row) * 16;
#pragma unroll 1
      for (int h = half * 32; h < D; h += 64) {
        uint32_t o[32];
        tmem_ld_x32_wait(lane_base + SM::kColO + h, o);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const int col = h + 4 * q;
          st_cluster_v4(map_to_cta(in0 + (col & (cols - 1)) * (kBM * 4), col >> cols_log2), __uint_as_float(o[4 * q]) * f,
                        __uint_as_float(o[4 * q + 1]) * f, __uint_as_float(o[4 * q + 2]) * f,
                        __uint_as_float(o[4 * q + 3]) * f);
        }
      }
    }
    __syncwarp();
    cluster_sync_all();
    if (warp < kSoftmaxWarps && m0 + row < p.M) {
      const float4* in = reinterpret_cast<const float4*>(smem + SM::kOffK) + row;
      uint8_t* dst = reinterpret_cast<uint8_t*>(p.out) + ((static_cast<size_t>(seq) * p.M + m0 + row) * p.out_ld + head_col) * 2;
#pragma unroll 1
      for (int c8 = half; c8 < cols / 8; c8 += 2) {
        const int col = part * cols + 8 * c8;        // widths are multiples of 16: whole 16-byte pieces
        if (col >= p.dv) break;
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
#pragma unroll 2
        for (int r = 0; r < parts; ++r) {
          const float4 u = in[(r * (cols / 4) + 2 * c8) * kBM], v = in[(r * (cols / 4) + 2 * c8 + 1) * kBM];
          a.x += u.x; a.y += u.y; a.z += u.z; a.w += u.w;
          b.x += v.x; b.y += v.y; b.z += v.z; b.w += v.w;
        }
        *reinterpret_cast<uint4*>(dst + col * 2) =
            make_uint4(pack2<BF16>(a.x, a.y), pack2<BF16>(a.z, a.w), pack2<BF16>(b.x, b.y), pack2<BF16>(b.z, b.w));
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
    tmem_dealloc(tmem_base, SM::kTmemCols);
    if (lane == 0 && bar->abort_word != 0 && p.status != nullptr) atomicCAS(p.status, 0, static_cast<int>(bar->abort_word));
  }
}

// ------------------------------------------------------------------ launcher
template <bool BF16, int D, int MODE, int PARTS, bool TWO>
static cudaError_t launch_s(const AttnParams& p, int ctas, cudaStream_t stream) {
  using SM = Layout<D, TWO>;
  auto kern = attention_short_kernel<BF16, D, MODE, PARTS, TWO>;
  static std::atomic<unsigned long long> configured{0};
  int dev = 0;
  cudaError_t e = current_device_checked(&dev);
  if (e != cudaSuccess) return e;
  if (!device_configured(configured, dev)) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SM::bytes(PARTS));
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    mark_device_configured(configured, dev);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(ctas), 1, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = SM::bytes(PARTS);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // see grid_dependency_wait in the kernel
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = static_cast<unsigned>(p.parts);
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = p.parts > 1 ? 2 : 1;
  return launch_kernel(cfg, kern, p);
}

cudaError_t launch_attention_short(const AttnParams& params, int batch, int d, bool bf16, int mode, int parts, bool two, cudaStream_t stream) {
  const int blocks = (params.L + kBN - 1) / kBN;
  const long long ctas = static_cast<long long>((params.M + kBM - 1) / kBM) * batch * parts;
  if ((parts != 1 && parts != 2 && parts != 4 && parts != 8) || parts > blocks || ctas > 0x7fffffffLL || (two && (d != 128 || parts > 1))) return cudaErrorInvalidValue;
  AttnParams p = params;
  p.parts = parts;
  const int n = static_cast<int>(ctas);
#define DITTO_DISPATCH(BF, DD, PA, TW) \
  if (bf16 == BF && d == DD && parts == PA && two == TW) \
    return mode == 0 ? launch_s<BF, DD, 0, PA, TW>(p, n, stream) : mode == 1 ? launch_s<BF, DD, 1, PA, TW>(p, n, stream) : launch_s<BF, DD, 2, PA, TW>(p, n, stream);
#define DITTO_DISPATCH_PARTS(BF, DD) \
  DITTO_DISPATCH(BF, DD, 1, false) DITTO_DISPATCH(BF, DD, 2, false) DITTO_DISPATCH(BF, DD, 4, false) DITTO_DISPATCH(BF, DD, 8, false)
  DITTO_DISPATCH_PARTS(false, 64)
  DITTO_DISPATCH_PARTS(false, 128)
  DITTO_DISPATCH_PARTS(true, 64)
  DITTO_DISPATCH_PARTS(true, 128)
  DITTO_DISPATCH(false, 128, 1, true)
  DITTO_DISPATCH(true, 128, 1, true)
#undef DITTO_DISPATCH_PARTS
#undef DITTO_DISPATCH
  return cudaErrorInvalidValue;
}

// Clusters of 1 << lg CTAs the device holds at once with a CTA an SM, asked for an instance at head dimension 128, whose shared memory
// allows no second one.  Instances at 64 and the kernel with a thread a row run two an SM.  The query does not see that: it rounds
// their ten or six warps up to a multiple of four and finds registers for one CTA, but 148 items of 64 blocks in two parts take
// 68 to 76 us (59 to 66 with a thread a row) where two waves of those parts would take 90.
static int cluster_places(int lg) {
  static std::atomic<int> places[kMaxDevices][4];       // 0: not looked up yet; else clusters + 1
  int dev = 0;
  if (current_device_checked(&dev) != cudaSuccess) return 0;
  int n = places[dev][lg].load(std::memory_order_relaxed);
  if (n == 0) {
    using SM = Layout<128, false>;
    auto kern = attention_short_kernel<false, 128, kModeSoftmax, 8, false>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1024, 1, 1);
    cfg.blockDim = dim3(kThreads, 1, 1);
    cfg.dynamicSmemBytes = SM::bytes(8);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1u << lg;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int count = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SM::bytes(8)) != cudaSuccess ||
        cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&count, kern, &cfg) != cudaSuccess)
      return 0;
    n = std::max(0, count) + 1;
    places[dev][lg].store(n, std::memory_order_relaxed);
  }
  return n - 1;
}

// Times of a launch (us, one call after another) by parts and 128-key blocks of a CTA, bf16, fitted to shapes of 1 to 148 items and 1 to 64 blocks
// (rms 1 to 7 %).  At head dimension 64 clusters share SMs once there are more than places at a CTA an SM (*Shared); more than the
// device holds at once would be a second wave, which costs more than a split saves (36 x 16 in eight parts 18.7 us, in four
// 14.8).  What the rule picks takes on average 0.3 % longer than the best form timed (softmax, 90 shapes), 0.5 % (chains), at head dimension 128 0.2 %; 8 % at worst.
namespace {
struct Whole { double fixed, block, full; };                    // full: over 100 CTAs
struct Split { double fixed, part, block, full; };              // full: over 100 CTAs; shared: times the share of SMs with two
constexpr Whole kWhole[2][2] = {{{2.89, 1.25, 0.32}, {2.39, 0.88, 0.36}}, {{3.65, 1.29, 0.70}, {2.84, 1.02, 0.69}}};      // [head dimension][no softmax]
constexpr Split kAlone[2][2] = {{{3.24, 0.18, 1.26, 0.36}, {2.76, 0.13, 0.87, 0.39}}, {{4.43, 0.24, 1.32, 0.89}, {3.75, 0.24, 1.04, 1.02}}};
constexpr Split kShared[2] = {{3.22, 0.44, 1.85, 0.80}, {3.40, 0.23, 1.10, 0.79}};
// the kernel with a thread a row
constexpr Split kRowAlone[2] = {{5.53, 0.04, 1.18, 0.65}, {4.37, 0.05, 0.69, 0.64}}, kRowShared[2] = {{6.49, 0.13, 1.65, 0.48}, {5.40, 0.13, 0.99, 0.42}};
// Blocks a part from which that one is taken at head dimension 64: a CTA an SM, two, and in eight parts, whose columns arrive in the K ring here.
constexpr int kRowFrom[2][2] = {{20, 8}, {12, 10}}, kRowFromEight = 8;
bool by_row(int parts, int own, int m, bool shared) { return own >= (parts == 8 ? kRowFromEight : kRowFrom[m][shared ? 1 : 0]); }
}  // namespace

// Where the lines lie, the forms without this kernel and with two CTAs an SM left out of count -> the choice now (us), items x blocks of
// sequences of 512 rows.  Softmax at head dimension 64: 24 x 1 5.3 -> 4.6, 24 x 2 6.5 -> 6.1, 24 x 4 7.3 -> 6.5 (4 parts), 24 x 16 11.0 -> 10.8 (4),
// 48 x 16 15.6 -> 14.4 (4), 100 x 2 6.9 -> 6.3, 148 x 4 10.2 -> 9.7, with a thread a row 24 x 64 25.3 -> 21.2 (8), 100 x 32 43.1 -> 33.6 (2),
// 148 x 64 83.1 -> 61.7 (2); at 128: 24 x 1 7.2 -> 5.2, 24 x 2 7.9 -> 6.7, 24 x 4 9.0 -> 8.3 (4), 24 x 16 14.3 -> 13.2 (4), 48 x 16 20.3 -> 18.9 (2),
// 100 x 32 64.4 -> 51.6; without a softmax 48 x 16 17.6 -> 14.5, 100 x 32 57.2 -> 39.5.
// At head dimension 64 the kernel with a thread a row costs less per block (1.18 against 1.26: no word from another warp before the
// exponentials) and more to combine.  This kernel / that one, split alike: 12 x 32 blocks in two parts 23.4 / 24.1, x 16 in four 9.1 / 10.5, in eight 7.7 / 8.7, 1 x 64 in eight
// 14.0 / 14.7; two CTAs an SM 148 x 16 in two 20.6 / 20.7, x 32 36.0 / 33.6.
// Unsplit and two CTAs an SM it serves one to four blocks: one block is faster here (200 x 1 5.8 -> 5.5), two to four are about as fast as
// in the kernel with 64-key blocks, whose references are those of shorter blocks (200 x 2 7.8 -> 7.7, 200 x 3 9.7 -> 10.2, 256 x 4
// 12.5 -> 13.1, at worst, of one tile a sequence, 296 x 3 11.8 -> 12.8; its error against float64 is 1 to 3 % larger at scale
// d^-0.5 and up to 10 % on uniform operands at scale 1); longer ones have no gain (296 x 8 20.2 -> 21.2).  Without a
// softmax it pays for up to three (148 x 1 4.4 -> 3.7, 200 x 1 4.7 -> 4.3, 200 x 2 5.9 -> 5.4).
// More than 148 items at head dimension 128: two CTAs an SM, each with a K and a V stage and P in the place of S, work beside each other, where the kernel
// with two tiles a CTA needs two tiles of one sequence.  One tile a sequence, us, before -> now: 150 x 4 17.7 -> 13.3, 296 x 1 9.0 -> 6.9, 450 x 8 61.3 -> 52.2, 600 x 3 38.4
// -> 35.9, 1000 x 8 136 -> 113, 2000 x 4 144 -> 116, without a softmax 150 x 4 14.0 -> 10.2, 600 x 4 46.5 -> 39.2; many items of one or two blocks are bound by what
// is loaded, which the other kernel asks for an item ahead (1000 x 1 28.9 -> 31.3, x 2 41.9 -> 43.7).  At 297 to 444 items, a second round of these CTAs, both builds in turn: chains
// of one block are slower here but for few rows (320 of 128 wide 8.97 -> 9.24, 400 10.6 -> 12.3, 80 wide 444 8.85 -> 9.14; of 48 rows and 64 keys 400 8.52 -> 8.21); with a softmax, and of
// two blocks, it depends on what an item brings: 128 wide with softmax 371 x 1 12.7 -> 12.1, 425 x 1 13.7 -> 15.5, without 400 of 160 keys 1.01, 425
// 17.0 -> 17.8; of 96 keys with softmax 425 0.95, 444 14.2 -> 15.0, of 64 444 13.7 -> 12.5; 96 wide 425 x 1 0.92 to 0.95, chains 444 x 2 1.00.  Two blocks with a softmax stay here, 371 x 2 19.7 -> 19.5, 425 x 2
// 20.3 -> 21.3: the other kernel's error is 3 to 13 % larger there (one block: the same).
// More tiles a sequence, up to 296 items: 296 x 1 8.0 -> 6.6, x 4 15.0 -> 14.0,
// with a softmax only as long as there are few blocks (160 x 8 21.1 -> 22.9, 150 x 16 35.9 -> 38.4; of 208 or 256 rows, 80 wide, x 4 12.4 -> 12.9; x 2 of 208
// keys 9.14 -> 9.01), without one always (150 x 64 122 -> 111); more items without a softmax
// where a sequence has two tiles and four blocks (512 x 16 of 208 rows 75.0 -> 69.3, 600 x 4 37.1 -> 33.6; x 2 19.3 -> 21.1; of 2048 rows 1024 x 4 37.0 -> 39.3) as long as the items are
// few or long: of 208 rows, 128 wide, 890 x 4 46.0 -> 44.6, 1000 x 4 50.0 -> 50.4, 2000 x 4 89.0 -> 95.8, x 8 158.6 -> 164.9, 2000 of 1200 keys 202 -> 195; 96 wide 1300 x 4 55.4 -> 55.8, 2000 x 4
// 78.5 -> 82.8, x 8 140 -> 141.
// Its error against float64 is 1 to 3 % smaller at scale d^-0.5, up to 14 % where the scores spread further: the other kernel keeps its references within 2^8 only.
AttnFew attention_few(int batch, int M, int L, int d, int widths, int mode) {
  constexpr int kSms = 148;
  const long long items = static_cast<long long>((M + kBM - 1) / kBM) * batch;
  const int blocks = (L + kBN - 1) / kBN;
  const int m = mode == kModeSoftmax ? 0 : 1, wide = d == 64 ? 0 : 1;
  AttnFew best = {1, false, false};
  if (items > kSms && d == 128) {
    const bool full = widths > 192;                        // of 256
    if (M <= kBM) {
      int most = 3 * kSms;
      if (m == 1 && blocks == 1) most = M <= 48 && L <= 96 ? 3 * kSms : 2 * kSms;
      else if (full && M > 80 && L > 64 && (m == 1 || blocks == 1)) most = L <= 96 ? 425 : L == kBN ? 380 : 400;
      best.two = items <= most || blocks >= 3;
    } else if (items <= 2 * kSms) {
      best.two = m == 1 || blocks <= (M <= 2 * kBM ? 3 : 4);
    } else {
      best.two = m == 1 && M <= 2 * kBM && blocks >= 4 && (items <= (full ? 7 : 9) * kSms || blocks >= (full ? 9 : 8));
    }
    best.here = best.two;
    return best;
  }
  if (items > 2 * kSms) return best;
  const Whole& w = kWhole[wide][m];
  double best_t = items <= kSms ? w.fixed + w.block * blocks + (items > 100 ? w.full : 0.0) : 1e30;
  for (int lg = 1; lg <= 3 && (1 << lg) <= blocks; ++lg) {
    const int parts = 1 << lg, own = (blocks + parts - 1) / parts, places = cluster_places(lg);
    if (items > (wide ? places : 2 * places)) break;
    const bool shared = items > places, row = !wide && by_row(parts, own, m, shared);
    const Split& s = row ? (shared ? kRowShared[m] : kRowAlone[m]) : shared ? kShared[m] : kAlone[wide][m];
    const double time = s.fixed + s.part * parts + s.block * own +
                        s.full * (shared ? static_cast<double>(items - places) / places : items * parts > 100 ? 1.0 : 0.0);
    if (time < best_t) {
      best.parts = parts;
      best.here = !row;
      best_t = time;
    }
  }
  if (d == 128) best.here = true;
  else if (best.parts > 1) return best;
  else if (items > kSms) best.here = blocks <= (m == 0 ? 4 : 3);
  else best.here = blocks <= (m == 0 ? 8 : 6);
  return best;
}

}  // namespace ditto_b200
