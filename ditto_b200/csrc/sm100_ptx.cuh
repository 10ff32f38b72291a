// Thin inline-PTX layer for sm_100a: mbarrier, TMA (cp.async.bulk.tensor, no
// cluster multicast anywhere), tcgen05 MMA / TMEM management, UMMA descriptors.
//
// Every wait on an mbarrier is bounded: after kSpinLimit polls it records an
// error code in a CTA-wide abort word (shared memory) and returns false, and
// all later waits in that CTA return false at once, so the CTA drains to its
// normal teardown (TMEM freed) instead of hanging the device.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "tmem_ops_gen.cuh"

namespace ditto_b200 {

// ---------------------------------------------------------------- addresses
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ---------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// Make generic-proxy writes to shared memory visible to the async proxy (TMA, UMMA).
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// One arrival for the warp, once every lane has come here.
__device__ __forceinline__ void mbar_arrive_warp(uint64_t* bar, int lane) {
  __syncwarp();
  if (lane == 0) mbar_arrive(bar);
}
// Arrive on the barrier at the same shared-memory offset in CTA `cta` of this cluster.
__device__ __forceinline__ void mbar_arrive_cluster(uint64_t* bar, uint32_t cta) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(bar)), "r"(cta));
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(remote) : "memory");
}
// A translation unit may define DITTO_TRY_WAIT_HINT_NS before including this header: its polls then
// carry the optional suspend-time hint of mbarrier.try_wait (the thread may stay suspended that long
// before the poll returns false).  The MLP chain kernel does: its waits are long and many, and fewer
// wake-ups of the waiting warps leave more issue slots to the working ones (+3 % measured); the
// attention kernels and the CTA-pair kernel lose 1-5 % with it and keep the default.
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
#ifdef DITTO_TRY_WAIT_HINT_NS
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity), "r"(static_cast<uint32_t>(DITTO_TRY_WAIT_HINT_NS))
      : "memory");
#else
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
#endif
  return ok != 0;
}

// polls before a bounded wait gives up: about a second either way (a hinted poll may take the hint's time)
#ifdef DITTO_TRY_WAIT_HINT_NS
constexpr uint32_t kSpinLimit = 1u << 18;
#else
constexpr uint32_t kSpinLimit = 1u << 22;
#endif

// Bounded wait.  `abort_word` lives in shared memory; `code` identifies the
// waiter so a timeout can be traced from the host-visible status word.
// A translation unit may define DITTO_WAIT_OUT_OF_LINE before including this header: everything after a wait's first poll
// is then a function of its own.  Inlined, every wait brings its loop, its clock and its error path into the code that a
// launch of a few microseconds has to fetch before it can run it; called, it costs long loops that wait often their registers.
// Measured, us, inline -> called: attention of one Bert-Base sequence 7.78 -> 7.39, its plain chain 5.96 -> 5.57, MLP chain 512 x 768 -> 3072 -> 768 13.8 -> 13.3; the
// other way with two tiles a CTA, 1024 slices of 2048 x 128 2068 -> 2182.
#ifdef DITTO_WAIT_OUT_OF_LINE
static __device__ __noinline__
#else
__device__ __forceinline__
#endif
bool mbar_wait_polling(uint64_t* bar, uint32_t parity, volatile uint32_t* abort_word, uint32_t code) {
  for (uint32_t spin = 0; spin < kSpinLimit; ++spin) {
    if (mbar_try_wait(bar, parity)) return true;
    if (*abort_word != 0u) return false;
    if (spin > 4096u) __nanosleep(64);
  }
  atomicCAS(const_cast<uint32_t*>(abort_word), 0u, code);
  return false;
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile uint32_t* abort_word,
                                          uint32_t code) {
  return mbar_try_wait(bar, parity) || mbar_wait_polling(bar, parity, abort_word, code);
}

// ---------------------------------------------------------------- TMA
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}
// 2-D tiled load global -> this CTA's shared memory, completion on `bar`.
// x is the innermost (contiguous) coordinate and must keep x * elem_size a
// multiple of 16 bytes.
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}
// 2-D tiled store shared -> global (bulk async group).
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, const void* src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(map),
               "r"(smem_u32(src)), "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void tma_store_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void tma_store_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}

// ---------------------------------------------------------------- TMEM / tcgen05
// TMEM addresses: bits [31:16] = lane (0..127), bits [15:0] = 32-bit column (0..511).
__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before_sync() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after_sync() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// All MMAs issued so far by this thread arrive (once) on `bar` when they retire.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// D[tmem] (+)= A[smem] * B[smem]; kind::f16 covers fp16 and bf16 inputs with fp32 accumulate.
__device__ __forceinline__ void umma_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem].
__device__ __forceinline__ void umma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Converged-warp issue.  tcgen05.mma / commit are single-thread instructions, but a warp that
// stays converged and predicates them on an elect.sync lane keeps descriptors and addresses in
// uniform registers; measured on B200 this sustains one 128 x 128 x 16 MMA per 64 clocks (and a
// 128 x 64 x 16 one per 32), whereas a divergent `if (lane == 0)` loop around computed
// descriptors does not.  `issuer` is the value returned by elect_one() for the calling lane.
__device__ __forceinline__ uint32_t elect_one() {
  uint32_t is_elected;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(is_elected));
  return is_elected;
}
__device__ __forceinline__ void umma_ss_elected(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                                uint32_t accumulate, uint32_t issuer) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(issuer)
      : "memory");
}
__device__ __forceinline__ void umma_ts_elected(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                                uint32_t accumulate, uint32_t issuer) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(issuer)
      : "memory");
}
__device__ __forceinline__ void umma_commit_elected(uint64_t* bar, uint32_t issuer) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.b32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
      ::"r"(smem_u32(bar)), "r"(issuer)
      : "memory");
}

// The same, arriving (once) on the barrier at this offset in every CTA of the cluster named by `cta_mask`
// (bit r = cluster rank r): a consumer's MMA completion releases a buffer in the producer's CTA directly.
__device__ __forceinline__ void umma_commit_mcast_elected(uint64_t* bar, uint32_t cta_mask, uint32_t issuer) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t.reg .b16 lo, hi;\n\t"
      "setp.ne.b32 q, %2, 0;\n\t"
      "mov.b32 {lo, hi}, %1;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], lo;\n\t}"
      ::"r"(smem_u32(bar)), "r"(cta_mask), "r"(issuer)
      : "memory");
}

// ---------------------------------------------------------------- CTA pairs (cta_group::2)
// Two CTAs with consecutive cluster ranks (even = leader) execute one MMA of M = 256: each holds
// its 128 rows of A and half of B's N extent in its own shared memory (same offsets in both) and
// receives its 128 rows of D in its own TMEM.  Only the leader issues; completion is signalled to
// barriers at the same offset in both CTAs.  No load here is multicast: each CTA fetches its own
// operands, and its TMA loads report their bytes to the leader's barrier.
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The two halves of a cluster barrier.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t map_to_cta(uint32_t local_smem_addr, uint32_t cta) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local_smem_addr), "r"(cta));
  return remote;
}
// distributed shared memory: addresses from map_to_cta
__device__ __forceinline__ void ld_cluster_v2(uint32_t addr, float& x, float& y) {
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(x), "=f"(y) : "r"(addr) : "memory");
}
__device__ __forceinline__ void st_cluster_v2(uint32_t addr, float x, float y) {
  asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(x), "f"(y) : "memory");
}
__device__ __forceinline__ void st_cluster_v4(uint32_t addr, float x, float y, float z, float w) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// 2-D tiled load into this CTA's shared memory whose byte count is reported to `bar_cluster_addr`,
// a shared::cluster address that may lie in the pair's leader CTA.
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, uint32_t bar_cluster_addr, int x,
                                                 int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(bar_cluster_addr), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void umma_ss_pair_elected(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                                     uint32_t accumulate, uint32_t issuer) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(issuer)
      : "memory");
}
// Arrive (once) on the barrier at this offset in every CTA named by `cta_mask` when all MMAs issued
// so far by this thread have retired.
__device__ __forceinline__ void umma_commit_pair_elected(uint64_t* bar, uint32_t cta_mask, uint32_t issuer) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t.reg .b16 lo, hi;\n\t"
      "setp.ne.b32 q, %2, 0;\n\t"
      "mov.b32 {lo, hi}, %1;\n\t"
      "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], lo;\n\t}"
      ::"r"(smem_u32(bar)), "r"(cta_mask), "r"(issuer)
      : "memory");
}

// Shared-memory matrix descriptor for 128-byte-swizzled tiles (what a TMA box
// with CU_TENSOR_MAP_SWIZZLE_128B and a 128-byte inner extent produces).
//   bits [0,14)  start address >> 4        bits [16,30) leading byte offset >> 4
//   bits [32,46) stride byte offset >> 4   bits [46,48) descriptor version (1 on sm_100)
//   bits [61,64) layout type (2 = SWIZZLE_128B)
// K-major operand (rows of 64 contiguous K elements): sbo = bytes between
// 8-row groups (1024 when rows are packed), lbo unused.
// MN-major operand (rows of 64 contiguous M/N elements, one row per K index):
// sbo = bytes between groups of 8 K-rows (1024), lbo = bytes between
// successive 64-element chunks along M/N.
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFFu) << 16;
  d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFFu) << 32;
  d |= 1ull << 46;
  d |= 2ull << 61;
  return d;
}

// Instruction descriptor for kind::f16, fp32 accumulate, dense.
//   [4,6) D format (1 = f32)  [7,10) A format (0 = f16, 1 = bf16)  [10,13) B format
//   [15] A major (0 = K, 1 = MN)  [16] B major  [17,23) N >> 3  [24,29) M >> 4
__host__ __device__ constexpr uint32_t umma_idesc_f16(bool bf16, uint32_t m, uint32_t n, bool a_mn_major,
                                                      bool b_mn_major) {
  return (1u << 4) | ((bf16 ? 1u : 0u) << 7) | ((bf16 ? 1u : 0u) << 10) | ((a_mn_major ? 1u : 0u) << 15) |
         ((b_mn_major ? 1u : 0u) << 16) | ((n >> 3) << 17) | ((m >> 4) << 24);
}

// ---------------------------------------------------------------- programmatic dependent launch
// wait: returns once the grids this one depends on have completed and their memory is visible (a no-op
// when the kernel was launched without the programmatic-serialization attribute);
// launch_dependents: lets the next kernel in the stream begin (it blocks at its own wait).
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// ---------------------------------------------------------------- math
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Two float32 values in a 64-bit register: one instruction of the multiply-add pipe for both.
__device__ __forceinline__ uint64_t pack_f32x2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack_f32x2(uint64_t v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// The larger of two values, NaN if either is.
__device__ __forceinline__ float max_nan(float a, float b) {
  float d;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
  return d;
}

// 2^x of a pair on the multiply-add pipe, for softmax exponents that a RowReference bounds: x <= 127 (above, the exponent's bits run
// over into the sign, where ex2.approx gives infinity); -inf and what lies below -127 give 0, NaN stays NaN.
// x = n + f with n the nearest integer: adding 1.5 * 2^23 + 127 leaves n + 127 in the low bits of the sum, which shifted up
// are 2^n.  2^f = 1 + f q(f) on [-1/2, 1/2] with q of degree 5, least maximum relative error (iteratively reweighted least squares, one
// coefficient after the other fixed at its float32 value): 3.0e-9.  As evaluated, against float64, largest / root mean square: 6.6e-8 / 2.6e-8;
// ex2.approx measured the same way 1.45e-7 / 5.3e-8.  (Degree 4: 1.7e-7 / 6.6e-8, more than it stands in for.)
__device__ __forceinline__ uint64_t ex2_fma_f32x2(uint64_t x_in) {
  float x0, x1, t0, t1;
  unpack_f32x2(x_in, x0, x1);
  const uint64_t x = pack_f32x2(max_nan(x0, -127.0f), max_nan(x1, -127.0f));
  constexpr float kShift = 12582912.0f + 127.0f;
  const uint64_t t = add_f32x2(x, pack_f32x2(kShift, kShift));
  const uint64_t n = add_f32x2(t, pack_f32x2(-kShift, -kShift));
  const uint64_t f = fma_f32x2(n, pack_f32x2(-1.0f, -1.0f), x);
  unpack_f32x2(t, t0, t1);
  const uint64_t s = pack_f32x2(__uint_as_float(__float_as_uint(t0) << 23), __uint_as_float(__float_as_uint(t1) << 23));
  uint64_t q = fma_f32x2(f, pack_f32x2(0x1.416b52p-13f, 0x1.416b52p-13f), pack_f32x2(0x1.5f082ep-10f, 0x1.5f082ep-10f));
  q = fma_f32x2(q, f, pack_f32x2(0x1.3b2de0p-7f, 0x1.3b2de0p-7f));
  q = fma_f32x2(q, f, pack_f32x2(0x1.c6af7cp-5f, 0x1.c6af7cp-5f));
  q = fma_f32x2(q, f, pack_f32x2(0x1.ebfbdcp-3f, 0x1.ebfbdcp-3f));
  q = fma_f32x2(q, f, pack_f32x2(0x1.62e430p-1f, 0x1.62e430p-1f));
  return fma_f32x2(q, mul_f32x2(f, s), s);
}

// Two exponentials per special-function instruction: 2^x0, 2^x1 evaluated on the packed 16-bit pair and
// returned packed (low half = first).  The softmax rounds its probabilities to the 16-bit input type
// before the second GEMM anyway; what is lost is the precision of the argument (x is rounded to 16 bit
// before the exponential instead of after).
template <bool BF16>
__device__ __forceinline__ uint32_t ex2_packed(float x0, float x1) {
  uint32_t w;
  if constexpr (BF16) {
    asm("{\n\t.reg .b32 t;\n\tcvt.rn.bf16x2.f32 t, %2, %1;\n\tex2.approx.ftz.bf16x2 %0, t;\n\t}" : "=r"(w) : "f"(x0), "f"(x1));
  } else {
    asm("{\n\t.reg .b32 t;\n\tcvt.rn.f16x2.f32 t, %2, %1;\n\tex2.approx.f16x2 %0, t;\n\t}" : "=r"(w) : "f"(x0), "f"(x1));
  }
  return w;
}
__device__ __forceinline__ float2 unpack_f16x2(uint32_t w) {
  float2 r;
  asm("{\n\t.reg .b16 lo, hi;\n\tmov.b32 {lo, hi}, %2;\n\tcvt.f32.f16 %0, lo;\n\tcvt.f32.f16 %1, hi;\n\t}" : "=f"(r.x), "=f"(r.y) : "r"(w));
  return r;
}
__device__ __forceinline__ float2 unpack_bf16x2(uint32_t w) {
  return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}

}  // namespace ditto_b200
