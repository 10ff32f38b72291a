// The running maximum of a softmax row, as the attention kernels use it.
#pragma once
#include <cstdint>

#include "sm100_ptx.cuh"

namespace ditto_b200 {

// Up to this |m * c| the exponent of a score s is one fused multiply-add, s * c - mc: rounding mc = m * c moves all of a row's
// exponents by at most 2^-13, which is below the rounding of the 16-bit probabilities.
constexpr float kFusedReference = 4096.0f;

// How far (log2 units) a row's maximum may run ahead of its reference in the kernels for few items, split or not, and in the one with
// 64-key blocks, at the second block and later (8 throughout in the others).  The largest weights decide a row's rounding error: one that the
// reference was taken from is exactly 1, one above a stale reference is rounded like any other.
constexpr float kCloseSecondBlock = 1.0f, kCloseRescale = 5.0f;

// m is the (possibly stale) maximum that a row's exponentials refer to, c = scale * log2(e): a score's weight is
// ex2(fmaf(s, c, -mc)), at most 2^(rescale threshold).
//
// Rows whose reference is large -- -inf as long as there is no finite score, or a mask of the type's lowest value that fills all
// blocks so far -- have it subtracted from their scores instead (mc = 0): the rounding error of m * c alone could be an
// exponent beyond the range (it is 2^101 at the lowest float32), and the infinity that comes of it, or the NaN of
// (-inf) - (-inf), stays in the row's sum however small the row's weight becomes later.  Such rows join the vote on
// rescaling at every block; where there are none it costs a block nothing.
struct RowReference {
  float m = -INFINITY, mc = 0.0f;
  bool large = true;

  __device__ __forceinline__ explicit RowReference(float /*c*/) {}
  __device__ __forceinline__ float offset(float /*c*/) const { return mc; }
  // Whether this row asks its warp to rescale, given the maximum up to and including the present block.
  __device__ __forceinline__ bool asks(float m_new, float c, float threshold) const {
    return large || (m_new - m) * c > threshold;
  }
  // Moves the reference to m_new and returns the factor for what the row has accumulated.  A row whose reference stays gets
  // exactly 1: a warp rescales together, and without a finite score yet the difference is NaN.
  __device__ __forceinline__ float move(float m_new, float c) {
    const float f = m_new == m ? 1.0f : ex2_approx((m - m_new) * c);
    m = m_new;
    mc = m * c;
    large = !(fabsf(mc) <= kFusedReference);
    return f;
  }
  // Behind move, by the whole warp: the present block's scores of rows with a large reference.
  template <int N>
  __device__ __forceinline__ void subtract(uint32_t (&s)[N]) {
    if (__any_sync(0xffffffffu, large)) {
      const float ref = large && m != -INFINITY ? m : 0.0f;      // (scores of -inf stay what they are)
#pragma unroll
      for (int i = 0; i < N; ++i) s[i] = __float_as_uint(__uint_as_float(s[i]) - ref);
      if (large) mc = 0.0f;
    }
  }
};

// The rule of the kernels that take a row's blocks in turn with 128 keys each: the reference starts at m * c = -2^40 and not at
// -inf, so that there is no difference of infinities and blocks whose scores all lie below -- -inf, masks of the lowest
// values -- weigh nothing.  References as large as that were no use before: rounding their product with c moves an exponent by
// 2^16.  No instruction more in the loop: the two-tile kernel has no registers left (RowReference made it 4 to 7 % slower).
struct PlainReference {
  float m;

  __device__ __forceinline__ explicit PlainReference(float c) : m(-1099511627776.0f / c) {}
  __device__ __forceinline__ float offset(float c) const { return m * c; }
  __device__ __forceinline__ bool asks(float m_new, float c, float threshold) const { return (m_new - m) * c > threshold; }
  __device__ __forceinline__ float move(float m_new, float c) {
    const float f = ex2_approx((m - m_new) * c);
    m = m_new;
    return f;
  }
  template <int N>
  __device__ __forceinline__ void subtract(uint32_t (&)[N]) {}
};

// Weights 2^(s c - mc) of two scores (c2 and nmc2 hold c and -mc twice), with the scale-and-subtract of both in one instruction.
// on_fma: on the multiply-add pipe instead of the special-function unit, for rows with a RowReference: exponents there stay below
// the few units of its rescale threshold.  Behind a PlainReference the rounding of m * c alone can pass what ex2_fma_f32x2 takes.
__device__ __forceinline__ uint64_t softmax_weights(uint32_t s0, uint32_t s1, uint64_t c2, uint64_t nmc2, bool on_fma) {
  const uint64_t x = fma_f32x2(pack_f32x2(__uint_as_float(s0), __uint_as_float(s1)), c2, nmc2);
  if (on_fma) return ex2_fma_f32x2(x);
  float x0, x1;
  unpack_f32x2(x, x0, x1);
  return pack_f32x2(ex2_approx(x0), ex2_approx(x1));
}

// Which of a row's pairs of weights the multiply-add pipe computes in the kernels whose exponentials are shared out: three of every 32.
__device__ __forceinline__ constexpr bool weights_on_fma(int pair) { return pair % 32 == 7 || pair % 32 == 15 || pair % 32 == 31; }

}  // namespace ditto_b200
