// fast_div.cuh -- divisions without CUDA's IEEE division sequence.
//
// div_by_recip: division by a per-ring constant whose reciprocal is known.
//
// Markstein's method (P. Markstein, "Computation of elementary functions on
// the IBM RISC System/6000 processor", IBM J. Res. Dev. 34(1), 1990; the
// correction step of Theorem 8.10 in Muller et al., Handbook of
// Floating-Point Arithmetic): with r = RN(1/d), the correctly rounded
// reciprocal, q0 = RN(x r) and the residual e = x - q0 d, exact in one fused
// multiply-add, q = RN(q0 + e r) is RN(x/d): the IEEE quotient, bit for bit.
// It is checked exhaustively on the GPU against CUDA's IEEE division for
// every pair of significands of the benchmark grids' denominators and for a
// sample of all others (tests/test_gpu_division.py).  Valid for normal x, d
// and quotients (no underflow or overflow on the way); x = 0 gives 0.
#pragma once

__device__ __forceinline__ float div_by_recip(float x, float d, float r) {
  const float q0 = __fmul_rn(x, r);
  const float e = __fmaf_rn(-q0, d, x);
  return __fmaf_rn(e, r, q0);
}

// The same where the quotient may overflow: there the correction would be
// inf - inf = NaN, and the quotient is the infinity itself.
__device__ __forceinline__ float div_by_recip_inf(float x, float d, float r) {
  const float q0 = __fmul_rn(x, r);
  const float q = __fmaf_rn(__fmaf_rn(-q0, d, x), r, q0);
  return isinf(q0) ? q0 : q;
}

// x / d in double from r = RN(1/d) (Markstein's method as in div_by_recip):
// the correctly rounded quotient for normal operands, in three operations.
__device__ __forceinline__ double div_by_recip_d(double x, double d, double r) {
  const double q0 = __dmul_rn(x, r);
  return __fma_rn(__fma_rn(-q0, d, x), r, q0);
}

// x / y for per-cell operands: the hardware's approximate reciprocal
// (rcp.approx, relative error below 2^-22), then the same residual
// correction: q0 = RN(x r), e = x - q0 y exact in one fused multiply-add,
// q = RN(q0 + e r).  The correction leaves q0's error times r's, so q is the
// IEEE quotient except when x/y lies within ~2^-22 ulp of a rounding
// boundary, and one ulp from it then (tests/test_gpu_division.py counts
// both).  For normal y and quotient; four instructions against the IEEE
// sequence's ~ten with its special-case branch.
__device__ __forceinline__ float rcp_approx(float y) {
  float r;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(y));
  return r;
}
__device__ __forceinline__ float div_refined(float x, float y) {
  const float r = rcp_approx(y);
  const float q0 = __fmul_rn(x, r);
  return __fmaf_rn(__fmaf_rn(-q0, y, x), r, q0);
}

// The transport's reciprocal is the flushing form: for a normal y (up to 2^126)
// it has the bits of rcp.approx.f32, and its product with x those of
// __fdividef(x, y) (no difference on 4e9 operand pairs), without the
// instructions by which those handle a subnormal y; a subnormal y counts as
// zero.  No divisor whose quotient the transport uses is subnormal: a slope is
// used where the product of its two differences is above zero, so at least one
// of them, and their sum, is above 2^-75; and S + 1e-20f, rounded to at least
// 2^-91 there, is zero or above that.  (Above 2^126 both forms give zero.)
__device__ __forceinline__ float rcp_ftz(float y) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y));
  return r;
}
// the fast quotient (2 ulp) of normal operands
__device__ __forceinline__ float div_fast(float x, float y) { return __fmul_rn(x, rcp_ftz(y)); }
// div_refined for a divisor that is zero, infinite or between 2^-126 and 2^126,
// the same bits: a square root is (2^-75 to 2^64).  Others keep the full range:
// flushing everywhere (densities, distances cubed) saved 1.4% of a substep
// (16 disks 317 -> 313 us, 1024x3072 345 -> 340 us) and lost the outer factors of
// four, where these divisors used to work.
__device__ __forceinline__ float div_refined_root(float x, float y) {
  const float r = rcp_ftz(y);
  const float q0 = __fmul_rn(x, r);
  return __fmaf_rn(__fmaf_rn(-q0, y, x), r, q0);
}
