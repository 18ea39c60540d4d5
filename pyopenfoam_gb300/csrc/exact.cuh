// Correctly rounded FP64 division and square root, and FP64 comparisons, on
// the integer and FP32 pipes.
//
// Why: GB300 issues about 2 FP64 operations per clock and SM (measured: fma
// 598 G/s, add / mul 509 G/s, compare 527 G/s) but 64-128 integer and FP32
// operations, so the assembly and corrector kernels, whose bits are the
// reference's and which therefore need every one of its IEEE divisions and
// square roots, were bound by those: __ddiv_rn 73 G/s, __dsqrt_rn 69 G/s on
// the whole chip.  div_rn measures 372 G/s and sqrt_rn 454 G/s, with the same
// bits (compared with __ddiv_rn / __dsqrt_rn on 6e9 operand pairs: any bit
// pattern, near-midpoint and exact quotients, mantissas at both ends).
//
// Method (long division with an approximate reciprocal, after Knuth, The Art
// of Computer Programming vol. 2, 4.3.1): the reciprocal of the divisor's top
// 24 bits (MUFU, error a few 2^-23) gives a first quotient of 22 fraction
// bits; twice, the exact remainder -- kept modulo 2^64, which suffices because
// it is small -- times that reciprocal gives the next ~20 bits.  The 64-bit
// quotient is then within 2 units of the true one (the bound was checked with
// the reciprocal moved by up to 2 ulp either way), so rounding it to 53 bits
// is right unless it lies within 3 units of a midpoint; there the sign of the
// exact remainder at the midpoint decides (a quotient or root of 53-bit
// numbers is never a midpoint itself).  The square root takes its digits the
// same way from m - s^2 with 1 / sqrt(m).  Operands outside the normal range,
// and quotients near its ends, go to the CUDA intrinsics.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace gbf {

__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ float rsqrt_approx(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Zeros, denormals, infinities, NaN and quotients near the ends of the
// exponent range.  Out of line: the callers keep their registers.  0 / b is
// common (upwind fluxes, zero fields), so it does not go through a division.
static __device__ __noinline__ double div_rn_slow(double a, double b) {
  const uint32_t bh = (uint32_t)__double2hiint(b);
  const uint32_t eb = (bh >> 20) & 0x7ffu;
  const uint32_t ah = (uint32_t)__double2hiint(a);
  if (((ah & 0x7fffffffu) | (uint32_t)__double2loint(a)) == 0u && eb - 1u < 2046u)
    return __hiloint2double((int)((ah ^ bh) & 0x80000000u), 0);
  return __ddiv_rn(a, b);
}
static __device__ __noinline__ double sqrt_rn_slow(double a) { return __dsqrt_rn(a); }

// y in [0.5, 1] (or s in [1, 2]) as a 22-bit fraction, rounded to nearest
__device__ __forceinline__ uint32_t fix22(float y) {
  return __float_as_uint(__fmaf_rn(y, 4194304.0f, 8388608.0f)) - 0x4b000000u;
}

// A division under way: the operands' words, mantissas and exponents and the
// quotient's digits.
struct DivDigits {
  uint32_t ah, bh, ea, eb;
  uint64_t ma, mb, q;  // q: mantissa quotient at 2^-63, within 2 units
  uint32_t up, half;   // up 1: quotient in [1, 2), 0: in (1/2, 1); half a result ulp of q

  __device__ __forceinline__ DivDigits(double a, double b) {
    ah = (uint32_t)__double2hiint(a);
    bh = (uint32_t)__double2hiint(b);
    const uint32_t al = (uint32_t)__double2loint(a), bl = (uint32_t)__double2loint(b);
    ea = (ah >> 20) & 0x7ffu;
    eb = (bh >> 20) & 0x7ffu;
    const uint32_t mah = (ah & 0xfffffu) | 0x100000u, mbh = (bh & 0xfffffu) | 0x100000u;
    ma = ((uint64_t)mah << 32) | al;
    mb = ((uint64_t)mbh << 32) | bl;
    // fa, fb in [1, 2): the mantissas' top 24 bits; quotient digits Q0 at
    // 2^-22, Q1 at 2^-48, q at 2^-63
    const float fa = __uint_as_float(__funnelshift_l(al, mah, 3) + 0x3f000000u);
    const float fb = __uint_as_float(__funnelshift_l(bl, mbh, 3) + 0x3f000000u);
    const float y = rcp_approx(fb);
    const int Y = (int)(fix22(y) << 8);
    const uint32_t Q0 = fix22(__fmul_rn(fa, y));
    const int64_t r0 = (int64_t)((ma << 22) - (uint64_t)Q0 * mb);
    const int D1 = __mulhi((int)(r0 >> 24), Y);
    const uint64_t Q1 = ((uint64_t)Q0 << 26) + (int64_t)D1;
    const int64_t r1 = (int64_t)((ma << 48) - Q1 * mb);
    const int D2 = __mulhi((int)(r1 >> 29), Y);
    q = (Q1 << 15) + (int64_t)(D2 >> 6);
    up = (uint32_t)(q >> 63);
    half = 512u << up;
  }
  // both operands and the quotient well inside the normal range
  __device__ __forceinline__ bool normal() const {
    return ea - 1u < 2046u && eb - 1u < 2046u && ea - eb + 1000u <= 2000u;
  }
  // within 3 units of a midpoint between two results
  __device__ __forceinline__ bool close() const {
    return (((uint32_t)q + half + 3u) & (2u * half - 1u)) < 6u;
  }
  __device__ __forceinline__ uint64_t rounded() const { return (q + half) >> (10 + up); }
  __device__ __forceinline__ double result(uint64_t m) const {
    const uint32_t ex = ea - eb + 1021u + up;
    const uint32_t hi = ((uint32_t)(m >> 32) + (ex << 20)) | ((ah ^ bh) & 0x80000000u);
    return __hiloint2double((int)hi, (int)(uint32_t)m);
  }
};

// a / b, the bits of __ddiv_rn.
__device__ __forceinline__ double div_rn(double a, double b) {
  const DivDigits d(a, b);
  if (!d.normal()) return div_rn_slow(a, b);
  uint64_t m = d.rounded();
  if (d.close()) {
    // mm - 1/2 is the midpoint next to q
    const uint64_t mm = (d.q + d.half + 3u) >> (10 + d.up);
    const int64_t rem = (int64_t)((d.ma << (54 - d.up)) - (2 * mm - 1) * d.mb);
    m = mm - (rem < 0);
  }
  return d.result(m);
}

// The common case of a / b without a branch, so that several overlap: where
// `ok` is false (6 in 1000 quotients lie close to a midpoint) the result is to
// be formed by div_rn.
__device__ __forceinline__ double div_try(double a, double b, bool& ok) {
  const DivDigits d(a, b);
  ok = d.normal() && !d.close();
  return d.result(d.rounded());
}

// sqrt(a), the bits of __dsqrt_rn: m = M / 2^52 in [1, 4), root digits S0 at
// 2^-22, S1 at 2^-46, s at 2^-62.
__device__ __forceinline__ double sqrt_rn(double a) {
  const uint32_t ah = (uint32_t)__double2hiint(a), al = (uint32_t)__double2loint(a);
  const uint32_t ea = ah >> 20;
  if (ea - 1u >= 2046u) return sqrt_rn_slow(a);
  const uint32_t odd = (ea & 1u) ^ 1u;
  const uint32_t mah = (ah & 0xfffffu) | 0x100000u;
  const uint64_t M = (((uint64_t)mah << 32) | al) << odd;
  const float f = __uint_as_float(__funnelshift_l(al, mah, 3) + 0x3f000000u + (odd << 23));
  const float y = rsqrt_approx(f);
  const int Y = (int)(fix22(y) << 8);
  const uint32_t S0 = fix22(__fmul_rn(f, y));
  const int64_t r0 = (int64_t)((M << 8) - (((uint64_t)S0 * S0) << 16));
  const int D1 = __mulhi((int)(r0 >> 13), Y);
  const uint64_t S1 = ((uint64_t)S0 << 24) + (int64_t)D1;
  const int64_t r1 = (int64_t)((M << 40) - S1 * S1);
  const int D2 = __mulhi((int)(r1 >> 23), Y);
  const uint64_t s = (S1 << 16) + (int64_t)(D2 >> 6);
  uint64_t m = (s + 512u) >> 10;
  if ((((uint32_t)s + 515u) & 1023u) < 6u) {
    const uint64_t mm = (s + 515u) >> 10, t = 2 * mm - 1;
    const int64_t rem = (int64_t)((M << 54) - t * t);
    m = mm - (rem < 0);
  }
  const uint32_t ex = ((ea + 1023u) >> 1) - 1u;
  return __hiloint2double((int)((uint32_t)(m >> 32) + (ex << 20)), (int)(uint32_t)m);
}

// Out of line, so that the product is not issued for every warp and predicated
// off (which would hold the FP64 pipe all the same); 0 * finite, common in
// fields and on axis-aligned faces, without it.
static __device__ __noinline__ double mul_rn_slow(double a, double b) {
  const unsigned long long ua = (unsigned long long)__double_as_longlong(a) << 1;
  const unsigned long long ub = (unsigned long long)__double_as_longlong(b) << 1;
  const unsigned long long inf2 = 0xffe0000000000000ull;  // infinity, sign shifted out
  if ((ua == 0 && ub < inf2) || (ub == 0 && ua < inf2))
    return __hiloint2double((__double2hiint(a) ^ __double2hiint(b)) & (int)0x80000000u, 0);
  return __dmul_rn(a, b);
}

// a * b, the bits of __dmul_rn, on the integer pipe: four 32 x 32 partial
// products, rounded to nearest even.  Alone it is no faster than the FP64 pipe
// (503 against 484 G/s on the chip), but the two run side by side: 928 G/s when
// every second operation is one of these.  For kernels that the FP64 pipe
// bounds, in place of about as many products as leave the pipes balanced: a
// warp takes 80 clocks of its SM quarter for one of these (a division or a root
// above about 100), 64 for an FP64 instruction.
__device__ __forceinline__ double mul_int(double a, double b) {
  const uint32_t ah = (uint32_t)__double2hiint(a), al = (uint32_t)__double2loint(a);
  const uint32_t bh = (uint32_t)__double2hiint(b), bl = (uint32_t)__double2loint(b);
  const uint32_t ea = (ah >> 20) & 0x7ffu, eb = (bh >> 20) & 0x7ffu, es = ea + eb;
  // zeros, denormals, infinities, NaN, products near the ends of the range
  if (ea - 1u >= 2046u || eb - 1u >= 2046u || es - 1100u > 1900u) return mul_rn_slow(a, b);
  // A: 64 bits, top one set; B: 53 bits; the product lies in [2^115, 2^117)
  const uint32_t Ah = __funnelshift_l(al, (ah & 0xfffffu) | 0x100000u, 11), Al = al << 11;
  const uint32_t Bh = (bh & 0xfffffu) | 0x100000u;
  const uint64_t p0 = (uint64_t)Al * bl;
  const uint64_t p1 = (uint64_t)Al * Bh + (p0 >> 32);
  const uint64_t p2 = (uint64_t)Ah * bl + (uint32_t)p1;
  const uint64_t top = (uint64_t)Ah * Bh + (p1 >> 32) + (p2 >> 32);  // [2^51, 2^53)
  const uint32_t low = (uint32_t)p2;  // the 32 bits below; then (uint32_t)p0, with no others set
  const uint32_t up = (uint32_t)(top >> 52);
  const uint64_t m = up ? top : (top << 1) | (low >> 31);
  const uint32_t r = up ? low : low << 1;
  const bool inc = r > 0x80000000u || (r == 0x80000000u && ((uint32_t)p0 != 0u || (m & 1u)));
  const uint64_t mm = m + (inc ? 1u : 0u);
  const uint32_t hi =
      ((uint32_t)(mm >> 32) + ((es - 1024u + up) << 20)) | ((ah ^ bh) & 0x80000000u);
  return __hiloint2double((int)hi, (int)(uint32_t)mm);
}

// Comparisons of doubles on the integer pipe (DSETP issues at the FP64 rate).
// a >= 0.0: false for NaN, true for -0.0.
__device__ __forceinline__ bool not_negative(double a) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(a);
  return b <= 0x7ff0000000000000ull || b == 0x8000000000000000ull;
}

// |a| clamped to at least 1e-30, NaN kept (torch.clamp(min=1e-30) of |a|).
__device__ __forceinline__ double clamp_abs_min(double a) {
  const long long b = __double_as_longlong(a) & 0x7fffffffffffffffLL;
  return b < __double_as_longlong(1e-30) ? 1e-30 : __longlong_as_double(b);
}

// a > t for a >= 0 or NaN (false for NaN) and a positive constant t.
__device__ __forceinline__ bool above(double a, double t) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(a);
  return b > (unsigned long long)__double_as_longlong(t) && b <= 0x7ff0000000000000ull;
}
__device__ __forceinline__ bool above_tiny(double a) { return above(a, 1e-30); }

// a >= t for a >= 0 or NaN (false for NaN) and a positive constant t.
__device__ __forceinline__ bool at_least(double a, double t) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(a);
  return b >= (unsigned long long)__double_as_longlong(t) && b <= 0x7ff0000000000000ull;
}

// max(|a|, 1e-30), 1e-30 for NaN.
__device__ __forceinline__ double max_abs_tiny(double a) {
  const double m = fabs(a);
  return above_tiny(m) ? m : 1e-30;
}

}  // namespace gbf
