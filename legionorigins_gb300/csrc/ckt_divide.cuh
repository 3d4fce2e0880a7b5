// ckt_divide.cuh -- correctly rounded fp32 quotients by a loop-invariant
// divisor without the divide routine.
//
// Every quotient of the reference's wire recurrence has a divisor that does
// not change inside the inner loop: dt, the wire's resistance R and its
// capacitance C (apps/circuit/circuit_gpu.cu:119-128, circuit.cc:391-400).
// EXACT mode must round each of them exactly as IEEE a / b does, because the
// recurrence's gain L/(dt R) >> 1 magnifies any one-ulp difference at every
// step.  Two constructions give RN(a / b) for a precomputed divisor:
//
//  * Division by dt = (float)1e-6, one multiply and one FMA:
//        q = RN(a*zh + RN(a*zl)),  zh = RN(1/dt) = 1e6,  zl = RN(1/dt - zh).
//    a*(zh + zl) is a/dt to about 2^-47 relative, so q can differ from
//    RN(a/dt) only where a/dt lies within that distance of a rounding
//    boundary; which dividends do is a property of the divisor (Brisebarre,
//    Muller and Raina, "Accelerating correctly rounded floating-point
//    division when the divisor is known in advance", IEEE Trans. Computers
//    53(8), 2004).  For this divisor every one of the 2^32 float dividends
//    was compared with IEEE division (tests/test_divide.py on the CPU,
//    tests/test_gpu_divide.py against __fdiv_rn on the GPU): q equals
//    RN(a/dt) for all of them, zeros, infinities and NaN included, except 98
//    dividends below 2^-124 in magnitude, where a*zl underflows.  Dividends
//    below kDtTiny therefore leave the fast path.
//
//  * Any other divisor b (per wire, or a dt other than (float)1e-6), three
//    FMAs and a multiply with y = RN(1/b), yl = RN(1/b - y), nb = -b:
//        q0 = RN(a*y + RN(a*yl))   within 1 ulp of a/b (error ~2^-46 a/b
//                                  plus half an ulp)
//        r  = RN(a + nb*q0)        exact, because q0 is within 1 ulp
//        q  = RN(q0 + r*y)         = RN(a/b) by Markstein's theorem
//    (P. W. Markstein, "Computation of elementary functions on the IBM RISC
//    System/6000 processor", IBM J. Res. Dev. 34(1), 1990; J.-M. Muller et
//    al., Handbook of Floating-Point Arithmetic, Birkhauser, the chapter on
//    FMA-based division).  The theorem needs every intermediate to stay
//    clear of overflow and of underflow: with |b| in [2^bmin, 2^bmax] and
//    |a| in [lo, hi] below, |a/b| lies in [2^-70, 2^120], the remainder's
//    quantum 2^(eb+eq-46) is at least 2^-147 (so r is representable), and
//    RN(a*yl)'s absolute error is far below an ulp of the quotient.
//    Dividends outside [lo, hi] -- zero, tiny, huge, infinite -- take
//    wide_quot below; NaN dividends stay on the fast path, where every
//    operation returns NaN as IEEE division does.
//
//  * Dividends outside [lo, hi] (wide_quot): scaling by a power of two
//    commutes with rounding while the scaled values stay normal, so
//    RN(a/b) = RN((a s)/b) / s.  A huge |a| in (hi, 2^128) is scaled by
//    2^-64 into (2^26, 2^64), inside both guarded ranges; the quotient is
//    normal, and when RN(a/b) overflows the scaled quotient is at least
//    2^64 (2^128 - 2^103, the overflow threshold, scaled to the midpoint
//    2^64 - 2^39, rounds up to the even 2^64), so multiplying back gives
//    the same infinity.  A tiny nonzero |a| below lo, subnormals included,
//    is scaled by 2^110 into [2^-39, 2^60), inside both ranges; multiplying
//    back is exact while RN(a/b) is normal, which |a| >= 2^-125 |b|
//    guarantees.  Zeros and infinities are a times RN(1/b), exact for them.
//    Dividends whose quotient may be subnormal (subnormal_quot) are left to
//    the divide routine.
//
//  * A checked divisor (check_split), one multiply and one FMA, as for dt:
//        q = RN(a*y + RN(a*yl)).
//    Scale a = A 2^-23 and b = B 2^-23 to 24-bit integers A, B in [2^23, 2^24)
//    (only signs and exponents change).  For A < B the quotient lies in
//    (1/2, 1) and the distance of a/b from the rounding boundary
//    (2m+1)/2^25 is |r| / (2^48 b) with r = 2^25 A - (2m+1) B; for A >= B it
//    is |r| / (2^47 b) with r = 2^24 A - (2m+1) B.  The sum rounded at the
//    end is off a/b by at most a |1/b - y - yl| + ulp(a yl) / 2 < 2^-49 + 2^-49
//    (|yl| <= 2^-25, so ulp(yl) <= 2^-49 and ulp(a yl) <= 2^-48).  b < 2, so
//    only A < B with |r| = 1 can be rounded to the wrong side; r is even for
//    even B, so only odd B, and A = +-2^-25 mod B: one dividend per divisor
//    (the other is below 2^23), which check_split finds by a modular inverse
//    and tries (Brisebarre, Muller and Raina's method, cited above, bounds and
//    tries the candidates the same way).  1.27% of all divisors fail there;
//    moving yl by one ulp up or down cures 95% of those.  The moved sum is off
//    by less than 2.5 2^-48, so its candidates are A < B with |r| in {1, 3}
//    and A >= B with |r| = 1, all tried.  A divisor that stays unchecked
//    (0.06%) keeps the corrected quotient, or takes the next form.  The bound
//    needs RN(a*yl) normal: |a| >= kSplitLo (|yl| is 0 or at least
//    2^-48 / |b|, and |b| <= 2^30).
//
//  * The same with the product rounded toward zero (cut_yl):
//        q = RN(a*y + RZ(a*yl)).
//    Other divisors fail here than above: with yl as made or one ulp larger
//    in magnitude 99.8% pass, and all of those left unchecked above that were
//    tried (2,000).  A warp's lanes share one form, so a warp with an
//    unchecked divisor takes this one if all its divisors pass.  With
//    |yl| <= 2^-25 the truncation is below 2^-48 and the sum is off a/b by
//    less than 2.5 2^-48 (1.5 2^-48 as made), so the dividends to try are
//    those with |r| < 5 for A < B and |r| < 2.5 for A >= B.  r has B's power
//    of two, 2^k, as a factor and is odd beyond it; with B = 2^k B' they are
//    A = +-2^(k-25) and +-3 2^(k-25) mod B' (A < B), +-2^(k-24) mod B'
//    (A >= B), and none from k = 3 on.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace ckt {

// dt = (float)1e-6 (DELTAT, apps/circuit/circuit.h:44) and its split
// reciprocal.
constexpr uint32_t kDtBits = 0x358637bdu;
constexpr uint32_t kDtZhBits = 0x49742400u;  // RN(1/dt) = 1e6
constexpr uint32_t kDtZlBits = 0x3b257666u;  // RN(1/dt - 1e6) = 2.5247573e-3
// The split-reciprocal quotient by dt is exact for |a| >= kDtTiny.
constexpr float kDtTiny = 0x1p-118f;

// Eligible divisors and guarded dividend ranges of the corrected quotient.
// R: |b| in [2^-8, 2^8], |a| in [2^-50, 2^100];
// C and a general dt: |b| in [2^-30, 2^30], |a| in [2^-40, 2^90].
// wide_quot is exact for every dividend but those subnormal_quot flags.
constexpr float kRMin = 0x1p-8f, kRMax = 0x1p8f, kRLo = 0x1p-50f, kRHi = 0x1p100f;
constexpr float kCMin = 0x1p-30f, kCMax = 0x1p30f, kCLo = 0x1p-40f, kCHi = 0x1p90f;

__device__ __forceinline__ float dt_zh() { return __int_as_float((int)kDtZhBits); }
__device__ __forceinline__ float dt_zl() { return __int_as_float((int)kDtZlBits); }

// a / (float)1e-6 for |a| >= kDtTiny, zeros, infinities and NaN.
__device__ __forceinline__ float dt_quot(float a) {
  return __fmaf_rn(a, dt_zh(), __fmul_rn(a, dt_zl()));
}
__device__ __forceinline__ float2 dt_quot2(float2 a) {
  const float zh = dt_zh(), zl = dt_zl();
  return __ffma2_rn(a, make_float2(zh, zh), __fmul2_rn(a, make_float2(zl, zl)));
}

// Per-divisor constants of the corrected quotient.
struct Recip {
  float nb, y, yl;
};
__device__ __forceinline__ Recip make_recip(float b) {
  Recip r;
  r.nb = -b;
  r.y = __frcp_rn(b);
  // 1 - b*y is exact for a correctly rounded reciprocal, so yl = RN(1/b - y)
  r.yl = __fdiv_rn(__fmaf_rn(-b, r.y, 1.0f), b);
  return r;
}

__device__ __forceinline__ bool divisor_ok(float b, float bmin, float bmax) {
  const float m = fabsf(b);
  return m >= bmin && m <= bmax;  // false for NaN
}

// True when the corrected quotient may not equal RN(a/b): |a| outside
// [lo, hi].  False for NaN.
__device__ __forceinline__ bool outside(float a, float lo, float hi) {
  const float m = fabsf(a);
  return (m < lo) | (m > hi);
}

__device__ __forceinline__ float recip_quot(float a, const Recip &k) {
  const float q0 = __fmaf_rn(a, k.y, __fmul_rn(a, k.yl));
  const float r = __fmaf_rn(q0, k.nb, a);
  return __fmaf_rn(r, k.y, q0);
}

// Two divisions at once (paired FP32 instructions); each lane rounds exactly
// as recip_quot.
struct Recip2 {
  float2 nb, y, yl;
};
__device__ __forceinline__ Recip2 make_recip2(float bx, float by) {
  const Recip a = make_recip(bx), b = make_recip(by);
  Recip2 r;
  r.nb = make_float2(a.nb, b.nb);
  r.y = make_float2(a.y, b.y);
  r.yl = make_float2(a.yl, b.yl);
  return r;
}
__device__ __forceinline__ float2 recip_quot2(float2 a, const Recip2 &k) {
  const float2 q0 = __ffma2_rn(a, k.y, __fmul2_rn(a, k.yl));
  const float2 r = __ffma2_rn(q0, k.nb, a);
  return __ffma2_rn(r, k.y, q0);
}

// a / b for a divisor check_split accepted, kSplitLo <= |a| < infinity or NaN.
// Divisors below kSplitMin are left out: a * yl could overflow beside a
// finite a, to an infinity of the wrong sign that nothing would show.
constexpr float kSplitLo = 0x1p-48f, kSplitMin = 0x1p-20f;
__device__ __forceinline__ float split_quot(float a, const Recip &k) {
  return __fmaf_rn(a, k.y, __fmul_rn(a, k.yl));
}
__device__ __forceinline__ float2 split_quot2(float2 a, const Recip2 &k) {
  return __ffma2_rn(a, k.y, __fmul2_rn(a, k.yl));
}

// b's significand in [1, 2) and the parts of its reciprocal: a power of two
// and a sign away from b's own, exact.
struct SplitBase {
  Recip n;
  uint32_t B, A1;  // the significand as an integer, 2^-25 mod B (odd B)
};
__device__ __forceinline__ SplitBase split_base(const Recip &k) {
  SplitBase s;
  const uint32_t bits = __float_as_uint(-k.nb);
  const float scale = __uint_as_float(bits & 0xff800000u);
  s.n.nb = -__uint_as_float(0x3f800000u | (bits & 0x7fffffu));
  s.n.y = __fmul_rn(k.y, scale);
  s.n.yl = __fmul_rn(k.yl, scale);
  const uint32_t B = (bits & 0x7fffffu) | 0x800000u;
  uint32_t x = (3u * B) ^ 2u;  // B^-1 mod 2^5, then by Newton mod 2^10, 2^20, 2^32
  x *= 2u - B * x;
  x *= 2u - B * x;
  x *= 2u - B * x;
  const uint32_t t = (0u - x) & 0x1ffffffu;  // -B^-1 mod 2^25
  s.B = B;
  s.A1 = (uint32_t)((1ull + (uint64_t)B * t) >> 25);
  return s;
}
// True when the split quotient with yl rounds a = A 2^-23 like the corrected
// one; A outside [2^23, 2^24) is no candidate.
__device__ __forceinline__ bool split_right_at(uint32_t A, const Recip &n, float yl) {
  const float a = __fmul_rn(__uint2float_rn(A), 0x1p-23f);
  const bool right = __fmaf_rn(a, n.y, __fmul_rn(a, yl)) == recip_quot(a, n);
  return (A - 0x800000u >= 0x800000u) | right;
}
// Whether split_quot is RN(a/b) for every dividend of its range, k as
// make_recip gives it.  (A1 and B - A1 add up to B < 2^24: only the larger
// can be a significand.)
__device__ __forceinline__ bool split_as_made(const Recip &k) {
  const SplitBase s = split_base(k);
  return !(s.B & 1u) | split_right_at(max(s.A1, s.B - s.A1), s.n, s.n.yl);
}
// How many ulps (-1 or 1) yl must move for that; 0: neither helps.  (The
// corrected quotient stays exact with the moved yl: its q0 is still within
// an ulp.)
__device__ __forceinline__ int split_move(const Recip &k) {
  const SplitBase s = split_base(k);
  const uint32_t B = s.B, A1 = s.A1;
  const uint32_t A2 = 2u * A1 >= B ? 2u * A1 - B : 2u * A1;  // 2^-24 mod B
  const uint32_t A3 = A1 + A2 >= B ? A1 + A2 - B : A1 + A2;  // 3 2^-25 mod B
#pragma unroll 1
  for (int d = -1; d <= 1; d += 2) {
    const float yl = __int_as_float(__float_as_int(s.n.yl) + d);
    if (split_right_at(max(A1, B - A1), s.n, yl) && split_right_at(max(A3, B - A3), s.n, yl) &&
        split_right_at(B + A2, s.n, yl) && split_right_at(2u * B - A2, s.n, yl))
      return d;
  }
  return 0;
}
// Checks N divisors, moving their yl where that makes the split quotient
// right; returns the mask of those it is right for.  The moves are rare
// (1.27% of divisors) and come last, one divisor of each lane at a time,
// whichever it is.
template <int N>
__device__ __forceinline__ uint32_t check_split(const float (&nb)[N], const float (&y)[N],
                                                float (&yl)[N]) {
  uint32_t fail = 0, right = 0;
#pragma unroll
  for (int d = 0; d < N; d++) {
    const Recip k = {nb[d], y[d], yl[d]};
    if (fabsf(nb[d]) < kSplitMin) continue;
    if (split_as_made(k)) right |= 1u << d;
    else fail |= 1u << d;
  }
#pragma unroll 1
  while (fail) {
    const uint32_t bit = fail & (0u - fail);
    Recip k = {nb[0], y[0], yl[0]};
#pragma unroll
    for (int d = 1; d < N; d++)
      if (bit == 1u << d) k = {nb[d], y[d], yl[d]};
    const int move = split_move(k);
    if (move) right |= bit;
#pragma unroll
    for (int d = 0; d < N; d++)
      if (bit == 1u << d) yl[d] = __int_as_float(__float_as_int(yl[d]) + move);
    fail ^= bit;
  }
  return right;
}

// a / b with cut_yl's yl: the split quotient with its product truncated.
__device__ __forceinline__ float cut_quot(float a, const Recip &k) {
  return __fmaf_rn(a, k.y, __fmul_rz(a, k.yl));
}
__device__ __forceinline__ float2 cut_quot2(float2 a, const Recip2 &k) {
  return __ffma2_rn(a, k.y, __fmul2_rz(a, k.yl));
}
// yl for which cut_quot is RN(a/b) for every dividend of split_quot's range;
// NaN if neither yl as made nor the next larger in magnitude is.  Out of
// line: 8% of paired warps call it, once.
static __device__ __noinline__ float cut_yl(float b) {
  const float none = __int_as_float(0x7fffffff);
  if (!(fabsf(b) >= kSplitMin)) return none;
  const Recip k = make_recip(b);
  const uint32_t bits = __float_as_uint(b), B = (bits & 0x7fffffu) | 0x800000u;
  const uint32_t twos = __ffs((int)B) - 1;
  if (twos > 2u) return k.yl;
  const float scale = __uint_as_float(bits & 0xff800000u);
  Recip n = {-__uint_as_float(0x3f800000u | (bits & 0x7fffffu)), __fmul_rn(k.y, scale),
             __fmul_rn(k.yl, scale)};
  const uint32_t Bo = B >> twos, e = 25u - twos;
  uint32_t x = (3u * Bo) ^ 2u;  // as split_base
  x *= 2u - Bo * x;
  x *= 2u - Bo * x;
  x *= 2u - Bo * x;
  const uint32_t t = (0u - x) & ((1u << e) - 1u);
  const uint32_t A1 = (uint32_t)((1ull + (uint64_t)Bo * t) >> e);  // 2^(k-25) mod B'
  const uint32_t A2 = 2u * A1 >= Bo ? 2u * A1 - Bo : 2u * A1;
  const uint32_t A3 = A1 + A2 >= Bo ? A1 + A2 - Bo : A1 + A2;
  // the members of those classes in [2^23, 2^24) (others are no dividends)
  const bool k0 = twos == 0u, k1 = twos == 1u;
  const uint32_t A[6] = {k0 ? max(A1, Bo - A1) : (k1 ? A1 + Bo : A1 + 2u * Bo),
                         k0 ? max(A3, Bo - A3) : (k1 ? 2u * Bo - A1 : A1 + 3u * Bo),
                         k0 ? Bo + A2 : (k1 ? A2 + 2u * Bo : 3u * Bo - A1),
                         k0 ? 2u * Bo - A2 : (k1 ? 3u * Bo - A2 : 4u * Bo - A1),
                         k1 ? A2 + 3u * Bo : 0u,
                         k1 ? 4u * Bo - A2 : 0u};
#pragma unroll 1
  for (int d = 0; d < 2; d++) {
    const Recip m = {n.nb, n.y, __int_as_float(__float_as_int(n.yl) + d)};
    bool right = fabsf(m.yl) <= 0x1p-25f;
#pragma unroll
    for (int i = 0; i < 6; i++) {
      const float a = __fmul_rn(__uint2float_rn(A[i]), 0x1p-23f);
      right &= (A[i] - 0x800000u >= 0x800000u) | (cut_quot(a, m) == recip_quot(a, n));
    }
    if (right) return __int_as_float(__float_as_int(k.yl) + d);
  }
  return none;
}

// The quotient of a free step.  kEither: split or cut, as `cut` says (3
// operations), where it is not worth a loop of its own.
enum QuotForm : uint32_t { kCorrected, kSplit, kCut, kEither };
template <QuotForm FORM>
__device__ __forceinline__ float free_quot(float a, const Recip &k, bool cut = false) {
  if (FORM == kEither)
    return __fmaf_rn(a, k.y, cut ? __fmul_rz(a, k.yl) : __fmul_rn(a, k.yl));
  return FORM == kCut ? cut_quot(a, k) : (FORM == kSplit ? split_quot(a, k) : recip_quot(a, k));
}
template <QuotForm FORM>
__device__ __forceinline__ float2 free_quot2(float2 a, const Recip2 &k, bool cut = false) {
  if (FORM == kEither) {
    const float2 n = __fmul2_rn(a, k.yl), z = __fmul2_rz(a, k.yl);
    return __ffma2_rn(a, k.y, make_float2(cut ? z.x : n.x, cut ? z.y : n.y));
  }
  return FORM == kCut ? cut_quot2(a, k)
                      : (FORM == kSplit ? split_quot2(a, k) : recip_quot2(a, k));
}

// True for a nonzero |a| below tiny (NaN: false).
__device__ __forceinline__ bool tiny_nonzero(float a, float tiny) {
  const float m = fabsf(a);
  return (m < tiny) & (m != 0.0f);
}

// True when RN(a/b) may be subnormal: a nonzero |a| below 2^-125 |b|
// (m * 2^125 is exact for the magnitudes compared; NaN: false).
__device__ __forceinline__ bool subnormal_quot(float a, const Recip &k) {
  const float m = fabsf(a);
  return (m != 0.0f) & (__fmul_rn(m, 0x1p125f) < fabsf(k.nb));
}
__device__ __forceinline__ bool subnormal_quot2(float2 a, const Recip2 &k) {
  const float2 m = __fmul2_rn(make_float2(fabsf(a.x), fabsf(a.y)), make_float2(0x1p125f, 0x1p125f));
  return ((a.x != 0.0f) & (m.x < fabsf(k.nb.x))) | ((a.y != 0.0f) & (m.y < fabsf(k.nb.y)));
}

// RN(a/b) for any a that subnormal_quot does not flag: the corrected
// quotient of a scaled into [lo, hi] (see above).
__device__ __forceinline__ float wide_quot(float a, const Recip &k, float lo, float hi) {
  const float m = fabsf(a);
  const float s = m > hi ? 0x1p-64f : (m < lo ? 0x1p110f : 1.0f);
  const float u = m > hi ? 0x1p64f : (m < lo ? 0x1p-110f : 1.0f);
  const float q = __fmul_rn(recip_quot(__fmul_rn(a, s), k), u);
  return (m == 0.0f || m == __int_as_float(0x7f800000)) ? __fmul_rn(a, k.y) : q;
}
__device__ __forceinline__ float2 wide_quot2(float2 a, const Recip2 &k, float lo, float hi) {
  const float mx = fabsf(a.x), my = fabsf(a.y);
  const float2 s = make_float2(mx > hi ? 0x1p-64f : (mx < lo ? 0x1p110f : 1.0f),
                               my > hi ? 0x1p-64f : (my < lo ? 0x1p110f : 1.0f));
  const float2 u = make_float2(mx > hi ? 0x1p64f : (mx < lo ? 0x1p-110f : 1.0f),
                               my > hi ? 0x1p64f : (my < lo ? 0x1p-110f : 1.0f));
  float2 q = __fmul2_rn(recip_quot2(__fmul2_rn(a, s), k), u);
  const float2 z = __fmul2_rn(a, k.y);
  const float inf = __int_as_float(0x7f800000);
  if (mx == 0.0f || mx == inf) q.x = z.x;
  if (my == 0.0f || my == inf) q.y = z.y;
  return q;
}

// RN(a/b) for any a and an eligible b: the corrected quotient inside the
// guarded range, the divide routine outside it.
__device__ __forceinline__ float quot_guarded(float a, float b, const Recip &k, float lo,
                                              float hi) {
  return outside(a, lo, hi) ? __fdiv_rn(a, b) : recip_quot(a, k);
}

}  // namespace ckt
