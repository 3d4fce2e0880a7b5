// ckt_kernels.cuh -- sm_103a kernels of the circuit hot path.
//
// Arithmetic follows the reference task bodies operation by operation
// (apps/circuit/circuit_gpu.cu:114-129, 281-283, 330-345; the CPU tasks at
// apps/circuit/circuit.cc:386-401, 430-431, 1300-1302).  Every operation of
// the EXACT paths uses an explicitly rounded intrinsic so that no multiply
// is ever contracted into an add: results are bit-identical to the
// reference's IEEE fp32 arithmetic.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "ckt.h"
#include "ckt_divide.cuh"

namespace ckt {

// ---------------------------------------------------------------------------
// calc_new_currents: one thread per wire.  The 10 segment currents and 11
// node/segment voltages of a wire live in registers across the whole inner
// time-step loop; wire fields are structure-of-arrays so a warp's loads and
// stores of any one field are one contiguous 128-byte line.
// ---------------------------------------------------------------------------
// Correctly rounded a / b.  A NaN dividend gives the quiet NaN every GPU
// arithmetic instruction returns for NaN operands (0x7fffffff, the same bits
// __fdiv_rn produces) without entering the divide routine's special-case
// path; once the recurrence has overflowed, every dividend is NaN.
__device__ __forceinline__ float div_rn(float a, float b) {
  return (a != a) ? __int_as_float(0x7fffffff) : __fdiv_rn(a, b);
}

// EXACT with the divide routine, one wire per thread:
// ((dv) - (L*(i-I0))/dt) / R and V0 + (dt*(i_k - i_k+1))/C, each operation
// rounded exactly as the reference's fp32 source.  CKT_MODE_EXACT_DIVIDE, and
// the wires of CKT_MODE_EXACT whose divisors lie outside the range of the
// corrected quotients (DualExact below).
struct DivideStep {
  float L, R, C, dt;
  __device__ __forceinline__ DivideStep(float l, float r, float c, float d) : L(l), R(r), C(c), dt(d) {}
  __device__ __forceinline__ void step(float (&ni)[10], float (&nv)[11], const float (&I0)[10],
                                       const float (&V0)[9]) const {
#pragma unroll
    for (int k = 0; k < 10; k++) {
      const float dv = __fsub_rn(nv[k + 1], nv[k]);
      const float q = div_rn(__fmul_rn(L, __fsub_rn(ni[k], I0[k])), dt);
      ni[k] = div_rn(__fsub_rn(dv, q), R);
    }
#pragma unroll
    for (int k = 0; k < 9; k++)
      nv[k + 1] = __fadd_rn(V0[k], div_rn(__fmul_rn(dt, __fsub_rn(ni[k], ni[k + 1])), C));
  }
};

// FAST: the three divisors are loop-invariant, so their quotients are
// computed once per wire (correctly rounded) and every inner-loop divide
// becomes a multiply.  The step works on j_k = i_k * R, the current before
// its 1/R scale, and carries d_k = i_k - I0_k from step to step:
//   j_k   <- (v_k+1 - v_k) + (-L/dt) * d_k
//   v_k+1 <- ((dt/C)(1/R)) * (j_k - j_k+1) + V0_k
//   d_k   <- (1/R) j_k - I0_k           (every step but the last)
//   i_k   <- (1/R) j_k                  (after the last step)
// starting from d_k = I0_k - I0_k.  3 FP32 operations per current and 2
// per voltage: 48 per wire-step, against the reference expression's 96
// counted flops.  Within 1e-5 relative of EXACT in the finite regime, with
// EXACT's NaN/Inf classes at the configured steps.
constexpr int kModeFastScalar = CKT_MODE_FAST_SCALAR;

struct FastConsts {
  float nLdt, rR, dtC, dtCrR;
  __device__ __forceinline__ FastConsts(float l, float r, float c, float d) {
    nLdt = -__fdiv_rn(l, d);
    rR = __fdiv_rn(1.0f, r);
    dtC = __fdiv_rn(d, c);
    dtCrR = __fmul_rn(dtC, rR);
  }
};

// Scalar form of the paired steppers below (bit-identical to them).
// LAST: write the currents i_k into di instead of the next d_k.
struct FastStep {
  FastConsts k;
  __device__ __forceinline__ FastStep(float l, float r, float c, float d) : k(l, r, c, d) {}
  template <bool LAST>
  __device__ __forceinline__ void step(float (&di)[10], float (&nv)[11], const float (&I0)[10],
                                       const float (&V0)[9]) const {
    float j[10];
#pragma unroll
    for (int q = 0; q < 10; q++) j[q] = __fmaf_rn(k.nLdt, di[q], __fsub_rn(nv[q + 1], nv[q]));
#pragma unroll
    for (int q = 0; q < 9; q++) nv[q + 1] = __fmaf_rn(k.dtCrR, __fsub_rn(j[q], j[q + 1]), V0[q]);
#pragma unroll
    for (int q = 0; q < 10; q++) di[q] = LAST ? __fmul_rn(k.rR, j[q]) : __fmaf_rn(k.rR, j[q], -I0[q]);
  }
};

// FAST, packed: the same operations, two at a time with Blackwell's paired
// FP32 instructions (add/mul/fma .f32x2).  Segment k is paired with k+5:
// currents (d_p, d_p+5) for p < 5 and voltages (v_q, v_q+5) for q <= 5, so
// every current operation and all voltages but v5 are one paired
// instruction for two segments.  A difference a - b is fma(b, -1, a):
// exact product, one rounding -- the same bits as the subtraction.  Each
// component is rounded exactly as in the scalar step: bit-identical to it.
struct PackedFast {
  float2 nLdt, rR, dtCrR, neg1;
  float dtCrR1;
  __device__ __forceinline__ PackedFast(float l, float r, float c, float d) {
    const FastConsts k(l, r, c, d);
    nLdt = make_float2(k.nLdt, k.nLdt);
    rR = make_float2(k.rR, k.rR);
    dtCrR = make_float2(k.dtCrR, k.dtCrR);
    neg1 = make_float2(-1.0f, -1.0f);
    dtCrR1 = k.dtCrR;
  }
  // dp[p] = (d_p, d_p+5); nI0[p] = (-I0_p, -I0_p+5); vp[q] = (v_q, v_q+5);
  // V0p[j] = (V0_j, V0_j+5) for j < 4; V04 = V0_4.
  template <bool LAST>
  __device__ __forceinline__ void step(float2 (&dp)[5], float2 (&vp)[6], const float2 (&nI0)[5],
                                       const float2 (&V0p)[4], float V04) const {
    float2 jp[5];
#pragma unroll
    for (int p = 0; p < 5; p++) jp[p] = __ffma2_rn(nLdt, dp[p], __ffma2_rn(vp[p], neg1, vp[p + 1]));
#pragma unroll
    for (int q = 1; q < 5; q++)
      vp[q] = __ffma2_rn(dtCrR, __ffma2_rn(jp[q], neg1, jp[q - 1]), V0p[q - 1]);
    const float v5 = __fmaf_rn(dtCrR1, __fmaf_rn(jp[0].y, -1.0f, jp[4].x), V04);
    vp[0].y = v5;
    vp[5].x = v5;
#pragma unroll
    for (int p = 0; p < 5; p++) dp[p] = LAST ? __fmul2_rn(rR, jp[p]) : __ffma2_rn(rR, jp[p], nI0[p]);
  }
};

// FAST, two wires per thread: wire a's segment k and wire b's segment k
// share every paired instruction, so all 48 operations of a wire-step pair
// up with no cross-lane moves (24 instructions per wire-step).  Each lane is
// rounded exactly as the scalar step: bit-identical to it.
struct DualFast {
  float2 nLdt, rR, dtCrR, neg1;
  __device__ __forceinline__ DualFast(float2 l, float2 r, float2 c, float d) {
    const FastConsts ka(l.x, r.x, c.x, d), kb(l.y, r.y, c.y, d);
    nLdt = make_float2(ka.nLdt, kb.nLdt);
    rR = make_float2(ka.rR, kb.rR);
    dtCrR = make_float2(ka.dtCrR, kb.dtCrR);
    neg1 = make_float2(-1.0f, -1.0f);
  }
  // d[k] = (d_k of a, d_k of b), nv[k] likewise; nI0 = -I0; V0 = wire voltages.
  template <bool LAST>
  __device__ __forceinline__ void step(float2 (&d)[10], float2 (&nv)[11], const float2 (&nI0)[10],
                                       const float2 (&V0)[9]) const {
    float2 j[10];
#pragma unroll
    for (int k = 0; k < 10; k++) j[k] = __ffma2_rn(nLdt, d[k], __ffma2_rn(nv[k], neg1, nv[k + 1]));
#pragma unroll
    for (int k = 0; k < 9; k++)
      nv[k + 1] = __ffma2_rn(dtCrR, __ffma2_rn(j[k + 1], neg1, j[k]), V0[k]);
#pragma unroll
    for (int k = 0; k < 10; k++) d[k] = LAST ? __fmul2_rn(rR, j[k]) : __ffma2_rn(rR, j[k], nI0[k]);
  }
};

// min(m, |a|, |b|); a NaN argument is ignored.
__device__ __forceinline__ float min_abs(float m, float a, float b) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(m), "f"(fabsf(a)), "f"(fabsf(b)));
  return r;
}
// a - b in both lanes, as the addition of -b: two register pairs read instead
// of the three of fma(b, -1, a) (all-NaN loop, 1,048,576 wires x 1000 steps:
// 3.49 -> 3.45 ms).
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
  return __fadd2_rn(a, make_float2(-b.x, -b.y));
}
// i, v: the least |I0| and |V0| of a wire (NaN ones apart; NaN when all are:
// what is added to them is NaN whatever it was).  See exact_steps.
__device__ __forceinline__ bool sound_wire(float i, float v, float L, float C, float dt) {
  return !(i < 0x1p-50f) & !(v < 0x1p-50f) & (fabsf(L) >= 0x1p-43f) & (fabsf(C) >= 0x1p-20f) &
         !(__fmul_rn(v, fabsf(C)) < __fmul_rn(0x1p-22f, dt));
}
// Orders magnitudes as integers, with zero above everything: finite values
// by magnitude, then infinity (kOrderInf), NaN, zero.
__device__ __forceinline__ uint32_t order(float a) { return 2u * __float_as_uint(a) - 1u; }
constexpr uint32_t kOrderInf = 0xfeffffffu;
// The same loop constants for the wide steps; i: the least order(I0).
__device__ __forceinline__ bool wide_wire(uint32_t i, float L, float C) {
  return (i >= order(0x1p-50f)) & (fabsf(L) >= 0x1p-43f) & (fabsf(C) >= 0x1p-20f);
}
// Which wires' values are NaN: bit 0 the first (or only) wire, bit 1 the second.
__device__ __forceinline__ uint32_t nan_bits(float a) { return a != a ? 1u : 0u; }
__device__ __forceinline__ uint32_t nan_bits(float2 a) {
  return (a.x != a.x ? 1u : 0u) | (a.y != a.y ? 2u : 0u);
}

__device__ __forceinline__ bool huge(float a) { return fabsf(a) > 0x1p60f; }
__device__ __forceinline__ bool huge(float2 a) { return huge(a.x) | huge(a.y); }
__device__ __forceinline__ bool tame(float a) { return fabsf(a) <= 0x1p60f; }  // NaN: false
__device__ __forceinline__ bool tame(float2 a) { return tame(a.x) & tame(a.y); }

// EXACT, two wires per thread: the reference's operations in the reference's
// order, each rounded as IEEE fp32 rounds it, with the 29 divisions of a
// wire-step done as correctly rounded quotients by precomputed reciprocals
// (ckt_divide.cuh) instead of the divide routine.  Wire a's and wire b's
// operation k share one paired instruction.  A step runs in two phases:
//   currents:  a1_k = L (i_k - I0_k),  a2_k = (v_k+1 - v_k) - a1_k / dt,
//              i_k <- a2_k / R
//   voltages:  a3_k = dt (i_k - i_k+1), v_k+1 <- V0_k + a3_k / C
// Each phase first forms all of its dividends, then takes the corrected
// quotients when every dividend of the thread's two wires lies in the
// guarded range, and wide_quot otherwise (zero dividends, as in a loop's
// first step, large ones and infinities while the recurrence overflows),
// the divide routine only for dividends too tiny for wide_quot.  Every
// branch rounds every quotient to the same float, so the bits never depend
// on which one ran.  DTF: dt is (float)1e-6 and its quotients use the
// split reciprocal (2 operations); otherwise they are corrected quotients too.
template <bool DTF>
struct DualExact {
  float2 L, dt2, neg1;
  Recip2 kR, kC, kdt;
  float dt;
  __device__ __forceinline__ DualExact(float2 l, float2 r, float2 c, float d) {
    L = l;
    dt = d;
    dt2 = make_float2(d, d);
    neg1 = make_float2(-1.0f, -1.0f);
    kR = make_recip2(r.x, r.y);
    kC = make_recip2(c.x, c.y);
    if (!DTF) kdt = make_recip2(d, d);
  }
  // Both wires' divisors lie in the range the corrected quotients need.
  static __device__ __forceinline__ bool eligible(float2 r, float2 c, float d) {
    return divisor_ok(r.x, kRMin, kRMax) && divisor_ok(r.y, kRMin, kRMax) &&
           divisor_ok(c.x, kCMin, kCMax) && divisor_ok(c.y, kCMin, kCMax) &&
           (DTF || divisor_ok(d, kCMin, kCMax));
  }
  __device__ __forceinline__ float2 dt_div(float2 a) const {
    if (DTF) return dt_quot2(a);
    return recip_quot2(a, kdt);
  }
  // With DTF no dividend of dt needs a guard of its own: the split quotient
  // is exact unless |a1| < 2^-118, and then |a1/dt| < 2^-98, far below half
  // an ulp of any dv with |dv - a1/dt| >= 2^-50 (the guard on a2), so
  // a2 = RN(dv - a1/dt) = dv either way; when a2's guard fails, the divide
  // routine recomputes the quotient from a1.
  __device__ __forceinline__ bool dt_outside(float a) const {
    if (DTF) return false;
    return outside(a, kCLo, kCHi);
  }
  // ni: currents i_k; nv: voltages v_0..v_10 (v_0, v_10 the node voltages);
  // nI0 = -I0; V0 = the wire's voltages at the start of the loop.
  __device__ __forceinline__ void step(float2 (&ni)[10], float2 (&nv)[11],
                                       const float2 (&nI0)[10], const float2 (&V0)[9]) const {
    float2 a1[10], a2[10];
    bool bad = false;
#pragma unroll
    for (int k = 0; k < 10; k++) {
      a1[k] = __fmul2_rn(L, __fadd2_rn(ni[k], nI0[k]));
      const float2 dv = __ffma2_rn(nv[k], neg1, nv[k + 1]);
      a2[k] = __ffma2_rn(dt_div(a1[k]), neg1, dv);
      bad |= dt_outside(a1[k].x) | dt_outside(a1[k].y) | outside(a2[k].x, kRLo, kRHi) |
             outside(a2[k].y, kRLo, kRHi);
    }
    // A phase that leaves the corrected quotient (zeros, huge values and
    // infinities as a loop's state starts or blows up) takes wide_quot, and
    // the divide routine only for the rare dividends wide_quot does not
    // cover: with DTF a dt dividend below kDtTiny (whose split quotient may
    // be off), an R or C dividend whose quotient may be subnormal; without
    // DTF, phase 1 always.
    bool wide = false;  // phase 1 left the corrected quotient
    if (!bad) {
#pragma unroll
      for (int k = 0; k < 10; k++) ni[k] = recip_quot2(a2[k], kR);
    } else {
      bool rare = !DTF;
      if (DTF) {
#pragma unroll
        for (int k = 0; k < 10; k++)
          rare |= tiny_nonzero(a1[k].x, kDtTiny) | tiny_nonzero(a1[k].y, kDtTiny) |
                  subnormal_quot2(a2[k], kR);
      }
      if (!rare) {
#pragma unroll
        for (int k = 0; k < 10; k++) ni[k] = wide_quot2(a2[k], kR, kRLo, kRHi);
      } else {
        const float2 R = make_float2(-kR.nb.x, -kR.nb.y);
#pragma unroll
        for (int k = 0; k < 10; k++) {
          const float dx = __fsub_rn(nv[k + 1].x, nv[k].x), dy = __fsub_rn(nv[k + 1].y, nv[k].y);
          ni[k] = make_float2(__fdiv_rn(__fsub_rn(dx, __fdiv_rn(a1[k].x, dt)), R.x),
                              __fdiv_rn(__fsub_rn(dy, __fdiv_rn(a1[k].y, dt)), R.y));
        }
      }
      wide = true;
    }
    // With DTF, currents from corrected quotients are at most 2^100 / 2^-8
    // in magnitude, so |a3| <= dt 2^109 < 2^90: only the lower bound needs a
    // check.  Currents from a phase 1 that left them may be anything.
    float2 a3[9];
    bad = false;
#pragma unroll
    for (int k = 0; k < 9; k++) {
      a3[k] = __fmul2_rn(dt2, __ffma2_rn(ni[k + 1], neg1, ni[k]));
      bad |= (fabsf(a3[k].x) < kCLo) | (fabsf(a3[k].y) < kCLo);
    }
    if (!DTF || wide) {
#pragma unroll
      for (int k = 0; k < 9; k++) bad |= (fabsf(a3[k].x) > kCHi) | (fabsf(a3[k].y) > kCHi);
    }
    if (!bad) {
#pragma unroll
      for (int k = 0; k < 9; k++) nv[k + 1] = __fadd2_rn(V0[k], recip_quot2(a3[k], kC));
    } else {
      bool rare = false;
#pragma unroll
      for (int k = 0; k < 9; k++)
        rare |= subnormal_quot2(a3[k], kC);
      if (!rare) {
#pragma unroll
        for (int k = 0; k < 9; k++) nv[k + 1] = __fadd2_rn(V0[k], wide_quot2(a3[k], kC, kCLo, kCHi));
      } else {
        const float2 C = make_float2(-kC.nb.x, -kC.nb.y);
#pragma unroll
        for (int k = 0; k < 9; k++)
          nv[k + 1] = make_float2(__fadd_rn(V0[k].x, __fdiv_rn(a3[k].x, C.x)),
                                  __fadd_rn(V0[k].y, __fdiv_rn(a3[k].y, C.y)));
      }
    }
  }
  // Which divisors take the split quotient in both wires (check_split):
  // bit 0 R, bit 1 C.
  __device__ __forceinline__ uint32_t check() {
    const float nb[4] = {kR.nb.x, kR.nb.y, kC.nb.x, kC.nb.y};
    const float y[4] = {kR.y.x, kR.y.y, kC.y.x, kC.y.y};
    float yl[4] = {kR.yl.x, kR.yl.y, kC.yl.x, kC.yl.y};
    const uint32_t right = check_split(nb, y, yl);
    kR.yl = make_float2(yl[0], yl[1]);
    kC.yl = make_float2(yl[2], yl[3]);
    return ((right & 3u) == 3u ? 1u : 0u) | (right >= 12u ? 2u : 0u);
  }
  static __device__ __forceinline__ float2 cut(const Recip2 &k) {
    return make_float2(cut_yl(-k.nb.x), cut_yl(-k.nb.y));
  }
  // step() without guards and branches.  FR, FC: the form of the quotients by
  // R and C: split, with a rounded or a truncated product (2 operations), or
  // corrected (4).
  // LOW: low collects the least |dividend| of
  // R and C (NaN ones apart).  exact_steps says when the result is step()'s.
  template <QuotForm FR, QuotForm FC, bool LOW>
  __device__ __forceinline__ void step_free(float2 (&ni)[10], float2 (&nv)[11],
                                            const float2 (&nI0)[10], const float2 (&V0)[9],
                                            float &low) const {
#pragma unroll
    for (int k = 0; k < 10; k++) {
      const float2 a1 = __fmul2_rn(L, __fadd2_rn(ni[k], nI0[k]));
      const float2 a2 = sub2(sub2(nv[k + 1], nv[k]), dt_div(a1));
      if (LOW) low = min_abs(low, a2.x, a2.y);
      ni[k] = free_quot2<FR>(a2, kR);
    }
#pragma unroll
    for (int k = 0; k < 9; k++) {
      const float2 a3 = __fmul2_rn(dt2, sub2(ni[k], ni[k + 1]));
      if (LOW) low = min_abs(low, a3.x, a3.y);
      nv[k + 1] = __fadd2_rn(V0[k], free_quot2<FC>(a3, kC));
    }
  }
  // The same with every zero and infinite dividend's quotient as well: a * y.
  // lowR, lowC collect the least order of the nonzero dividends.
  template <QuotForm FORM>
  static __device__ __forceinline__ float2 wide(float2 a, const Recip2 &k, bool cut,
                                                uint32_t &low) {
    const uint32_t tx = order(a.x), ty = order(a.y);
    const float2 q = free_quot2<FORM>(a, k, cut), z = __fmul2_rn(a, k.y);
    low = min(low, min(tx, ty));
    return make_float2(tx >= kOrderInf ? z.x : q.x, ty >= kOrderInf ? z.y : q.y);
  }
  template <QuotForm FORM>
  __device__ __forceinline__ void step_wide(float2 (&ni)[10], float2 (&nv)[11],
                                            const float2 (&nI0)[10], const float2 (&V0)[9],
                                            bool cutR, bool cutC, uint32_t &lowR,
                                            uint32_t &lowC) const {
#pragma unroll
    for (int k = 0; k < 10; k++) {
      const float2 a1 = __fmul2_rn(L, __fadd2_rn(ni[k], nI0[k]));
      ni[k] = wide<FORM>(sub2(sub2(nv[k + 1], nv[k]), dt_div(a1)), kR, cutR, lowR);
    }
#pragma unroll
    for (int k = 0; k < 9; k++)
      nv[k + 1] = __fadd2_rn(
          V0[k], wide<FORM>(__fmul2_rn(dt2, sub2(ni[k], ni[k + 1])), kC, cutC, lowC));
  }
  __device__ __forceinline__ bool can_wide(const float2 (&nI0)[10]) const {
    uint32_t x = ~0u, y = ~0u;
#pragma unroll
    for (int k = 0; k < 10; k++) {
      x = min(x, order(nI0[k].x));
      y = min(y, order(nI0[k].y));
    }
    return wide_wire(x, L.x, kC.nb.x) & wide_wire(y, L.y, kC.nb.y);
  }
  static __device__ __forceinline__ uint32_t least_order(const float2 (&ni)[10]) {
    uint32_t m = ~0u;
#pragma unroll
    for (int k = 0; k < 10; k++) m = min(m, min(order(ni[k].x), order(ni[k].y)));
    return m;
  }
  __device__ __forceinline__ float most_C() const { return fmaxf(fabsf(kC.nb.x), fabsf(kC.nb.y)); }
  // Dividends like those these currents come of and lead to keep LOW's bound,
  // and nothing is about to overflow (NaN apart).
  static __device__ __forceinline__ bool calm(const float2 (&ni)[10]) {
    float most = 0.0f, drop = __int_as_float(0x7f800000);
#pragma unroll
    for (int k = 0; k < 10; k++) most = fmaxf(most, fmaxf(fabsf(ni[k].x), fabsf(ni[k].y)));
#pragma unroll
    for (int k = 0; k < 9; k++) {
      const float2 d = sub2(ni[k], ni[k + 1]);
      drop = min_abs(drop, d.x, d.y);
    }
    return (least_current(ni) >= 0x1p-48f) & (drop >= 0x1p-20f) & (most <= 0x1p40f);
  }
  static __device__ __forceinline__ bool starts_zero(const float2 (&ni)[10]) {
    return ((ni[4].x == 0.0f) & (ni[5].x == 0.0f)) | ((ni[4].y == 0.0f) & (ni[5].y == 0.0f));
  }
  // The loop's constants keep every dividend's tininess from mattering
  // (exact_steps).
  __device__ __forceinline__ bool sound(const float2 (&nI0)[10], const float2 (&V0)[9]) const {
    float ix = fabsf(nI0[0].x), iy = fabsf(nI0[0].y), vx = fabsf(V0[0].x), vy = fabsf(V0[0].y);
#pragma unroll
    for (int k = 1; k < 10; k++) {
      ix = fminf(ix, fabsf(nI0[k].x));
      iy = fminf(iy, fabsf(nI0[k].y));
    }
#pragma unroll
    for (int k = 1; k < 9; k++) {
      vx = fminf(vx, fabsf(V0[k].x));
      vy = fminf(vy, fabsf(V0[k].y));
    }
    return sound_wire(ix, vx, L.x, kC.nb.x, dt) & sound_wire(iy, vy, L.y, kC.nb.y, dt);
  }
  // step() for a state whose 10 currents and 9 wire voltages are all NaN,
  // in both wires.  Such a state stays NaN -- every new current and voltage
  // depends on a NaN of the previous step -- so every dividend is NaN and any
  // form of quotient gives step()'s NaN: the split quotients, no compares.
  __device__ __forceinline__ void step_all_nan(float2 (&ni)[10], float2 (&nv)[11],
                                               const float2 (&nI0)[10],
                                               const float2 (&V0)[9]) const {
#pragma unroll
    for (int k = 0; k < 10; k++) {
      const float2 a1 = __fmul2_rn(L, __fadd2_rn(ni[k], nI0[k]));
      ni[k] = split_quot2(sub2(sub2(nv[k + 1], nv[k]), dt_div(a1)), kR);
    }
#pragma unroll
    for (int k = 0; k < 9; k++)
      nv[k + 1] = __fadd2_rn(
          V0[k], split_quot2(__fmul2_rn(dt2, sub2(ni[k], ni[k + 1])), kC));
  }
  static constexpr uint32_t kWires = 3u;  // nan_bits of both wires
  static constexpr bool kFrontHere = true;  // exact_steps' first guarded steps not by a call
  // NaN where any of a wire's currents or voltages is NaN (or infinities
  // cancel).
  static __device__ __forceinline__ float2 state_sum(const float2 (&ni)[10],
                                                     const float2 (&nv)[11]) {
    float2 s = ni[9], t = nv[9];
#pragma unroll
    for (int k = 0; k < 9; k++) s = __fadd2_rn(s, ni[k]);
#pragma unroll
    for (int k = 1; k < 9; k++) t = __fadd2_rn(t, nv[k]);
    return __fadd2_rn(s, t);
  }
  static __device__ __forceinline__ float least_current(const float2 (&ni)[10]) {
    float m = __int_as_float(0x7f800000);
#pragma unroll
    for (int k = 0; k < 10; k++) m = min_abs(m, ni[k].x, ni[k].y);
    return m;
  }
  // The wires whose 10 currents and 9 wire voltages are all NaN.
  static __device__ __forceinline__ uint32_t all_nan(const float2 (&ni)[10],
                                                     const float2 (&nv)[11]) {
    uint32_t nan = nan_bits(ni[0]);
    if (nan) {
#pragma unroll
      for (int k = 1; k < 10; k++) nan &= nan_bits(ni[k]) & nan_bits(nv[k]);
    }
    return nan;
  }
};

// The inner loop of DualExact and SoloExact.  The steps run in blocks; at a
// block's start, once the states of all the warp's wires have become all NaN
// (as the reference's recurrence does within ~10-30 steps at the benchmark's
// inductances, and stays), the remaining steps run with step_all_nan -- every
// operation of every step still computed, the same bits.
//
// A block runs without guards (step_free) and is checked as a whole at its
// end; if the check fails in any lane the warp returns to the state saved in
// shared memory and runs the block with step().  What could be wrong in a
// free block, and why its check finds it:
//  * Huge and infinite dividends.  A finite dividend gives the correctly
//    rounded quotient or (the corrected quotient's q0 overflowing) NaN; an
//    infinite one gives its infinity or NaN.  A NaN in place of a number does
//    not get lost: a NaN current makes its own next value NaN, a NaN voltage
//    the currents beside it.  So a wire's state that holds no NaN at the end
//    was right throughout; one that was all NaN at the start stays so.
//  * Tiny dividends and zeros.  Both quotients are right for |a| >= 2^-77 |b|
//    (split: a yl, rounded or truncated, is normal, |yl| >= 2^-48 / |b|;
//    corrected: the remainder is representable, |b| >= 2^-20).  Below that the true quotient and the
//    computed one are both at most 2^-76 -- the wrong bits, or a zero of the
//    wrong sign, of something that small.  A block of LOW steps fails when it
//    met a dividend below kSplitLo (corrected: kCLo).  Steps without LOW need
//    sound constants (sound_wire), with which such a quotient never matters:
//      - by C: V0 + q = V0 when |V0| >= 2^-50;
//      - by R, in the wire's next step: i - I0 = -I0 when |I0| >= 2^-50;
//      - by R, in the same step's i_k - i_k+1: if the neighbour is at least
//        2^-50 the difference is the neighbour either way; otherwise the
//        difference is at most 2^-49 and, divided by C, at most
//        2^-48 dt/|C|, which V0 absorbs when |V0| >= 2^-22 dt/|C|;
//      - by R, as the loop's result: the last block fails when a current's
//        magnitude is below 2^-75;
//      - a1 / dt is right: i - I0 is 0 or at least half an ulp of I0, 2^-75,
//        so with |L| >= 2^-43 a1 is 0 or at least 2^-118 = kDtTiny.
//    (With LOW a1 needs no check either, see dt_outside.)
// Where the constants are not sound, or a block failed, the next blocks are
// careful ones, of the form whose bounds the currents at hand let expect:
//  * LOW ones, when those currents are calm (of ordinary size and distance);
//    not after a free block's failure, which they would share.
//  * Wide steps otherwise, which also divide zeros and infinities rightly (a
//    times RN(1/b)) and collect the least nonzero dividends -- by C, at least
//    2^-77 |C| wanted, by R, 2^-66, so that a nonzero current is at least
//    2^-74 and, I0 being 0 or at least 2^-50 (wide_wire) and so the currents
//    at the block's start, a1 is 0 or at least kDtTiny.  They take split or
//    truncated products (kEither); with corrected quotients, whose overflow
//    shows as NaN, a block must not end with a new NaN.
//  * Guarded steps, where neither may be expected or the block failed: the next
//    32, 64 and 128 in one call, then all the rest of the loop, as in launches
//    of few steps.  (A warp with sound constants goes on trying.)
// After a failure sound blocks pause for 16, 32, 64 and 128 steps; before an
// overflow (a state whose sum is past 2^60) for one careful block, as from
// nodes that are.  A failed block costs its own steps once more, so the first
// blocks are short.  A careful block is a call that loads the wires' constants
// anew and divides for their reciprocals, about as long as 5 steps, so those
// that come out right grow to 64 steps.
//
// Why: the guards' 58 compares and two branches per paired step held the loop
// at 75% of the FP32 pipe, and the corrected quotients are 76 of its 163
// operations.  A free step has 125 operations and nothing else.  The 19
// three-input minima of LOW are not free beside it: FMAs of three register
// pairs keep the register ports busy.  1,048,576 wires, 1000 steps, GB300:
// guarded 5.88 ms, free with LOW 4.64 ms, without 3.75 ms, all NaN 3.49 ms
// (4.80 ms with corrected quotients); the 125 operations at the pipe's full
// rate take 3.25 ms.  From the generated state (zeros, overflow, all NaN
// after 26 steps) 5.13 ms guarded, 3.96 ms with its first 32 steps guarded,
// 3.64 ms with 10 guarded and 16 wide ones.  The careful forms, 1,048,576 /
// 32,768 / 4096 wires, ms per 1000 steps, guarded one or two wires per thread /
// with short careful blocks, wide first, all tried again / as here: zeros in 2%
// of the wires' starting values 5.87 0.27 0.17 / 7.11 0.35 0.13 / 4.55 0.23
// 0.10; loops from zeros with ordinary nodes, most segments staying below
// 2^-66, 18.96 0.80 0.51 / 21.94 0.91 0.75 / 18.69 0.81 0.45; everything zero
// 17.29 0.75 0.48 / 10.82 0.83 0.99 / 7.11 0.29 0.11; no inductance 5.61 0.27
// 0.35 / 7.33 0.26 0.36 / 4.78 0.30 0.33.  Slower than guarded throughout:
// 32 steps with such a start (5 to 25%; half a launch's warps with NaN nodes
// 50%), and loops whose quotients are nearly all subnormal (119 / 125 / 145
// ms), in which the divide routine is all that counts.
constexpr int kGuardedRun = 16;  // steps between looks for all NaN (guarded loop)
constexpr int kCarefulRun = 16;  // steps of the first careful block
// From zero currents or voltages the first steps run guarded: what the node
// voltages start reaches one segment further per step, falling to 2^-110 on
// its way, below what the other forms divide rightly.
constexpr int kFrontRun = 10;
// From states with single zeros or tiny values 2 guarded steps: then the
// dividends mostly are neither.
constexpr int kCalmRun = 2;
constexpr int kFirstRun = 8, kMostRun = 64;  // steps of a free or careful block
constexpr int kMostPause = 128;  // steps before what failed is tried again
// Values per thread in shared memory: the state at a block's start (10
// currents, 9 voltages), the two node voltages and yl of R and C.
constexpr int kSavedState = 23;
// Launches of fewer steps run guarded throughout: checking the divisors costs
// about as much as 5 steps, the blocks that fail from the generated state
// (zeros, overflow) 20.  1,000,000 wires: 16 steps 104 us guarded, 102 us free
// from finite values, 107 and 208 us from the generated state; 32 steps 192
// and 153, 164 and 143 us.
constexpr int kFreeSteps = 32;
// The quotient forms of a warp's free steps.  8% of paired warps hold a divisor
// that check_split leaves unchecked; with corrected quotients by R (C) such a
// warp's steps are 16% (14%) longer, and a small launch takes as long as its
// slowest warp.  So those warps try truncated products, which all but 7% (solo;
// paired 14%) of them can take; the trial costs them about 3 steps.  us per
// 1000 steps, GB300, before / with it / with no divisor unchecked: 1024 wires
// 61 / 57 / 55, 4096 68 / 64 / 63, 16,000 104 / 97..118 / 90 (a corrected warp
// left or not), 124,867 521 / 508 / 494, 262,144 1021 / 991 / 935, 4,194,304
// 14439 / 14127 / 14010.
// Corrected quotients remain for C alone (divisors below kSplitMin) or for both.
__device__ __forceinline__ void normalize_forms(QuotForm &FR, QuotForm &FC) {
  const bool mixed = (FR == kCorrected) != (FC == kCorrected);
  if (FR == kCorrected || (mixed && FR == kCut)) FR = FC = kCorrected;
}
template <int STRIDE, typename F>
__device__ __forceinline__ void save_state(F *save, const F (&ni)[10], const F (&nv)[11]) {
#pragma unroll
  for (int k = 0; k < 10; k++) save[k * STRIDE] = ni[k];
#pragma unroll
  for (int k = 0; k < 9; k++) save[(10 + k) * STRIDE] = nv[k + 1];
}
template <int STRIDE, typename F>
__device__ __forceinline__ void load_state(const F *save, F (&ni)[10], F (&nv)[11]) {
#pragma unroll
  for (int k = 0; k < 10; k++) ni[k] = save[k * STRIDE];
#pragma unroll
  for (int k = 0; k < 9; k++) nv[k + 1] = save[(10 + k) * STRIDE];
}

// The loop with guarded steps only: few steps, a general dt, or states that the
// other forms do not take.
template <typename Stepper, typename F>
__device__ __forceinline__ void exact_steps_guarded(const Stepper &pk, int steps, F (&ni)[10],
                                                    F (&nv)[11], const F (&nI0)[10],
                                                    const F (&V0)[9]) {
  const uint32_t lanes = __activemask();
  int j = 0;
#pragma unroll 1
  while (j < steps) {
    if (__all_sync(lanes, Stepper::all_nan(ni, nv) == Stepper::kWires)) break;
    const int n = min(kGuardedRun, steps - j);
#pragma unroll 1
    for (int i = 0; i < n; i++) pk.step(ni, nv, nI0, V0);
    j += n;
  }
#pragma unroll 1
  for (; j < steps; j++) pk.step_all_nan(ni, nv, nI0, V0);
}

// The wires' constants and the state in `save`, as the steps take them.
template <typename Stepper, int STRIDE, typename Wires, typename F>
__device__ __forceinline__ Stepper resume(const Wires &wires, const F *save, F (&ni)[10],
                                          F (&nv)[11], F (&nI0)[10], F (&V0)[9]) {
  Stepper pk = wires.template stepper<Stepper>();
  pk.kR.yl = save[21 * STRIDE];
  pk.kC.yl = save[22 * STRIDE];
  wires.load(nI0, V0);
  nv[0] = save[19 * STRIDE];
  nv[10] = save[20 * STRIDE];
  load_state<STRIDE>(save, ni, nv);
  return pk;
}
// ni, nv: the state before the first step, and after the last.  wires: the
// thread's wires in global memory (SoloWire, DualWires), unchanged until the
// loop is done: their constants are loaded again for each stretch of blocks
// rather than kept over a guarded one.
template <int STRIDE, typename Stepper, typename Wires, typename F>
__device__ __forceinline__ void exact_steps(const Wires &wires, int steps, F (&ni)[10],
                                            F (&nv)[11], F *save) {
  const uint32_t lanes = __activemask();
  QuotForm FR, FC;  // of the warp
  bool sound, wide;
  // pause: steps before the next try of free blocks; guard: steps to run
  // guarded before the next try of the careful forms
  int j = 0, run = kFirstRun, pause = 0, penalty = kCarefulRun;
  int guard = 0, again = 2 * kCarefulRun, careful = kCarefulRun;
  if (!Stepper::kFrontHere) save_state<STRIDE>(save, ni, nv);
  save[19 * STRIDE] = nv[0];
  save[20 * STRIDE] = nv[10];
  {
    Stepper pk = wires.template stepper<Stepper>();
    const uint32_t checked = pk.check();
    FR = __all_sync(lanes, checked & 1u) ? kSplit : kCorrected;
    FC = __all_sync(lanes, checked & 2u) ? kSplit : kCorrected;
    if (FR == kCorrected) {
      const F yl = Stepper::cut(pk.kR);
      if (__all_sync(lanes, !nan_bits(yl))) {
        FR = kCut;
        pk.kR.yl = yl;
      }
    }
    if (FC == kCorrected) {
      const F yl = Stepper::cut(pk.kC);
      if (__all_sync(lanes, !nan_bits(yl))) {
        FC = kCut;
        pk.kC.yl = yl;
      }
    }
    normalize_forms(FR, FC);
    F nI0[10], V0[9];
    wires.load(nI0, V0);
    sound = __all_sync(lanes, pk.sound(nI0, V0));
    wide = __all_sync(lanes, pk.can_wide(nI0));
    // NaN or overflow from a node reaches the far end within 10 steps
    if (__any_sync(lanes, !(tame(nv[0]) & tame(nv[10])))) pause = kCarefulRun;
    int front = 0;
    if (__any_sync(lanes, Stepper::starts_zero(ni))) front = kFrontRun;
    else if (!sound && !__all_sync(lanes, Stepper::calm(ni))) front = kCalmRun;
    if (Stepper::kFrontHere) {
#pragma unroll 1
      for (; j < front; j++) pk.step(ni, nv, nI0, V0);
      save_state<STRIDE>(save, ni, nv);
    } else {
      guard = front;
    }
    save[21 * STRIDE] = pk.kR.yl;
    save[22 * STRIDE] = pk.kC.yl;
  }
#pragma unroll 1
  while (j < steps) {
    load_state<STRIDE>(save, ni, nv);
    uint32_t nan = Stepper::all_nan(ni, nv);
    // the switch only when every thread of the warp can take it, so that a
    // warp never runs the two loops one after the other
    if (__all_sync(lanes, nan == Stepper::kWires)) break;
    if (sound && pause <= 0) {
      Stepper pk = wires.template stepper<Stepper>();
      pk.kR.yl = save[21 * STRIDE];
      pk.kC.yl = save[22 * STRIDE];
      F nI0[10], V0[9];
      wires.load(nI0, V0);
      nv[0] = save[19 * STRIDE];
      nv[10] = save[20 * STRIDE];
      bool right = true, leave = false;
      float none = 0.0f;
#pragma unroll 1
      while (!leave && j < steps) {
        const int n = min(run, steps - j);
        // A loop per pair of quotient forms: a warp with one unchecked divisor
        // keeps the other's split quotients.  The usual pair last (as a chain
        // of ifs or with it first the loops' code differs by 1 to 4% either way).
        switch (FR * 3 + FC) {
          case kCut * 3 + kSplit:
#pragma unroll 1
            for (int i = 0; i < n; i++)
              pk.template step_free<kCut, kSplit, false>(ni, nv, nI0, V0, none);
            break;
          case kSplit * 3 + kCut:
#pragma unroll 1
            for (int i = 0; i < n; i++)
              pk.template step_free<kSplit, kCut, false>(ni, nv, nI0, V0, none);
            break;
          case kCut * 3 + kCut:
#pragma unroll 1
            for (int i = 0; i < n; i++)
              pk.template step_free<kCut, kCut, false>(ni, nv, nI0, V0, none);
            break;
          case kSplit * 3 + kCorrected:
#pragma unroll 1
            for (int i = 0; i < n; i++)
              pk.template step_free<kSplit, kCorrected, false>(ni, nv, nI0, V0, none);
            break;
          case kCorrected * 3 + kCorrected:
#pragma unroll 1
            for (int i = 0; i < n; i++)
              pk.template step_free<kCorrected, kCorrected, false>(ni, nv, nI0, V0, none);
            break;
          default:
#pragma unroll 1
            for (int i = 0; i < n; i++)
              pk.template step_free<kSplit, kSplit, false>(ni, nv, nI0, V0, none);
            break;
        }
        const F sum = Stepper::state_sum(ni, nv);
        const bool done =
            j + n < steps || Stepper::least_current(ni) >= 0x1p-75f;  // as a result
        if (!__all_sync(lanes, tame(sum) & done)) {
          right = __all_sync(lanes, (nan_bits(sum) & ~nan) == 0u && done);
          if (!right) break;
          nan = Stepper::all_nan(ni, nv);
          leave = __all_sync(lanes, nan == Stepper::kWires);
          // about to overflow: wide steps, which also get that right
          if (__any_sync(lanes, huge(sum))) {
            leave = true;
            pause = kCarefulRun;
          }
        }
        j += n;
        if (run == kMostRun) penalty = kCarefulRun;
        run = min(2 * run, kMostRun);
        save_state<STRIDE>(save, ni, nv);
      }
      if (!right) {
        pause = penalty;
        penalty = min(2 * penalty, kMostPause);
        run = kFirstRun;
      }
      continue;
    }
    // the form whose bounds the state is likely to keep
    const bool calm = !sound && __all_sync(lanes, Stepper::calm(ni));
    const bool can =
        calm || (wide && __all_sync(lanes, Stepper::least_order(ni) >= order(0x1p-74f)));
    const int left = steps - j;
    int n;
    if (guard <= 0) {
      n = min(left, sound ? min(careful, pause) : careful);
      if (can && wires.template careful<Stepper, STRIDE>(n, calm, FR, FC, nan, lanes, save)) {
        again = 2 * kCarefulRun;
        careful = min(2 * careful, kMostRun);
      } else {
        if (!sound && (again == kMostPause || left <= kMostPause)) break;
        guard = again;
        again = min(2 * again, kMostPause);
        careful = kCarefulRun;
        continue;
      }
    } else {
      n = wires.template guarded<Stepper, STRIDE>(min(left, guard), lanes, save);
      guard -= n;
    }
    j += n;
    pause -= n;
  }
  if (j < steps) {
    F nI0[10], V0[9];
    const Stepper pk = resume<Stepper, STRIDE>(wires, save, ni, nv, nI0, V0);
    exact_steps_guarded(pk, steps - j, ni, nv, nI0, V0);
  } else {
    load_state<STRIDE>(save, ni, nv);
  }
}

// EXACT, one wire per thread: DualExact's arithmetic and guards on scalar
// instructions (the batched kernel's one-wire tiles).  Bit-identical to it.
template <bool DTF>
struct SoloExact {
  float L, dt;
  Recip kR, kC, kdt;
  __device__ __forceinline__ SoloExact(float l, float r, float c, float d) {
    L = l;
    dt = d;
    kR = make_recip(r);
    kC = make_recip(c);
    if (!DTF) kdt = make_recip(d);
  }
  static __device__ __forceinline__ bool eligible(float r, float c, float d) {
    return divisor_ok(r, kRMin, kRMax) && divisor_ok(c, kCMin, kCMax) &&
           (DTF || divisor_ok(d, kCMin, kCMax));
  }
  __device__ __forceinline__ void step(float (&ni)[10], float (&nv)[11], const float (&I0)[10],
                                       const float (&V0)[9]) const {
    float a1[10], a2[10];
    bool bad = false;
#pragma unroll
    for (int k = 0; k < 10; k++) {
      a1[k] = __fmul_rn(L, __fsub_rn(ni[k], I0[k]));
      const float q1 = DTF ? dt_quot(a1[k]) : recip_quot(a1[k], kdt);
      a2[k] = __fsub_rn(__fsub_rn(nv[k + 1], nv[k]), q1);
      if (!DTF) bad |= outside(a1[k], kCLo, kCHi);
      bad |= outside(a2[k], kRLo, kRHi);
    }
    // Leaving the corrected quotient as DualExact::step does.
    bool wide = false;
    if (!bad) {
#pragma unroll
      for (int k = 0; k < 10; k++) ni[k] = recip_quot(a2[k], kR);
    } else {
      bool rare = !DTF;
      if (DTF) {
#pragma unroll
        for (int k = 0; k < 10; k++)
          rare |= tiny_nonzero(a1[k], kDtTiny) | subnormal_quot(a2[k], kR);
      }
      if (!rare) {
#pragma unroll
        for (int k = 0; k < 10; k++) ni[k] = wide_quot(a2[k], kR, kRLo, kRHi);
      } else {
        const float R = -kR.nb;
#pragma unroll
        for (int k = 0; k < 10; k++)
          ni[k] = __fdiv_rn(__fsub_rn(__fsub_rn(nv[k + 1], nv[k]), __fdiv_rn(a1[k], dt)), R);
      }
      wide = true;
    }
    float a3[9];
    bad = false;
#pragma unroll
    for (int k = 0; k < 9; k++) {
      a3[k] = __fmul_rn(dt, __fsub_rn(ni[k], ni[k + 1]));
      bad |= fabsf(a3[k]) < kCLo;
    }
    if (!DTF || wide) {
#pragma unroll
      for (int k = 0; k < 9; k++) bad |= fabsf(a3[k]) > kCHi;
    }
    if (!bad) {
#pragma unroll
      for (int k = 0; k < 9; k++) nv[k + 1] = __fadd_rn(V0[k], recip_quot(a3[k], kC));
    } else {
      bool rare = false;
#pragma unroll
      for (int k = 0; k < 9; k++) rare |= subnormal_quot(a3[k], kC);
      if (!rare) {
#pragma unroll
        for (int k = 0; k < 9; k++) nv[k + 1] = __fadd_rn(V0[k], wide_quot(a3[k], kC, kCLo, kCHi));
      } else {
        const float C = -kC.nb;
#pragma unroll
        for (int k = 0; k < 9; k++) nv[k + 1] = __fadd_rn(V0[k], __fdiv_rn(a3[k], C));
      }
    }
  }
  // As in DualExact.
  __device__ __forceinline__ uint32_t check() {
    const float nb[2] = {kR.nb, kC.nb}, y[2] = {kR.y, kC.y};
    float yl[2] = {kR.yl, kC.yl};
    const uint32_t right = check_split(nb, y, yl);
    kR.yl = yl[0];
    kC.yl = yl[1];
    return right;
  }
  static __device__ __forceinline__ float cut(const Recip &k) { return cut_yl(-k.nb); }
  template <QuotForm FR, QuotForm FC, bool LOW>
  __device__ __forceinline__ void step_free(float (&ni)[10], float (&nv)[11],
                                            const float (&I0)[10], const float (&V0)[9],
                                            float &low) const {
    float a[10];
#pragma unroll
    for (int k = 0; k < 10; k++) {
      const float a1 = __fmul_rn(L, __fsub_rn(ni[k], I0[k]));
      a[k] = __fsub_rn(__fsub_rn(nv[k + 1], nv[k]), dt_quot(a1));
      ni[k] = free_quot<FR>(a[k], kR);
    }
#pragma unroll
    for (int k = 0; k < 10; k += 2)
      if (LOW) low = min_abs(low, a[k], a[k + 1]);
#pragma unroll
    for (int k = 0; k < 9; k++) {
      a[k] = __fmul_rn(dt, __fsub_rn(ni[k], ni[k + 1]));
      nv[k + 1] = __fadd_rn(V0[k], free_quot<FC>(a[k], kC));
    }
#pragma unroll
    for (int k = 0; k < 8; k += 2)
      if (LOW) low = min_abs(low, a[k], a[k + 1]);
    if (LOW) low = fminf(low, fabsf(a[8]));
  }
  template <QuotForm FORM>
  static __device__ __forceinline__ float wide(float a, const Recip &k, bool cut, uint32_t &low) {
    const uint32_t t = order(a);
    const float q = free_quot<FORM>(a, k, cut), z = __fmul_rn(a, k.y);
    low = min(low, t);
    return t >= kOrderInf ? z : q;
  }
  template <QuotForm FORM>
  __device__ __forceinline__ void step_wide(float (&ni)[10], float (&nv)[11],
                                            const float (&I0)[10], const float (&V0)[9], bool cutR,
                                            bool cutC, uint32_t &lowR, uint32_t &lowC) const {
#pragma unroll
    for (int k = 0; k < 10; k++) {
      const float a1 = __fmul_rn(L, __fsub_rn(ni[k], I0[k]));
      ni[k] = wide<FORM>(__fsub_rn(__fsub_rn(nv[k + 1], nv[k]), dt_quot(a1)), kR, cutR, lowR);
    }
#pragma unroll
    for (int k = 0; k < 9; k++)
      nv[k + 1] =
          __fadd_rn(V0[k], wide<FORM>(__fmul_rn(dt, __fsub_rn(ni[k], ni[k + 1])), kC, cutC, lowC));
  }
  __device__ __forceinline__ bool can_wide(const float (&I0)[10]) const {
    return wide_wire(least_order(I0), L, kC.nb);
  }
  static __device__ __forceinline__ uint32_t least_order(const float (&ni)[10]) {
    uint32_t m = ~0u;
#pragma unroll
    for (int k = 0; k < 10; k++) m = min(m, order(ni[k]));
    return m;
  }
  __device__ __forceinline__ float most_C() const { return fabsf(kC.nb); }
  static __device__ __forceinline__ bool calm(const float (&ni)[10]) {
    float most = 0.0f, drop = __int_as_float(0x7f800000);
#pragma unroll
    for (int k = 0; k < 10; k++) most = fmaxf(most, fabsf(ni[k]));
#pragma unroll
    for (int k = 0; k < 9; k++) drop = fminf(drop, fabsf(__fsub_rn(ni[k], ni[k + 1])));
    return (least_current(ni) >= 0x1p-48f) & (drop >= 0x1p-20f) & (most <= 0x1p40f);
  }
  static __device__ __forceinline__ bool starts_zero(const float (&ni)[10]) {
    return (ni[4] == 0.0f) & (ni[5] == 0.0f);
  }
  __device__ __forceinline__ bool sound(const float (&I0)[10], const float (&V0)[9]) const {
    float i = fabsf(I0[0]), v = fabsf(V0[0]);
#pragma unroll
    for (int k = 1; k < 10; k++) i = fminf(i, fabsf(I0[k]));
#pragma unroll
    for (int k = 1; k < 9; k++) v = fminf(v, fabsf(V0[k]));
    return sound_wire(i, v, L, kC.nb, dt);
  }
  __device__ __forceinline__ void step_all_nan(float (&ni)[10], float (&nv)[11],
                                               const float (&I0)[10],
                                               const float (&V0)[9]) const {
#pragma unroll
    for (int k = 0; k < 10; k++) {
      const float a1 = __fmul_rn(L, __fsub_rn(ni[k], I0[k]));
      const float q1 = DTF ? dt_quot(a1) : split_quot(a1, kdt);
      ni[k] = split_quot(__fsub_rn(__fsub_rn(nv[k + 1], nv[k]), q1), kR);
    }
#pragma unroll
    for (int k = 0; k < 9; k++)
      nv[k + 1] = __fadd_rn(V0[k], split_quot(__fmul_rn(dt, __fsub_rn(ni[k], ni[k + 1])), kC));
  }
  static constexpr uint32_t kWires = 1u;
  static constexpr bool kFrontHere = false;
  static __device__ __forceinline__ float state_sum(const float (&ni)[10], const float (&nv)[11]) {
    float s = ni[9], t = nv[9];
#pragma unroll
    for (int k = 0; k < 9; k++) s = __fadd_rn(s, ni[k]);
#pragma unroll
    for (int k = 1; k < 9; k++) t = __fadd_rn(t, nv[k]);
    return __fadd_rn(s, t);
  }
  static __device__ __forceinline__ float least_current(const float (&ni)[10]) {
    float m = __int_as_float(0x7f800000);
#pragma unroll
    for (int k = 0; k < 10; k += 2) m = min_abs(m, ni[k], ni[k + 1]);
    return m;
  }
  static __device__ __forceinline__ uint32_t all_nan(const float (&ni)[10], const float (&nv)[11]) {
    uint32_t nan = nan_bits(ni[0]);
    if (nan) {
#pragma unroll
      for (int k = 1; k < 10; k++) nan &= nan_bits(ni[k]) & nan_bits(nv[k]);
    }
    return nan;
  }
};

__device__ __forceinline__ const float *pick_instance(uint8_t loc, const float *pvt,
                                                      const float *shr, const float *ghost) {
  // get_node (apps/circuit/circuit_gpu.cu:40-59) without its assert: a
  // location outside {0,1,2} reads the ghost instance; ckt_sanity_check_wires
  // and ckt_graph_create reject such wires.
  return loc == CKT_PRIVATE_PTR ? pvt : (loc == CKT_SHARED_PTR ? shr : ghost);
}

// Device views of the wire region and of the node voltages CNC reads.
struct WireArrays {
  const uint32_t *in_ptr, *out_ptr;
  const uint8_t *in_loc, *out_loc;
  const float *L, *R, *C;
  float *cur, *vol;
  int64_t S;  // segment stride
};
struct NodeVolts {
  const float *pvt, *shr, *ghost;
};

// The wires of a thread, as exact_steps takes them.
struct WireSource {
  const float *L, *R, *C, *cur, *vol;
  int64_t S;
  float dt;
};
// n LOW or wide steps on the state in `save`.  FR, FC: the warp's quotient
// forms.  Returns whether they came out right; otherwise the state there is as
// it was.  Out of line, as guarded_steps: rare, and the registers of either
// would spill the free steps' loop, and each other's.
template <typename Stepper, int STRIDE, typename Wires, typename F>
__device__ __noinline__ bool careful_steps(const Wires wires, int n, bool calm, QuotForm FR,
                                           QuotForm FC, uint32_t nan, uint32_t lanes, F *save) {
  F nI0[10], V0[9], ni[10], nv[11];
  const Stepper pk = resume<Stepper, STRIDE>(wires, save, ni, nv, nI0, V0);
  bool right;
  if (calm) {
    float low = __int_as_float(0x7f800000);
    if (FR == kSplit && FC == kSplit) {
#pragma unroll 1
      for (int i = 0; i < n; i++) pk.template step_free<kSplit, kSplit, true>(ni, nv, nI0, V0, low);
    } else {
#pragma unroll 1
      for (int i = 0; i < n; i++)
        pk.template step_free<kCorrected, kCorrected, true>(ni, nv, nI0, V0, low);
    }
    right = low >= kCLo;
  } else {
    uint32_t lowR = ~0u, lowC = ~0u;
    if (FR == kSplit && FC == kSplit) {
#pragma unroll 1
      for (int i = 0; i < n; i++)
        pk.template step_wide<kSplit>(ni, nv, nI0, V0, false, false, lowR, lowC);
    } else if (FR != kCorrected && FC != kCorrected) {
#pragma unroll 1
      for (int i = 0; i < n; i++)
        pk.template step_wide<kEither>(ni, nv, nI0, V0, FR == kCut, FC == kCut, lowR, lowC);
    } else {
#pragma unroll 1
      for (int i = 0; i < n; i++)
        pk.template step_wide<kCorrected>(ni, nv, nI0, V0, false, false, lowR, lowC);
    }
    right = lowR >= order(0x1p-66f) && lowC >= order(__fmul_rn(0x1p-77f, pk.most_C()));
  }
  if (calm || FR == kCorrected || FC == kCorrected)
    right &= (nan_bits(Stepper::state_sum(ni, nv)) & ~nan) == 0u;
  if (!__all_sync(lanes, right)) return false;
  save_state<STRIDE>(save, ni, nv);
  return true;
}
// n guarded steps, fewer if a look finds all of the warp's states all NaN.
// Returns their number.
template <typename Stepper, int STRIDE, typename Wires, typename F>
__device__ __noinline__ int guarded_steps(const Wires wires, int n, uint32_t lanes, F *save) {
  F nI0[10], V0[9], ni[10], nv[11];
  const Stepper pk = resume<Stepper, STRIDE>(wires, save, ni, nv, nI0, V0);
  int done = 0;
  do {
    const int m = min(kGuardedRun, n - done);
#pragma unroll 1
    for (int i = 0; i < m; i++) pk.step(ni, nv, nI0, V0);
    done += m;
  } while (done < n && !__all_sync(lanes, Stepper::all_nan(ni, nv) == Stepper::kWires));
  save_state<STRIDE>(save, ni, nv);
  return done;
}
struct SoloWire : WireSource {
  int64_t w;
  template <typename Stepper>
  __device__ __forceinline__ Stepper stepper() const {
    return Stepper(L[w], R[w], C[w], dt);
  }
  __device__ __forceinline__ void load(float (&I0)[10], float (&V0)[9]) const {
#pragma unroll
    for (int k = 0; k < 10; k++) I0[k] = cur[k * S + w];
#pragma unroll
    for (int k = 0; k < 9; k++) V0[k] = vol[k * S + w];
  }
  template <typename Stepper, int STRIDE>
  __device__ __forceinline__ bool careful(int n, bool calm, QuotForm FR, QuotForm FC, uint32_t nan,
                                          uint32_t lanes, float *save) const {
    return careful_steps<Stepper, STRIDE>(*this, n, calm, FR, FC, nan, lanes, save);
  }
  template <typename Stepper, int STRIDE>
  __device__ __forceinline__ int guarded(int n, uint32_t lanes, float *save) const {
    return guarded_steps<Stepper, STRIDE>(*this, n, lanes, save);
  }
};
struct DualWires : WireSource {
  int64_t wa, wb;
  template <typename Stepper>
  __device__ __forceinline__ Stepper stepper() const {
    return Stepper(make_float2(L[wa], L[wb]), make_float2(R[wa], R[wb]),
                   make_float2(C[wa], C[wb]), dt);
  }
  __device__ __forceinline__ void load(float2 (&nI0)[10], float2 (&V0)[9]) const {
#pragma unroll
    for (int k = 0; k < 10; k++) nI0[k] = make_float2(-cur[k * S + wa], -cur[k * S + wb]);
#pragma unroll
    for (int k = 0; k < 9; k++) V0[k] = make_float2(vol[k * S + wa], vol[k * S + wb]);
  }
  template <typename Stepper, int STRIDE>
  __device__ __forceinline__ bool careful(int n, bool calm, QuotForm FR, QuotForm FC, uint32_t nan,
                                          uint32_t lanes, float2 *save) const {
    return careful_steps<Stepper, STRIDE>(*this, n, calm, FR, FC, nan, lanes, save);
  }
  template <typename Stepper, int STRIDE>
  __device__ __forceinline__ int guarded(int n, uint32_t lanes, float2 *save) const {
    return guarded_steps<Stepper, STRIDE>(*this, n, lanes, save);
  }
};

// One wire's whole inner loop: load, S steps in registers, store.
// EXACT: save is this thread's column of kSavedState rows of STRIDE floats in
// shared memory, and dt (float)1e-6; STRIDE 0: guarded steps, any dt.
template <int MODE, int INIT, int STRIDE = 0>
__device__ __forceinline__ void cnc_wire(int64_t w, const WireArrays &a, const NodeVolts &nv_in,
                                         int steps, float dt, float *save = nullptr,
                                         float *i0_out = nullptr, float *i9_out = nullptr) {
  const int64_t S = a.S;
  float I0[10], V0[9], ni[10], nv[11];
#pragma unroll
  for (int k = 0; k < 10; k++) I0[k] = a.cur[k * S + w];
#pragma unroll
  for (int k = 0; k < 9; k++) V0[k] = a.vol[k * S + w];
  const uint32_t in = a.in_ptr[w], out = a.out_ptr[w];
  const float v_out = pick_instance(a.out_loc[w], nv_in.pvt, nv_in.shr, nv_in.ghost)[out];
#pragma unroll
  for (int k = 0; k < 10; k++) ni[k] = I0[k];
  if (INIT == CKT_INIT_KERNEL) {
    nv[0] = pick_instance(a.in_loc[w], nv_in.pvt, nv_in.shr, nv_in.ghost)[in];
#pragma unroll
    for (int k = 0; k < 9; k++) nv[k + 1] = V0[k];
  } else {
#pragma unroll
    for (int k = 0; k < 9; k++) nv[k] = V0[k];
    nv[9] = 0.0f;
  }
  nv[10] = v_out;

  if constexpr (MODE == CKT_MODE_FAST) {
    const PackedFast pk(a.L[w], a.R[w], a.C[w], dt);
    float2 dp[5], nI0[5], vp[6], V0p[4];
#pragma unroll
    for (int p = 0; p < 5; p++) {
      nI0[p] = make_float2(-I0[p], -I0[p + 5]);
      dp[p] = __fadd2_rn(make_float2(I0[p], I0[p + 5]), nI0[p]);
    }
#pragma unroll
    for (int q = 0; q < 6; q++) vp[q] = make_float2(nv[q], nv[q + 5]);
#pragma unroll
    for (int q = 0; q < 4; q++) V0p[q] = make_float2(V0[q], V0[q + 5]);
    if (steps > 0) {
      int j = 1;
#pragma unroll 1
      for (; j < steps; j++) pk.step<false>(dp, vp, nI0, V0p, V0[4]);
      pk.step<true>(dp, vp, nI0, V0p, V0[4]);
#pragma unroll
      for (int p = 0; p < 5; p++) {
        ni[p] = dp[p].x;
        ni[p + 5] = dp[p].y;
      }
#pragma unroll
      for (int q = 0; q < 6; q++) {
        nv[q] = vp[q].x;
        nv[q + 5] = vp[q].y;
      }
    }
  } else if constexpr (MODE == kModeFastScalar) {
    const FastStep fs(a.L[w], a.R[w], a.C[w], dt);
    if (steps > 0) {
      float d[10];
#pragma unroll
      for (int k = 0; k < 10; k++) d[k] = __fsub_rn(I0[k], I0[k]);
      int j = 1;
#pragma unroll 1
      for (; j + 2 <= steps; j += 2) {
        fs.step<false>(d, nv, I0, V0);
        fs.step<false>(d, nv, I0, V0);
      }
      if (j < steps) fs.step<false>(d, nv, I0, V0);
      fs.step<true>(d, nv, I0, V0);
#pragma unroll
      for (int k = 0; k < 10; k++) ni[k] = d[k];
    }
  } else if (MODE == CKT_MODE_EXACT && (STRIDE || __float_as_uint(dt) == kDtBits) &&
             SoloExact<true>::eligible(a.R[w], a.C[w], dt)) {
    if constexpr (STRIDE > 0) {
      const SoloWire ws = {{a.L, a.R, a.C, a.cur, a.vol, S, dt}, w};
      exact_steps<STRIDE, SoloExact<true>>(ws, steps, ni, nv, save);
    } else {
      const SoloExact<true> ws(a.L[w], a.R[w], a.C[w], dt);
      exact_steps_guarded(ws, steps, ni, nv, I0, V0);
    }
  } else if (MODE == CKT_MODE_EXACT && !STRIDE && __float_as_uint(dt) != kDtBits &&
             SoloExact<false>::eligible(a.R[w], a.C[w], dt)) {
    const SoloExact<false> ws(a.L[w], a.R[w], a.C[w], dt);
    exact_steps_guarded(ws, steps, ni, nv, I0, V0);
  } else {
    static_assert(MODE == CKT_MODE_EXACT || MODE == CKT_MODE_EXACT_DIVIDE, "unknown mode");
    const DivideStep ws(a.L[w], a.R[w], a.C[w], dt);
    int j = 0;
#pragma unroll 1
    for (; j + 2 <= steps; j += 2) {
      ws.step(ni, nv, I0, V0);
      ws.step(ni, nv, I0, V0);
    }
    if (j < steps) ws.step(ni, nv, I0, V0);
  }

#pragma unroll
  for (int k = 0; k < 10; k++) a.cur[k * S + w] = ni[k];
#pragma unroll
  for (int k = 0; k < 9; k++) a.vol[k * S + w] = nv[k + 1];
  if (i0_out) *i0_out = ni[0];
  if (i9_out) *i9_out = ni[9];
}

// Two wires per thread (FAST: DualFast, EXACT: DualExact): thread t of a
// block handles wires base + t and base + t + block size, so each field's
// loads and stores stay one contiguous line per warp.  Without a partner wire the
// thread runs its wire in both lanes and stores one.
// save, STRIDE: as cnc_wire's, of float2.
template <int MODE, int INIT, int STRIDE>
__device__ __forceinline__ void cnc_wire_pair(int64_t wa, int64_t wb, bool has_b,
                                              const WireArrays &a, const NodeVolts &nvin,
                                              int steps, float dt, float2 *save,
                                              float2 *i0_out = nullptr,
                                              float2 *i9_out = nullptr) {
  static_assert(MODE == CKT_MODE_FAST || MODE == CKT_MODE_EXACT, "paired modes: FAST, EXACT");
  const int64_t S = a.S;
  const float2 L2 = make_float2(a.L[wa], a.L[wb]), R2 = make_float2(a.R[wa], a.R[wb]),
               C2 = make_float2(a.C[wa], a.C[wb]);
  const bool dt_fixed = STRIDE || __float_as_uint(dt) == kDtBits;
  if (MODE == CKT_MODE_EXACT &&
      !(dt_fixed ? DualExact<true>::eligible(R2, C2, dt) : DualExact<false>::eligible(R2, C2, dt))) {
    // a divisor outside the corrected quotients' range: the divide routine
    float ia0, ia9, ib0, ib9;
    cnc_wire<CKT_MODE_EXACT_DIVIDE, INIT>(wa, a, nvin, steps, dt, nullptr, &ia0, &ia9);
    ib0 = ia0;
    ib9 = ia9;
    if (has_b) cnc_wire<CKT_MODE_EXACT_DIVIDE, INIT>(wb, a, nvin, steps, dt, nullptr, &ib0, &ib9);
    if (i0_out) *i0_out = make_float2(ia0, ib0);
    if (i9_out) *i9_out = make_float2(ia9, ib9);
    return;
  }
  // FAST: ni holds d_k = i_k - I0_k during the loop, then the currents;
  // EXACT: ni holds the currents throughout.
  float2 ni[10], nI0[10], nv[11], V0[9];
#pragma unroll
  for (int k = 0; k < 10; k++) {
    const float x = a.cur[k * S + wa], y = a.cur[k * S + wb];
    nI0[k] = make_float2(-x, -y);
    ni[k] = MODE == CKT_MODE_FAST ? __fadd2_rn(make_float2(x, y), nI0[k]) : make_float2(x, y);
  }
#pragma unroll
  for (int k = 0; k < 9; k++) V0[k] = make_float2(a.vol[k * S + wa], a.vol[k * S + wb]);
  const float out_a = pick_instance(a.out_loc[wa], nvin.pvt, nvin.shr, nvin.ghost)[a.out_ptr[wa]];
  const float out_b = pick_instance(a.out_loc[wb], nvin.pvt, nvin.shr, nvin.ghost)[a.out_ptr[wb]];
  if (INIT == CKT_INIT_KERNEL) {
    nv[0] = make_float2(pick_instance(a.in_loc[wa], nvin.pvt, nvin.shr, nvin.ghost)[a.in_ptr[wa]],
                        pick_instance(a.in_loc[wb], nvin.pvt, nvin.shr, nvin.ghost)[a.in_ptr[wb]]);
#pragma unroll
    for (int k = 0; k < 9; k++) nv[k + 1] = V0[k];
  } else {
#pragma unroll
    for (int k = 0; k < 9; k++) nv[k] = V0[k];
    nv[9] = make_float2(0.0f, 0.0f);
  }
  nv[10] = make_float2(out_a, out_b);
  if constexpr (MODE == CKT_MODE_FAST) {
    const DualFast pk(L2, R2, C2, dt);
    if (steps > 0) {
      // Not unrolled: one step's 48 instructions stay in the scheduler's
      // instruction cache (4,194,304 wires x 1000 steps: 1 / 2 / 4 steps per
      // iteration 5.55 / 5.76 / 6.25 ms).
#pragma unroll 1
      for (int j = 1; j < steps; j++) pk.step<false>(ni, nv, nI0, V0);
      pk.step<true>(ni, nv, nI0, V0);
    } else {
#pragma unroll
      for (int k = 0; k < 10; k++) ni[k] = make_float2(-nI0[k].x, -nI0[k].y);  // no step: I0
    }
  } else if constexpr (STRIDE > 0) {
    const DualWires ws = {{a.L, a.R, a.C, a.cur, a.vol, S, dt}, wa, wb};
    exact_steps<STRIDE, DualExact<true>>(ws, steps, ni, nv, save);
  } else if (dt_fixed) {
    const DualExact<true> pk(L2, R2, C2, dt);
    exact_steps_guarded(pk, steps, ni, nv, nI0, V0);
  } else {
    const DualExact<false> pk(L2, R2, C2, dt);
    exact_steps_guarded(pk, steps, ni, nv, nI0, V0);
  }
#pragma unroll
  for (int k = 0; k < 10; k++) a.cur[k * S + wa] = ni[k].x;
#pragma unroll
  for (int k = 0; k < 9; k++) a.vol[k * S + wa] = nv[k + 1].x;
  if (has_b) {
#pragma unroll
    for (int k = 0; k < 10; k++) a.cur[k * S + wb] = ni[k].y;
#pragma unroll
    for (int k = 0; k < 9; k++) a.vol[k * S + wb] = nv[k + 1].y;
  }
  if (i0_out) *i0_out = ni[0];
  if (i9_out) *i9_out = ni[9];
}

// A block of BLOCK threads covers 2 * BLOCK wires.  FREE (EXACT): at least
// kFreeSteps steps of (float)1e-6.
template <int MODE, int INIT, bool FREE, int BLOCK>
__global__ void __launch_bounds__(BLOCK, 512 / BLOCK)
    cnc_pair_kernel(uint32_t first_wire, uint32_t num_wires, WireArrays a, NodeVolts v, int steps,
                    float dt) {
  __shared__ float2 save[FREE ? kSavedState * BLOCK : 1];
  const uint32_t ta = blockIdx.x * (2 * BLOCK) + threadIdx.x, tb = ta + BLOCK;
  if (ta >= num_wires) return;
  const bool has_b = tb < num_wires;
  cnc_wire_pair<MODE, INIT, FREE ? BLOCK : 0>(
      (int64_t)first_wire + ta, (int64_t)first_wire + (has_b ? tb : ta), has_b, a, v, steps, dt,
      save + (FREE ? threadIdx.x : 0));
}

// FREE: as above, in one-warp blocks.
template <int MODE, int INIT, bool FREE>
__global__ void __launch_bounds__(256)
    cnc_kernel(uint32_t first_wire, uint32_t num_wires, WireArrays a, NodeVolts v, int steps,
               float dt) {
  __shared__ float save[FREE ? kSavedState * 32 : 1];
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= num_wires) return;
  cnc_wire<MODE, INIT, FREE ? 32 : 0>((int64_t)first_wire + t, a, v, steps, dt,
                                      save + (FREE ? threadIdx.x : 0));
}

// ---------------------------------------------------------------------------
// calc_new_currents, EXACT, small launches: five lanes per wire.  Lane g of a
// wire holds segments 2g and 2g+1 -- their currents and the voltages v_2g,
// v_2g+1, v_2g+2 around them, the outer two of which its neighbours compute
// too, so that one exchange of currents per step (two shuffles, in flight
// together) is all the lanes tell each other.  A warp takes six wires; lanes
// 30 and 31 idle.
//
// Why: with about one warp per scheduler a step takes as long as that warp
// needs to issue it and its chain of dependent operations.  One wire per
// thread issues 125 operations one after another; here 13 paired ones and 5
// single ones, and the chain shows: 9 dependent operations and a shuffle, from
// a current over the neighbour's voltage to the next current.
//
// The arithmetic, the blocks of free steps and their checks are
// exact_steps'; the rollback state stays in registers.
// ---------------------------------------------------------------------------
constexpr int kLanesPerWire = 5;
constexpr uint32_t kLaneWires = 6;  // per warp

// What a lane carries from step to step.  The signs let every difference of
// a free step be a paired addition; negation is exact.
struct LaneState {
  float2 x;  // -i_2g, i_2g+1
  float2 e;  // v_2g, v_2g+2
  float nb;  // -v_2g+1
};

// RN(a / b) of N dividends and any divisor: corrected quotients where all are
// in their range, wide_quot where no quotient is subnormal (zero dividends, as
// at rest, above all), the divide routine elsewhere.
template <int N>
__device__ __forceinline__ void any_quot(const float (&a)[N], float (&q)[N], const Recip &k,
                                         bool eligible, float lo, float hi) {
  bool off = !eligible, rare = !eligible;
#pragma unroll
  for (int i = 0; i < N; i++) off |= outside(a[i], lo, hi);
  if (!off) {
#pragma unroll
    for (int i = 0; i < N; i++) q[i] = recip_quot(a[i], k);
    return;
  }
#pragma unroll
  for (int i = 0; i < N; i++) rare |= subnormal_quot(a[i], k);
#pragma unroll
  for (int i = 0; i < N; i++) q[i] = rare ? div_rn(a[i], -k.nb) : wide_quot(a[i], k, lo, hi);
}

struct LaneWire {
  Recip2 R, E;  // R twice; C of v_2g and v_2g+2, 1 / infinity where the wire ends there
  Recip C;
  float L, dt;
  float2 nX0, Ve;  // starting currents I_2g, -I_2g+1; starting voltages of v_2g, v_2g+2
  float nVb;       // minus that of v_2g+1
  int left, right;  // lanes of the neighbours (the lane itself at the wire's ends)
  bool first, last, okR, okC;  // okR, okC: eligible divisors (divisor_ok)

  // FR, FC, LOW: as DualExact::step_free.  The voltages at the wire's ends
  // stay, V + a * 0, but for the sign of a zero (settle_zeros).
  template <QuotForm FR, QuotForm FC, bool LOW>
  __device__ __forceinline__ void step_free(LaneState &s, float &low) const {
    const float2 neg1 = make_float2(-1.0f, -1.0f);
    const float2 a1 = __fmul2_rn(make_float2(L, L), __fadd2_rn(s.x, nX0));
    const float2 a2 =
        __ffma2_rn(dt_quot2(a1), neg1, __fadd2_rn(s.e, make_float2(s.nb, s.nb)));
    s.x = free_quot2<FR>(a2, R);
    const float l = __shfl_sync(0xffffffffu, s.x.y, left);
    const float r = __shfl_sync(0xffffffffu, s.x.x, right);
    const float a3 = __fmul_rn(dt, __fadd_rn(s.x.x, s.x.y));
    s.nb = __fadd_rn(nVb, free_quot<FC>(a3, C));
    const float2 ae = __fmul2_rn(make_float2(dt, dt), __fadd2_rn(make_float2(l, r), s.x));
    s.e = __fadd2_rn(Ve, free_quot2<FC>(ae, E));
    if (LOW) {
      low = min_abs(low, a2.x, a2.y);
      low = min_abs(low, a3, first ? 1.0f : ae.x);
      low = fminf(low, last ? 1.0f : fabsf(ae.y));
    }
  }
  // After accepted free steps.  Where V0 + q cancels, so does -V0 - q, and both
  // sums are +0: nb is +0 where minus the voltage is -0.  (V0 + q has no other
  // zeros: V0 is not zero, or q, of a dividend of at least kCLo, is not.)  And
  // V + a * 0 is +0 where V is -0 and a positive.  Inside the block those signs
  // matter no more than those of the zero quotients (exact_steps): they reach a
  // difference of voltages only where it is zero.
  __device__ __forceinline__ void settle_zeros(LaneState &s) const {
    if (s.nb == 0.0f) s.nb = -0.0f;
    if (first) s.e.x = Ve.x;
    if (last) s.e.y = Ve.y;
  }
  // As DualExact::step_wide, on the values themselves: a difference of
  // negated values has the other sign only where it is not zero.
  template <QuotForm FORM>
  __device__ __forceinline__ void step_wide(LaneState &s, bool cutR, bool cutC, uint32_t &lowR,
                                            uint32_t &lowC) const {
    const float2 i = make_float2(-s.x.x, s.x.y), I0 = make_float2(nX0.x, -nX0.y);
    const float vb = -s.nb;
    const float2 a1 = __fmul2_rn(make_float2(L, L), sub2(i, I0));
    const float2 dv = sub2(make_float2(vb, s.e.y), make_float2(s.e.x, vb));
    const float2 q = DualExact<true>::wide<FORM>(sub2(dv, dt_quot2(a1)), R, cutR, lowR);
    const float l = __shfl_sync(0xffffffffu, q.y, left);
    const float r = __shfl_sync(0xffffffffu, q.x, right);
    s.x = make_float2(-q.x, q.y);
    s.nb = -__fadd_rn(-nVb, SoloExact<true>::wide<FORM>(__fmul_rn(dt, __fsub_rn(q.x, q.y)), C, cutC, lowC));
    const float va = __fadd_rn(
        Ve.x, SoloExact<true>::wide<FORM>(first ? 1.0f : __fmul_rn(dt, __fsub_rn(l, q.x)), C, cutC, lowC));
    const float vc = __fadd_rn(
        Ve.y, SoloExact<true>::wide<FORM>(last ? 1.0f : __fmul_rn(dt, __fsub_rn(q.y, r)), C, cutC, lowC));
    if (!first) s.e.x = va;
    if (!last) s.e.y = vc;
  }
  // The reference's step for every state and divisor.
  __device__ __forceinline__ float dt_div(float a) const {
    return tiny_nonzero(a, kDtTiny) ? __fdiv_rn(a, dt) : dt_quot(a);
  }
  __device__ __forceinline__ void step(LaneState &s) const {
    const Recip r = {R.nb.x, R.y.x, R.yl.x};
    const float va = s.e.x, vb = -s.nb, vc = s.e.y;
    const float q0 = dt_div(__fmul_rn(L, __fsub_rn(-s.x.x, nX0.x)));
    const float q1 = dt_div(__fmul_rn(L, __fsub_rn(s.x.y, -nX0.y)));
    const float ar[2] = {__fsub_rn(__fsub_rn(vb, va), q0), __fsub_rn(__fsub_rn(vc, vb), q1)};
    float i[2], q[3];
    any_quot(ar, i, r, okR, kRLo, kRHi);
    const float l = __shfl_sync(0xffffffffu, i[1], left);
    const float n = __shfl_sync(0xffffffffu, i[0], right);
    // a voltage at the wire's end stays: the middle one's dividend again
    const float db = __fmul_rn(dt, __fsub_rn(i[0], i[1]));
    const float ac[3] = {first ? db : __fmul_rn(dt, __fsub_rn(l, i[0])), db,
                         last ? db : __fmul_rn(dt, __fsub_rn(i[1], n))};
    any_quot(ac, q, C, okC, kCLo, kCHi);
    s.x = make_float2(-i[0], i[1]);
    s.nb = -__fadd_rn(-nVb, q[1]);
    if (!first) s.e.x = __fadd_rn(Ve.x, q[0]);
    if (!last) s.e.y = __fadd_rn(Ve.y, q[2]);
  }
  template <QuotForm FR, QuotForm FC, bool LOW>
  __device__ __forceinline__ void steps_free(LaneState &s, int n, float &low) const {
#pragma unroll 4
    for (int i = 0; i < n; i++) step_free<FR, FC, LOW>(s, low);
  }
};

template <int INIT>
__global__ void __launch_bounds__(32)
    cnc_lanes_kernel(uint32_t first_wire, uint32_t num_wires, WireArrays a, NodeVolts v, int steps,
                     float dt) {
  constexpr uint32_t kAll = 0xffffffffu;
  const uint32_t lane = threadIdx.x, g = lane % kLanesPerWire, slot = lane / kLanesPerWire;
  const uint32_t t = blockIdx.x * kLaneWires + min(slot, kLaneWires - 1u);
  // Lanes without a wire of their own run along on the warp's last: another
  // warp's would be read while that warp stores it.
  const bool mine = slot < kLaneWires && t < num_wires;
  const int64_t w = (int64_t)first_wire + min(t, num_wires - 1u), S = a.S;
  const uint32_t wire_lanes = 0x1fu << (slot * kLanesPerWire);

  auto start_voltage = [&](uint32_t k) -> float {  // v_k before the first step
    if (k == 10) return pick_instance(a.out_loc[w], v.pvt, v.shr, v.ghost)[a.out_ptr[w]];
    if (INIT == CKT_INIT_CPU_TASK) return k < 9 ? a.vol[k * S + w] : 0.0f;
    return k ? a.vol[(k - 1) * S + w]
             : pick_instance(a.in_loc[w], v.pvt, v.shr, v.ghost)[a.in_ptr[w]];
  };
  const float r = a.R[w], c = a.C[w];
  const float I0 = a.cur[2 * g * S + w], I1 = a.cur[(2 * g + 1) * S + w];
  LaneState s = {make_float2(-I0, I1), make_float2(start_voltage(2 * g), start_voltage(2 * g + 2)),
                 -start_voltage(2 * g + 1)};
  LaneWire x;
  x.R = make_recip2(r, r);
  x.C = make_recip(c);
  x.L = a.L[w];
  x.dt = dt;
  x.nX0 = make_float2(I0, -I1);
  x.first = g == 0;
  x.last = g == kLanesPerWire - 1;
  x.Ve = make_float2(x.first ? s.e.x : a.vol[(2 * g - 1) * S + w],
                     x.last ? s.e.y : a.vol[(2 * g + 1) * S + w]);
  x.nVb = -a.vol[2 * g * S + w];
  x.left = (int)lane - (x.first ? 0 : 1);
  x.right = (int)lane + (x.last || lane == 31u ? 0 : 1);
  x.okR = divisor_ok(r, kRMin, kRMax);
  x.okC = divisor_ok(c, kCMin, kCMax);

  QuotForm FR = kCorrected, FC = kCorrected;
  bool sound = false, wide = false;
  const bool eligible = __all_sync(kAll, x.okR && x.okC);
  if (eligible) {
    const float nb[2] = {x.R.nb.x, x.C.nb}, y[2] = {x.R.y.x, x.C.y};
    float yl[2] = {x.R.yl.x, x.C.yl};
    const uint32_t checked = check_split(nb, y, yl);
    x.R.yl = make_float2(yl[0], yl[0]);
    x.C.yl = yl[1];
    FR = __all_sync(kAll, checked & 1u) ? kSplit : kCorrected;
    FC = __all_sync(kAll, checked & 2u) ? kSplit : kCorrected;
    if (FR == kCorrected) {
      const float cut = cut_yl(r);
      if (__all_sync(kAll, cut == cut)) {
        FR = kCut;
        x.R.yl = make_float2(cut, cut);
      }
    }
    if (FC == kCorrected) {
      const float cut = cut_yl(c);
      if (__all_sync(kAll, cut == cut)) {
        FC = kCut;
        x.C.yl = cut;
      }
    }
    normalize_forms(FR, FC);
    sound = __all_sync(kAll, sound_wire(fminf(fabsf(I0), fabsf(I1)),
                                        min_abs(fabsf(x.nVb), x.first ? 1.0f : x.Ve.x,
                                                x.last ? 1.0f : x.Ve.y),
                                        x.L, c, dt));
    wide = __all_sync(kAll, wide_wire(min(order(I0), order(I1)), x.L, c));
  }
  x.E.nb = make_float2(x.C.nb, x.C.nb);
  x.E.y = make_float2(x.first ? 0.0f : x.C.y, x.last ? 0.0f : x.C.y);
  x.E.yl = make_float2(x.first ? 0.0f : x.C.yl, x.last ? 0.0f : x.C.yl);

  // as exact_steps
  int j = 0, run = kFirstRun, pause = 0, penalty = kCarefulRun;
  int again = 2 * kCarefulRun, careful = kCarefulRun;
  int guard = sound ? 0 : (__any_sync(kAll, s.x.x == 0.0f && s.x.y == 0.0f) ? kFrontRun : kCalmRun);
#pragma unroll 1
  while (j < steps) {
    // which lanes' state is all NaN (each answers for what it computes)
    const uint32_t nan = __ballot_sync(
        kAll, (s.x.x != s.x.x && s.x.y != s.x.y && s.nb != s.nb && (x.first || s.e.x != s.e.x) &&
               (x.last || s.e.y != s.e.y)) ||
                  !mine);
    const bool exempt = !mine || (nan & wire_lanes) == wire_lanes;
    float low = __int_as_float(0x7f800000);
    if (nan == kAll) {  // stays so: any form of quotient gives NaN, nothing to check
      x.steps_free<kSplit, kSplit, false>(s, steps - j, low);
      break;
    }
    auto holds_nan = [&s]() {
      const float sum = __fadd_rn(__fadd_rn(s.x.x, s.x.y), __fadd_rn(__fadd_rn(s.e.x, s.e.y), s.nb));
      return sum != sum;
    };
    const LaneState start = s;
    if (sound && pause <= 0) {
      const int n = min(run, steps - j);
      if (FR == kSplit && FC == kSplit) x.steps_free<kSplit, kSplit, false>(s, n, low);
      else if (FR == kCut && FC == kSplit) x.steps_free<kCut, kSplit, false>(s, n, low);
      else if (FR == kSplit && FC == kCut) x.steps_free<kSplit, kCut, false>(s, n, low);
      else if (FR == kCut && FC == kCut) x.steps_free<kCut, kCut, false>(s, n, low);
      else if (FR == kSplit && FC == kCorrected) x.steps_free<kSplit, kCorrected, false>(s, n, low);
      else x.steps_free<kCorrected, kCorrected, false>(s, n, low);
      bool right = !holds_nan();
      if (j + n == steps) right &= fminf(fabsf(s.x.x), fabsf(s.x.y)) >= 0x1p-75f;
      if (__all_sync(kAll, right || exempt)) {
        x.settle_zeros(s);
        j += n;
        if (run == kMostRun) penalty = kCarefulRun;
        run = min(2 * run, kMostRun);
        continue;
      }
      s = start;
      run = kFirstRun;
      pause = penalty;
      penalty = min(2 * penalty, kMostPause);
    }
    const bool guarded = guard > 0 || !eligible;
    int n = min(guarded ? (eligible ? min(guard, kGuardedRun) : kGuardedRun) : careful, steps - j);
    if (sound) n = min(n, pause);
    bool right = false;
    if (!guarded) {
      right = wide ? min(order(s.x.x), order(s.x.y)) >= order(0x1p-74f)
                   : min_abs(low, s.x.x, s.x.y) >= 0x1p-48f;
      right = __all_sync(kAll, right || exempt);
    }
    if (right) {
      if (wide) {
        uint32_t lowR = ~0u, lowC = ~0u;
        if (FR == kSplit && FC == kSplit) {
#pragma unroll 1
          for (int i = 0; i < n; i++) x.step_wide<kSplit>(s, false, false, lowR, lowC);
        } else if (FR != kCorrected && FC != kCorrected) {
#pragma unroll 1
          for (int i = 0; i < n; i++)
            x.step_wide<kEither>(s, FR == kCut, FC == kCut, lowR, lowC);
        } else {
#pragma unroll 1
          for (int i = 0; i < n; i++) x.step_wide<kCorrected>(s, false, false, lowR, lowC);
          right = !holds_nan();
        }
        right &= lowR >= order(0x1p-66f) && lowC >= order(__fmul_rn(0x1p-77f, fabsf(c)));
      } else {
        x.steps_free<kCorrected, kCorrected, true>(s, n, low);
        right = low >= kCLo && !holds_nan();
        x.settle_zeros(s);
      }
      right = __all_sync(kAll, right || exempt);
      if (!right) s = start;
    }
    if (guarded) {
      guard -= n;
    } else if (right) {
      again = 2 * kCarefulRun;
      careful = min(2 * careful, kMostRun);
    } else {
      guard = again;
      again = min(2 * again, kMostPause);
      careful = kCarefulRun;
    }
    if (!right) {
#pragma unroll 1
      for (int i = 0; i < n; i++) x.step(s);
    }
    j += n;
    pause -= n;
  }
  if (mine) {
    a.cur[2 * g * S + w] = -s.x.x;
    a.cur[(2 * g + 1) * S + w] = s.x.y;
    a.vol[2 * g * S + w] = -s.nb;
    if (!x.last) a.vol[(2 * g + 1) * S + w] = s.e.y;
  }
}

// ---------------------------------------------------------------------------
// distribute_charge.  The reference adds -dt*I[0] to the in-node and
// +dt*I[9] to the out-node of every wire with atomicAdd (unordered).  Here
// each node GATHERS its contributions from a static CSR whose order is the
// reference CPU runtime's: wire order within a piece, private nodes updated
// in place, shared/ghost contributions folded per piece (identity 0) and the
// folds applied in ascending piece order.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float contribution(uint32_t wire, uint32_t end,
                                              const float *__restrict__ I0,
                                              const float *__restrict__ I9, float dt) {
  // -dt * current[0] (in end) and dt * current[9] (out end),
  // apps/circuit/circuit.cc:430-431.
  return end ? __fmul_rn(dt, I9[wire]) : __fmul_rn(-dt, I0[wire]);
}

// Whole circuit, canonical order.  A block owns BLOCK consecutive nodes,
// whose contributions are one contiguous span of the CSR.  The block first
// stages the span in shared memory -- coalesced entry loads and independent
// current gathers, so every thread has many loads in flight -- then each
// thread sums its own node's run sequentially, in the reference order.
// COHERENT loads bypass L1: used when the currents were written by other
// blocks of the same (persistent) launch.
constexpr uint32_t kDcChunk = 4096;

template <bool COHERENT>
__device__ __forceinline__ float ld_f32(const float *p) {
  return COHERENT ? __ldcg(p) : *p;
}

// Returns the thread's node's new charge; STORE = false leaves charge[]
// unwritten for a caller that consumes the value itself.
template <uint32_t BLOCK, bool COHERENT, bool STORE = true>
__device__ __forceinline__ float dc_block(uint32_t x0, uint32_t xe,
                                         const uint32_t *__restrict__ off,
                                         const uint32_t *__restrict__ ent,
                                         const float *__restrict__ I0,
                                         const float *__restrict__ I9,
                                         float *__restrict__ charge, float dt, float *sval,
                                         uint32_t *smask) {
  const uint32_t x = x0 + threadIdx.x;
  const uint32_t lo = off[x0] & 0x7fffffffu, hi = off[xe] & 0x7fffffffu;
  uint32_t b = 0, e = 0;
  bool priv = true;
  float acc = 0.0f, fold = 0.0f;
  if (x < xe) {
    const uint32_t o0 = off[x], o1 = off[x + 1];
    priv = (o0 & 0x80000000u) != 0;
    b = o0 & 0x7fffffffu;
    e = o1 & 0x7fffffffu;
    acc = charge[x];
  }
  for (uint32_t c0 = lo; c0 < hi; c0 += kDcChunk) {
    const uint32_t cn = min(kDcChunk, hi - c0);
    // Stage in batches of kDcBatch entries per thread: all entry loads of a
    // batch first, then all of its current gathers, so every thread keeps
    // kDcBatch independent loads in flight at each of the two levels.
    constexpr uint32_t kDcBatch = 8;
    for (uint32_t j0 = 0; j0 < cn; j0 += kDcBatch * BLOCK) {
      uint32_t u[kDcBatch];
#pragma unroll
      for (uint32_t r = 0; r < kDcBatch; r++) {
        const uint32_t j = j0 + r * BLOCK + threadIdx.x;
        u[r] = j < cn ? ent[c0 + j] : 0u;
      }
      float v[kDcBatch];
#pragma unroll
      for (uint32_t r = 0; r < kDcBatch; r++) {
        const uint32_t w = u[r] >> 2;
        v[r] = (u[r] & 2u) ? ld_f32<COHERENT>(I9 + w) : ld_f32<COHERENT>(I0 + w);
      }
#pragma unroll
      for (uint32_t r = 0; r < kDcBatch; r++) {
        const uint32_t j = j0 + r * BLOCK + threadIdx.x;
        // group-start flags of the warp's 32 consecutive entries, one word
        const uint32_t m = __ballot_sync(0xffffffffu, (u[r] & 1u) != 0u);
        if (j < cn) {
          sval[j] = (u[r] & 2u) ? __fmul_rn(dt, v[r]) : __fmul_rn(-dt, v[r]);
          if ((threadIdx.x & 31u) == 0u) smask[j >> 5] = m;
        }
      }
    }
    __syncthreads();
    const uint32_t i0 = max(b, c0), i1 = min(e, c0 + cn);
    if (priv) {
      for (uint32_t i = i0; i < i1; i++) acc = __fadd_rn(acc, sval[i - c0]);
    } else {
      for (uint32_t i = i0; i < i1; i++) {
        if (((smask[(i - c0) >> 5] >> ((i - c0) & 31u)) & 1u) && i != b) {
          acc = __fadd_rn(acc, fold);
          fold = 0.0f;
        }
        fold = __fadd_rn(fold, sval[i - c0]);
      }
    }
    __syncthreads();
  }
  if (x < xe) {
    if (!priv && e > b) acc = __fadd_rn(acc, fold);
    if (STORE) charge[x] = acc;
  }
  return acc;
}

// The simple schedule: one thread per node walks its own run with dependent
// loads (no staging).  Same order, same bits.
template <bool COHERENT>
__device__ __forceinline__ void dc_node(uint32_t x, const uint32_t *__restrict__ off,
                                        const uint32_t *__restrict__ ent,
                                        const float *__restrict__ I0,
                                        const float *__restrict__ I9,
                                        float *__restrict__ charge, float dt) {
  const uint32_t o0 = off[x], o1 = off[x + 1];
  const uint32_t b = o0 & 0x7fffffffu, e = o1 & 0x7fffffffu;
  float acc = charge[x];
  if (o0 & 0x80000000u) {
    for (uint32_t i = b; i < e; i++) {
      const uint32_t u = ent[i], w = u >> 2;
      acc = __fadd_rn(acc, (u & 2u) ? __fmul_rn(dt, ld_f32<COHERENT>(I9 + w))
                                    : __fmul_rn(-dt, ld_f32<COHERENT>(I0 + w)));
    }
  } else {
    float fold = 0.0f;
    for (uint32_t i = b; i < e; i++) {
      const uint32_t u = ent[i], w = u >> 2;
      if ((u & 1u) && i != b) {
        acc = __fadd_rn(acc, fold);
        fold = 0.0f;
      }
      fold = __fadd_rn(fold, (u & 2u) ? __fmul_rn(dt, ld_f32<COHERENT>(I9 + w))
                                      : __fmul_rn(-dt, ld_f32<COHERENT>(I0 + w)));
    }
    if (e > b) acc = __fadd_rn(acc, fold);
  }
  charge[x] = acc;
}

constexpr uint32_t kDcBlock = 256;

static __global__ void __launch_bounds__(kDcBlock)
    dc_all_kernel(uint32_t node_begin, uint32_t node_end, const uint32_t *__restrict__ off,
                  const uint32_t *__restrict__ ent, const float *__restrict__ I0,
                  const float *__restrict__ I9, float *__restrict__ charge, float dt) {
  __shared__ float sval[kDcChunk];
  __shared__ uint32_t smask[kDcChunk / 32];
  const uint32_t x0 = node_begin + blockIdx.x * kDcBlock;
  dc_block<kDcBlock, false>(x0, min(node_end, x0 + kDcBlock), off, ent, I0, I9, charge, dt, sval,
                            smask);
}

// One piece: one thread per node the piece touches; private nodes are
// updated in place, shared/ghost nodes fold into the given instances.
static __global__ void __launch_bounds__(256)
    dc_piece_kernel(uint32_t t0, uint32_t nt, const uint32_t *__restrict__ touch_node,
                    const uint8_t *__restrict__ touch_loc, const uint32_t *__restrict__ touch_off,
                    const uint32_t *__restrict__ pent, const float *__restrict__ I0,
                    const float *__restrict__ I9, float *charge, float *shr_fold,
                    float *ghost_fold, float dt) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nt) return;
  const uint32_t t = t0 + i;
  const uint32_t x = touch_node[t];
  const uint8_t loc = touch_loc[t];
  float *tgt = loc == CKT_PRIVATE_PTR ? charge : (loc == CKT_SHARED_PTR ? shr_fold : ghost_fold);
  float acc = tgt[x];
  for (uint32_t e = touch_off[t]; e < touch_off[t + 1]; e++) {
    const uint32_t u = pent[e];
    acc = __fadd_rn(acc, contribution(u >> 1, u & 1u, I0, I9, dt));
  }
  tgt[x] = acc;
}

// One piece without the contribution graph (distribute_charge_kernel,
// apps/circuit/circuit_gpu.cu:245-286): one thread per wire adds -dt*I[0]
// to its in-node and dt*I[9] to its out-node with atomic adds -- private
// nodes into pvt's charge, shared and ghost nodes into their fold instances
// (reduce_local, circuit_gpu.cu:219-243).  Lanes of a warp whose wire ends
// land on the same node of the same instance first combine their
// contributions: __match_any_sync groups them, and the group's first lane
// adds the group's sum, in lane order, with one atomic.  The order of the
// additions at a node is unspecified, as with the reference's atomicAdd.
__device__ __forceinline__ void warp_aggregated_add(float *target, float v, uint64_t key,
                                                    float *sbuf) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t peers = __match_any_sync(__activemask(), key);
  if (peers == (1u << lane)) {
    atomicAdd(target, v);
    return;
  }
  sbuf[lane] = v;
  __syncwarp(peers);
  if (lane == (uint32_t)(__ffs(peers) - 1)) {
    float sum = sbuf[lane];
    for (uint32_t m = peers & (peers - 1); m; m &= m - 1) sum = __fadd_rn(sum, sbuf[__ffs(m) - 1]);
    atomicAdd(target, sum);
  }
  __syncwarp(peers);  // sbuf is reused by the wire's other end
}

static __global__ void __launch_bounds__(256)
    dc_atomic_kernel(uint32_t first_wire, uint32_t num_wires, const uint32_t *__restrict__ in_ptr,
                     const uint32_t *__restrict__ out_ptr, const uint8_t *__restrict__ in_loc,
                     const uint8_t *__restrict__ out_loc, const float *__restrict__ I0,
                     const float *__restrict__ I9, float *pvt_charge, float *shr_fold,
                     float *ghost_fold, float dt) {
  __shared__ float sbuf[256];
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= num_wires) return;
  const uint32_t w = first_wire + t;
  float *warp_buf = sbuf + (threadIdx.x & ~31u);
  const uint32_t a = in_ptr[w], b = out_ptr[w];
  const uint8_t la = in_loc[w], lb = out_loc[w];
  const float ca = __fmul_rn(-dt, I0[w]), cb = __fmul_rn(dt, I9[w]);
  float *ta = la == CKT_PRIVATE_PTR ? pvt_charge : (la == CKT_SHARED_PTR ? shr_fold : ghost_fold);
  float *tb = lb == CKT_PRIVATE_PTR ? pvt_charge : (lb == CKT_SHARED_PTR ? shr_fold : ghost_fold);
  warp_aggregated_add(ta + a, ca, ((uint64_t)(la > 2 ? 2 : la) << 32) | a, warp_buf);
  warp_aggregated_add(tb + b, cb, ((uint64_t)(lb > 2 ? 2 : lb) << 32) | b, warp_buf);
}

// Application of one piece's reduction instances.
static __global__ void __launch_bounds__(256)
    apply_fold_kernel(uint32_t t0, uint32_t nt, const uint32_t *__restrict__ touch_node,
                      const uint8_t *__restrict__ touch_loc, float *shr_fold, float *ghost_fold,
                      float *charge) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nt) return;
  const uint32_t t = t0 + i;
  const uint8_t loc = touch_loc[t];
  if (loc == CKT_PRIVATE_PTR) return;
  const uint32_t x = touch_node[t];
  float *fold = loc == CKT_SHARED_PTR ? shr_fold : ghost_fold;
  charge[x] = __fadd_rn(charge[x], fold[x]);
  fold[x] = 0.0f;
}

// ---------------------------------------------------------------------------
// update_voltages: v += q/C; v *= (1 - leak); q = 0
// (apps/circuit/circuit_gpu.cu:330-335, circuit.cc:1300-1302).
// ---------------------------------------------------------------------------
__device__ __forceinline__ float uv_one(float v, float q, float c, float l) {
  return __fmul_rn(__fadd_rn(v, __fdiv_rn(q, c)), __fsub_rn(1.0f, l));
}

// Whole node range, four nodes per thread with 16-byte loads and stores; the
// last N mod 4 one by one, in the same launch.
static __global__ void __launch_bounds__(256)
    uv_all_vec4_kernel(uint32_t N, float *__restrict__ charge, float *__restrict__ voltage,
                       const float *__restrict__ cap, const float *__restrict__ leak) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N / 4u) {
    if (i == N / 4u)
      for (uint32_t x = N & ~3u; x < N; x++) {
        voltage[x] = uv_one(voltage[x], charge[x], cap[x], leak[x]);
        charge[x] = 0.0f;
      }
    return;
  }
  float4 *q = reinterpret_cast<float4 *>(charge), *v = reinterpret_cast<float4 *>(voltage);
  const float4 qq = q[i], vv = v[i], cc = reinterpret_cast<const float4 *>(cap)[i],
               ll = reinterpret_cast<const float4 *>(leak)[i];
  float4 r;
  r.x = uv_one(vv.x, qq.x, cc.x, ll.x);
  r.y = uv_one(vv.y, qq.y, cc.y, ll.y);
  r.z = uv_one(vv.z, qq.z, cc.z, ll.z);
  r.w = uv_one(vv.w, qq.w, cc.w, ll.w);
  v[i] = r;
  q[i] = make_float4(0.f, 0.f, 0.f, 0.f);
}

static __global__ void __launch_bounds__(256)
    uv_all_scalar_kernel(uint32_t first, uint32_t n, float *__restrict__ q, float *__restrict__ v,
                         const float *__restrict__ c, const float *__restrict__ l) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t x = first + i;
  v[x] = uv_one(v[x], q[x], c[x], l[x]);
  q[x] = 0.0f;
}

// One piece, instance chosen by the locator (circuit_gpu.cu:321-346).
static __global__ void __launch_bounds__(256)
    uv_piece_kernel(uint32_t first, uint32_t n, const int32_t *__restrict__ locator,
                    ckt_nodes pvt, ckt_nodes shr) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t x = first + i;
  const ckt_nodes &s = locator[x] ? pvt : shr;
  s.voltage[x] = uv_one(s.voltage[x], s.charge[x], s.capacitance[x], s.leakage[x]);
  s.charge[x] = 0.0f;
}

// distribute_charge + update_voltages in one node pass (the fused loop): the
// staged gather of dc_block, and each node's final charge goes straight into
// the voltage update instead of through memory.  Same order, same bits as
// dc_all_kernel followed by the update_voltages kernels.
static __global__ void __launch_bounds__(kDcBlock)
    dcuv_kernel(uint32_t N, const uint32_t *__restrict__ off, const uint32_t *__restrict__ ent,
                const float *__restrict__ I0, const float *__restrict__ I9,
                float *__restrict__ charge, float *__restrict__ voltage,
                const float *__restrict__ cap, const float *__restrict__ leak, float dt) {
  __shared__ float sval[kDcChunk];
  __shared__ uint32_t smask[kDcChunk / 32];
  const uint32_t x0 = blockIdx.x * kDcBlock;
  const uint32_t xe = min(N, x0 + kDcBlock);
  const uint32_t x = x0 + threadIdx.x;
  float v = 0.0f, c = 1.0f, l = 0.0f;
  if (x < xe) {  // independent of the gather: in flight while it runs
    v = voltage[x];
    c = cap[x];
    l = leak[x];
  }
  const float q = dc_block<kDcBlock, false, false>(x0, xe, off, ent, I0, I9, charge, dt, sval,
                                                  smask);
  if (x < xe) {
    voltage[x] = uv_one(v, q, c, l);
    charge[x] = 0.0f;
  }
}

// ---------------------------------------------------------------------------
// Wire validation (sanity_check_positions, circuit_gpu.cu:151-184, with an
// error word instead of assert).  Records the smallest failing wire index.
// ---------------------------------------------------------------------------
static __global__ void __launch_bounds__(256)
    sanity_kernel(ckt_piece piece, const uint32_t *__restrict__ in_ptr,
                  const uint32_t *__restrict__ out_ptr, const uint8_t *__restrict__ in_loc,
                  const uint8_t *__restrict__ out_loc, uint32_t num_nodes_total,
                  unsigned long long *first_bad) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= piece.num_wires) return;
  const uint32_t w = piece.first_wire + t;
  const uint32_t a = in_ptr[w], b = out_ptr[w];
  const uint8_t la = in_loc[w], lb = out_loc[w];
  const uint32_t lo = piece.first_node, hi = piece.first_node + piece.num_nodes;
  bool ok = la <= CKT_SHARED_PTR && lb <= CKT_GHOST_PTR;  // in-node is never a ghost
  ok = ok && a >= lo && a < hi;
  ok = ok && b < num_nodes_total;
  if (ok) {
    const bool b_inside = b >= lo && b < hi;
    ok = (lb == CKT_GHOST_PTR) ? !b_inside : b_inside;
  }
  if (!ok) atomicMin(first_bad, (unsigned long long)w);
}

}  // namespace ckt
