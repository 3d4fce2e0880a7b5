// ckt_drand.cuh -- the generator's drand48 expressions evaluated exactly in
// integer arithmetic where that is possible.
//
// load_circuit (apps/circuit/circuit.cc:1121-1186) turns each 48-bit LCG state
// x into u = x * 2^-48 (drand48) and evaluates a few double expressions.
// Several of them are exact rationals over 2^48 before their final rounding,
// and the others round a product of x by an integer to 53 bits; both can be
// computed with integer instructions, which matters on GPUs whose FP64 rate
// is a small fraction of the FP32 rate.  Each helper states the expression it
// reproduces and why the result is bit-identical.  The host build of this
// header (plain C++) lets the CPU check every helper against the double
// arithmetic it replaces.
#pragma once

#include <cstdint>
#include <cstring>

#if defined(__CUDACC__)
#define CKT_HD __host__ __device__ __forceinline__
#else
#define CKT_HD inline
#endif

namespace ckt {
namespace drand {

CKT_HD int msb64(uint64_t v) {  // index of the highest set bit, v != 0
#if defined(__CUDA_ARCH__)
  return 63 - __clzll((long long)v);
#else
  return 63 - __builtin_clzll(v);
#endif
}

CKT_HD uint64_t mulhi64(uint64_t a, uint64_t b) {
#if defined(__CUDA_ARCH__)
  return __umul64hi(a, b);
#else
  return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}

// drand48's value u = x * 2^-48 (x < 2^48), assembled from its bits: exact.
CKT_HD double value(uint64_t x) {
  if (x == 0) return 0.0;
  const int m = msb64(x);  // <= 47
  const uint64_t bits = ((uint64_t)(m - 48 + 1023) << 52) | ((x << (52 - m)) & ((1ull << 52) - 1));
  double d;
  memcpy(&d, &bits, sizeof(d));
  return d;
}

// Rounds the integer q = hi * 2^64 + lo (< 2^80) to 53 significant bits, to
// nearest with ties to even, as the double product x * n does, and returns
// floor(result / 2^48).
CKT_HD uint64_t rn53_shr48(uint64_t hi, uint64_t lo) {
  if (hi == 0 && lo == 0) return 0;
  const int m = hi ? 64 + msb64(hi) : msb64(lo);
  if (m <= 52) return lo >> 48;  // exact (hi is 0)
  const int shift = m - 52;       // 1 .. 27
  uint64_t r = (lo >> shift) | (hi << (64 - shift));
  const uint64_t rem = lo & ((1ull << shift) - 1), half = 1ull << (shift - 1);
  if (rem > half || (rem == half && (r & 1u))) r++;
  return r >> (48 - shift);
}

// (int)(drand48() * n): u * n rounded to a double, truncated (n < 2^31).
CKT_HD uint32_t trunc_mul(uint64_t x, uint32_t n) {
  return (uint32_t)rn53_shr48(mulhi64(x, n), x * (uint64_t)n);
}

// Threshold of the in-piece test: ceil(pct * 2^48), 0 when pct <= 0.
inline uint64_t pct_threshold(double pct) {
  const double t = pct * 281474976710656.0;  // * 2^48, exact
  if (!(t > 0)) return 0;
  if (t >= 9223372036854775808.0) return ~0ull;
  const uint64_t f = (uint64_t)t;
  return ((double)f == t) ? f : f + 1;
}

// 100 * drand48() < pct: 100 * u rounded to a double (100 x < 2^55 keeps its
// top 53 bits), compared with pct; as integers, RN53(100 x) < pct * 2^48.
CKT_HD bool pct_below(uint64_t x, uint64_t threshold) {
  const uint64_t p = 100 * x;
  uint64_t r = p;
  if (p >> 53) {
    const int shift = msb64(p) - 52;  // 1 or 2
    r = p >> shift;
    const uint64_t rem = p & ((1ull << shift) - 1), half = 1ull << (shift - 1);
    if (rem > half || (rem == half && (r & 1u))) r++;
    r <<= shift;
  }
  return r < threshold;
}

CKT_HD float u64_to_float(uint64_t v) {
#if defined(__CUDA_ARCH__)
  return __ull2float_rn(v);
#else
  return (float)v;
#endif
}

CKT_HD float i64_to_float(int64_t v) {
#if defined(__CUDA_ARCH__)
  return __ll2float_rn(v);
#else
  return (float)v;
#endif
}

constexpr float kTwoM48 = 3.5527136788005009e-15f;  // 2^-48, exact

// (float)(drand48() * 10 + 1) = (10 x + 2^48) / 2^48 exactly (< 2^52), so the
// only rounding is the float conversion.
CKT_HD float resistance(uint64_t x) {
  return u64_to_float(10 * x + (1ull << 48)) * kTwoM48;
}

// (float)(2 * drand48() - 1) = (2 x - 2^48) / 2^48 exactly.
CKT_HD float node_voltage(uint64_t x) {
  return i64_to_float((int64_t)(2 * x) - (int64_t)(1ull << 48)) * kTwoM48;
}

// (float)(drand48() + 1) = (x + 2^48) / 2^48 exactly.
CKT_HD float node_capacitance(uint64_t x) {
  return u64_to_float(x + (1ull << 48)) * kTwoM48;
}

// The least x that fails the in-piece test (pct_below is monotone in x: 100 x
// rounded to 53 bits never decreases); 2^48 when none does.
inline uint64_t first_crossing(uint64_t threshold) {
  uint64_t lo = 0, hi = 1ull << 48;
  while (lo < hi) {
    const uint64_t mid = (lo + hi) / 2;
    if (pct_below(mid, threshold)) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// trunc_mul by two 32-bit products: rounding x n to 53 bits can reach the next
// multiple of 2^48 only from the last 2^32 before it.
CKT_HD uint32_t trunc_mul_fast(uint64_t x, uint32_t n) {
  const uint64_t low = (x & 0xffffffffull) * n, high = (x >> 32) * n + (low >> 32);
  if ((high & 0xffffu) == 0xffffu) return trunc_mul(x, n);
  return (uint32_t)(high >> 16);
}

// (float)(u * scale + offset), double arithmetic, u = x * 2^-48: evaluated as
// a 64-bit fixed-point sum where that settles the float.
struct Affine {
  uint64_t scale, offset;  // in units of 2^(e - 64)
  int32_t exponent;        // e: scale + offset <= 2^(e - 1); 0x7fffffff: not usable
};
inline Affine make_affine(double scale, double offset) {
  Affine a = {0, 0, 0x7fffffff};
  const double sum = scale + offset;
  if (!(scale >= 0) || !(offset >= 0) || !(sum > 8.6736173798840355e-19) ||  // 2^-60
      !(sum < 1152921504606846976.0))                                       // 2^60
    return a;
  int e = -60;
  double lim = 8.6736173798840355e-19;
  while (!(sum <= lim)) {
    lim *= 2;
    e++;
  }
  e++;  // sum <= 2^(e - 1)
  double unit = 1.0;  // 2^(64 - e)
  for (int i = 0; i < 64 - e; i++) unit *= 2;
  for (int i = 0; i < e - 64; i++) unit /= 2;
  a.scale = (uint64_t)(scale * unit + 0.5);
  a.offset = (uint64_t)(offset * unit + 0.5);
  a.exponent = e;
  return a;
}
// The sum is right to two units; the double expression's two roundings move
// it by at most 2^-52 of itself.  Unless a boundary between two floats lies
// that near, the float of the one is the float of the other; otherwise (and
// for very small sums) false.
CKT_HD bool affine_float(uint64_t x, const Affine &a, float *out) {
  const uint64_t f = mulhi64(x << 16, a.scale) + a.offset;
  if (f < (1ull << 40) || a.exponent == 0x7fffffff) return false;
  const int shift = 63 - msb64(f);  // <= 23
  const uint64_t g = f << shift, low = g & ((1ull << 40) - 1), half = 1ull << 39;
  const uint64_t margin = (4ull << shift) + (1ull << 13);
  if (low - (half - margin) <= 2 * margin) return false;
  // f units of 2^(e - 64): the top bit weighs 2^(63 - shift + e - 64)
  const uint32_t bits = ((uint32_t)(126 - shift + a.exponent) << 23) +
                        ((uint32_t)(g >> 40) - 0x800000u) + (low > half ? 1u : 0u);
  memcpy(out, &bits, sizeof(bits));
  return true;
}

}  // namespace drand
}  // namespace ckt
