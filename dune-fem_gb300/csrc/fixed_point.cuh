// 64-bit block fixed-point arithmetic for FP64 data on the integer pipes.
//
// This GPU issues 2 FP64 operations per clock and SM, but 64 integer
// multiply-adds (32 x 32 + 64 bits) and 128 additions (measured with
// independent chains: DFMA 2.00, DADD 1.68, IMAD.WIDE 64.0, IADD 128 lanes per
// clock and SM).  A short dot product with constant coefficients is therefore
// cheaper in fixed point, three integer multiply-adds per term, by about a
// factor of ten, the conversions included by about four.
//
// A group of values shares the exponent of its largest one.  With E the
// biased binary64 exponent of that value (|x| < 2^(E-1022)), x is held as the
// integer X = x 2^(61-(E-1022)), truncated: |X| < 2^61, and one unit of X is
// 2^-61 of the largest value's binade, 256 times finer than that value's own
// last place.  A coefficient c, |c| <= s (s a power of two), is the integer
// C = round(c / s 2^CB), CB <= 62.  Both are split into a high and a low signed
// 32-bit limb, X = h 2^32 + l, and a dot product keeps
//     sum (X C) / 2^64 = sum h ch + (sum (h cl + l ch) + round) / 2^32,
// dropping l cl (below a quarter unit per term); round = 2^31 rounds to nearest.  The middle sum stays below
// 2^63 for up to 2 terms with CB = 62 and up to 5 with CB = 61.
#pragma once
#include <cstdint>
#include <cstring>

namespace gbfem {

#ifdef __CUDACC__
#define GBFEM_HD __host__ __device__ __forceinline__
#else
#define GBFEM_HD inline
#endif

constexpr int kFxBits = 61;          // |X| < 2^kFxBits
constexpr int kFxMinExp = 200;       // biased exponents handled in fixed point
constexpr int kFxMaxExp = 1800;
constexpr int kFxRowExpMax = 100;    // largest |log2 s| of a coefficient row

struct FxCoef {  // C = h 2^32 + l
  int h, l;
};

struct FxLimbs {
  int h, l;
};

GBFEM_HD FxLimbs fx_split(long long v) {
  FxLimbs r;
  r.l = int(uint32_t(uint64_t(v)));
  r.h = int(uint32_t(uint64_t(v) >> 32) + (uint32_t(r.l) >> 31));
  return r;
}

// acc + a b, and a b.  Written out: left to itself the compiler widens one factor
// first and multiplies 64 by 32 bits in three instructions (64^3 Q3 closed form 319
// -> 295 us with these two, kappa at the Gauss points 712 -> 620).
GBFEM_HD long long fx_mad(int a, int b, long long acc) {
#if defined(__CUDA_ARCH__)
  asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(acc) : "r"(a), "r"(b));
  return acc;
#else
  return acc + (long long)a * b;
#endif
}
GBFEM_HD long long fx_mul(int a, int b) {
#if defined(__CUDA_ARCH__)
  long long r;
  asm("mul.wide.s32 %0, %1, %2;" : "=l"(r) : "r"(a), "r"(b));
  return r;
#else
  return (long long)a * b;
#endif
}

// running sums of a dot product; `start` joins the result.  (no_hh, no_mid: nothing
// in that sum yet; known at compile time in unrolled code, they save the zeros.)
struct FxAcc {
  long long hh, mid;
  bool no_hh, no_mid;
  GBFEM_HD FxAcc() : hh(0), mid(0), no_hh(true), no_mid(true) {}
  GBFEM_HD FxAcc(long long start, long long round) : hh(start), mid(round), no_hh(false), no_mid(false) {}
  GBFEM_HD static FxAcc rounded() {
    FxAcc r;
    r.mid = 1ll << 31;
    r.no_mid = false;
    return r;
  }
  GBFEM_HD void add(FxLimbs x, FxCoef c) {
    hh = no_hh ? fx_mul(x.h, c.h) : fx_mad(x.h, c.h, hh);
    mid = no_mid ? fx_mul(x.h, c.l) : fx_mad(x.h, c.l, mid);
    mid = fx_mad(x.l, c.h, mid);
    no_hh = no_mid = false;
  }
  GBFEM_HD long long value() const { return hh + (mid >> 32); }
  // the sum times 2^K, with K more of its digits
  template <int K>
  GBFEM_HD long long value_up() const { return (long long)(uint64_t(hh) << K) + (mid >> (32 - K)); }
};

GBFEM_HD uint64_t fx_bits(double v) {
#if defined(__CUDA_ARCH__)
  return uint64_t(__double_as_longlong(v));
#else
  uint64_t b;
  std::memcpy(&b, &v, 8);
  return b;
#endif
}
GBFEM_HD double fx_from_bits(uint64_t b) {
#if defined(__CUDA_ARCH__)
  return __longlong_as_double((long long)b);
#else
  double v;
  std::memcpy(&v, &b, 8);
  return v;
#endif
}

// high word of |v| (orders by magnitude: exponent, then leading fraction bits)
GBFEM_HD uint32_t fx_abs_hi(double v) { return uint32_t(fx_bits(v) >> 32) & 0x7FFFFFFFu; }

// right shift by 0 <= s < 64 (masked: one funnel shift per word)
GBFEM_HD long long fx_shr(long long v, int s) { return v >> (s & 63); }

// X of v in a group of exponent E >= v's.  A subnormal v gets a spurious
// leading bit, but E >= kFxMinExp shifts it out.
GBFEM_HD long long fx_from_double(double v, int E) {
  const uint64_t b = fx_bits(v);
  const uint32_t hi = uint32_t(b >> 32);
  int s = E - int((hi >> 20) & 0x7FFu);
  s = s < 63 ? s : 63;
  const uint64_t m = ((uint64_t((hi & 0xFFFFFu) | 0x100000u) << 32) | uint32_t(b)) << (kFxBits - 53);
  const long long x = (long long)(m >> (s & 63));
  return int(hi) < 0 ? -x : x;
}

// The power of two with the given high word (biased exponent << 20).
GBFEM_HD double fx_pow2(int hi) { return fx_from_bits(uint64_t(uint32_t(hi)) << 32); }

}  // namespace gbfem
