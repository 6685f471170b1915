// exp of an FP64 value on the integer pipes, table driven (P. T. P. Tang, ACM
// Trans. Math. Softw. 15 (1989), 144-157) in 64-bit fixed point:
//   |x| log2(e) = k + f exactly as a 128-bit product (of the 53-bit mantissa and
//   log2(e) to 64 bits), f = j / 32 + g, 2^f = 2^(j/32) e^y, y = g ln 2 < 0.0217,
//   e^y by its Taylor polynomial of degree 8 (the remainder is below 2^-68).
// All steps truncate at 2^-63 or finer, log2(e) contributes |x| 2^-64: the result is
// within 0.51 units in the last place for |x| <= 64 and 0.6 up to 700.  About 110
// integer instructions; CUDA's exp is about 20 on the FP64 pipe, 10 clocks of an SM.
#pragma once
#include <cmath>

#include "fixed_point.cuh"

namespace gbfem {

struct FxExpTables {
  uint64_t log2e;     // log2(e) 2^63
  uint64_t ln2;       // ln(2) 2^64
  uint64_t c[9];      // 2^63 / k!
  uint64_t pow[32];   // 2^(j/32) 2^63
};

inline FxExpTables fx_make_exp_tables() {
  FxExpTables t;
  auto round64 = [](long double v) { return uint64_t(v + 0.5L); };
  t.log2e = round64(ldexpl(1.0L / logl(2.0L), 63));
  t.ln2 = round64(ldexpl(logl(2.0L), 64));
  long double f = 1.0L;
  for (int k = 0; k < 9; ++k) {
    if (k) f *= k;
    t.c[k] = round64(ldexpl(1.0L / f, 63));
  }
  for (int j = 0; j < 32; ++j) t.pow[j] = round64(ldexpl(exp2l(j / 32.0L), 63));
  return t;
}

GBFEM_HD uint64_t fx_mulhi(uint64_t a, uint64_t b) {
#if defined(__CUDA_ARCH__)
  return __umul64hi(a, b);
#else
  return uint64_t((unsigned __int128)a * b >> 64);
#endif
}

// exp(x); pow: t.pow where each thread can index it
GBFEM_HD double fx_exp(double x, const FxExpTables& t, const uint64_t* pow) {
  const uint64_t b = fx_bits(x);
  const int e = int((b >> 52) & 0x7FFu) - 1023;
  const uint32_t ahi = uint32_t(b >> 32) & 0x7FFFFFFFu;
  if (ahi >= 0x4085E000u) return exp(x);  // |x| >= 700, infinity, NaN
  if (e < -54) return 1.0 + x;
  const uint64_t m = ((b & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull) << 11;
  const uint64_t hi = fx_mulhi(m, t.log2e), lo = m * t.log2e;  // |x| log2(e) 2^(62-e) = hi + lo / 2^64
  const int s = e + 2;
  uint64_t f;
  int k = 0;
  if (s > 0) {
    f = (hi << s) | (lo >> (64 - s));
    k = int(hi >> (64 - s));
  } else {
    f = hi >> -s;
  }
  if (int(uint32_t(b >> 32)) < 0) {  // -(k + f) = (-k - 1) + (1 - f)
    k = f ? -k - 1 : -k;
    f = 0ull - f;
  }
  const uint64_t y = fx_mulhi(f << 5, t.ln2) >> 5;
  uint64_t p = t.c[8];
#ifdef __CUDACC__
#pragma unroll
#endif
  for (int i = 7; i >= 1; --i) p = t.c[i] + fx_mulhi(p, y);
  const uint64_t r = fx_mulhi((1ull << 63) + fx_mulhi(p, y), pow[f >> 59]);  // in [2^62, 2^63)
  return fx_from_bits((uint64_t(uint32_t(k + 1022)) << 52) + ((r + 0x200u) >> 10));
}

}  // namespace gbfem
