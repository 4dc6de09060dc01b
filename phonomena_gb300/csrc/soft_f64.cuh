// IEEE FP64 multiply and divide by a known operand in integer arithmetic.
//
// GB300 issues an FP64 instruction at 1/64 of the FP32 and integer rate, so
// the leapfrog (about 105 FP64 operations a node, 48 of them for divisions by
// mesh spacings and 15 multiplications by material constants) is bound by the
// FP64 pipe while the other pipes idle.  The functions here move those
// multiplications and divisions to the integer pipe: about 20 integer
// instructions each in place of one or two FP64 ones, with the same bits.
//
// The known operand (a spacing, a stiffness, dt^2/rho) is held as a record:
// a 64-bit left-aligned significand F (of 1/b for a divisor b, of c for a
// factor c) and the exponent it adds.  With M the 64-bit left-aligned
// significand of x, Q = floor-ish(M * F / 2^64) holds the 53 result bits and
// 10 or 11 more.  Q is below the exact value by less than 4 units (F of a
// divisor is truncated: 1; the low partial product is left out: 1; two
// partial products are truncated: 2), 8 after the one-bit normalisation, so
// the result bits follow from Q unless its low 11 bits lie in [1016, 1024]
// (the rounding midpoint is 1024) or Q is about to carry into the next
// binade.  In those cases (0.5% of operands) the exact product, or the sign
// of the exact remainder against the midpoint, decides.  Operands outside
// the exponent range in which nothing can overflow or turn subnormal, and
// zero factors, go to the FP64 operations themselves.
#pragma once
#include <cstdint>
#include <cstring>
#include <cmath>

#ifdef __CUDACC__
#define SOFT_HD __host__ __device__ __forceinline__
#else
#define SOFT_HD inline
#endif

namespace phono {

// known operand: divisor or factor.  hi has its top bit set, except for
// records the integer path must not take (zero factors, exponents out of
// range), where hi = lo = 0.  de: what the operand adds to the sign/exponent
// word of x when Q has its top bit set (one less in the exponent otherwise), and
// SOFT_BIAS, which keeps its exponent positive and its top bit the sign;
// idx: the operand itself at vals[idx].
struct alignas(16) SoftRec {
  uint32_t lo, hi, de, idx;
};

// a nonzero x taken apart: left-aligned 64-bit significand (top bit set), sign
// and exponent word
struct SoftNum {
  uint32_t hi, lo, se;
};

SOFT_HD uint32_t soft_mulhi(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
  return __umulhi(a, b);
#else
  return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
SOFT_HD uint64_t soft_bits(double x) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t u;
  std::memcpy(&u, &x, 8);
  return u;
#endif
}
SOFT_HD double soft_double(uint32_t hi, uint32_t lo) {
#ifdef __CUDA_ARCH__
  return __hiloint2double((int)hi, (int)lo);
#else
  uint64_t u = ((uint64_t)hi << 32) | lo;
  double x;
  std::memcpy(&x, &u, 8);
  return x;
#endif
}

// biased exponents the integer path takes, 2^-723..2^677: a record moves the
// exponent by at most 129, a factor and a divisor by 258, so every result is
// normal
constexpr uint32_t SOFT_EXP_MIN = 300, SOFT_EXP_SPAN = 1400;
constexpr int SOFT_REC_EXP = 128;
constexpr uint32_t SOFT_BIAS = 2u * SOFT_REC_EXP << 20;

SOFT_HD SoftNum soft_split(double x, bool& ok) {
  const uint64_t u = soft_bits(x);
  const uint32_t xh = (uint32_t)(u >> 32), xl = (uint32_t)u;
  SoftNum n;
  n.hi = (xh << 11) | (xl >> 21) | 0x80000000u;
  n.lo = xl << 11;
  n.se = xh & 0xfff00000u;
  ok = xh * 2u - (SOFT_EXP_MIN << 21) <= ((SOFT_EXP_SPAN << 21) | 0x1fffffu);  // a multiply-add and a compare
  return n;
}

// Q before normalisation (see above): never above the exact value
SOFT_HD uint64_t soft_core(uint32_t mh, uint32_t ml, uint32_t fh, uint32_t fl) {
  return (uint64_t)mh * fh + soft_mulhi(mh, fl) + soft_mulhi(ml, fh);
}

// exact significand product of x and a factor, rounded to nearest even:
// left-aligned, `up` = it is in [2, 4)
SOFT_HD uint64_t soft_mul_exact(uint32_t mh, uint32_t ml, uint32_t fh, uint32_t fl, bool& up) {
  const uint64_t p00 = (uint64_t)ml * fl, p01 = (uint64_t)ml * fh, p10 = (uint64_t)mh * fl;
  const uint64_t mid = (p00 >> 32) + (uint32_t)p01 + (uint32_t)p10;
  uint64_t h = (uint64_t)mh * fh + (p01 >> 32) + (p10 >> 32) + (mid >> 32);
  uint64_t l = (mid << 32) | (uint32_t)p00;
  up = (int64_t)h < 0;
  if (!up) {
    h = (h << 1) | (l >> 63);
    l <<= 1;
  }
  const uint32_t f = (uint32_t)h & 0x7ffu;
  h &= ~(uint64_t)0x7ff;
  if (f > 0x400u || (f == 0x400u && (l != 0 || (h & 0x800u)))) {
    h += 0x800u;
    if (h == 0) {  // 1.11..1 rounded up to 2: only the lower binade can (the upper ends at 4 - 2^-51)
      h = 1ull << 63;
      up = true;
    }
  }
  return h;
}

// quotient of x's significand by b's, rounded to nearest, from the truncated
// quotient q of soft_core: the sign of 2 N - (2 q0 + 1) B with N the shifted
// significand of x (the difference fits in 64 bits; a tie cannot occur)
SOFT_HD uint64_t soft_div_exact(uint32_t mh, uint32_t ml, uint64_t q, double b, bool& up) {
  const uint64_t m = (((uint64_t)mh << 32) | ml) >> 11;
  const uint64_t B = (soft_bits(b) & ((1ull << 52) - 1)) | (1ull << 52);
  up = m >= B;
  const uint64_t q0 = (up ? q : q << 1) >> 11;
  const int64_t d = (int64_t)((m << (up ? 53 : 54)) - (2 * q0 + 1) * B);
  return (q0 + (d > 0 ? 1 : 0)) << 11;
}

SOFT_HD bool soft_ambiguous(uint64_t q) {
  return ((uint32_t)q & 0x7ffu) - 1016u <= 8u || (uint32_t)(q >> 32) == 0xffffffffu;
}

// x * c for a factor record with its top bit set; x inside the range
SOFT_HD SoftNum soft_mul(const SoftNum& x, const SoftRec& c) {
  uint64_t q = soft_core(x.hi, x.lo, c.hi, c.lo);
  bool up = (int64_t)q < 0;
  if (!up) q += q;
  uint64_t r = (q + 0x400u) & ~(uint64_t)0x7ff;
  if (soft_ambiguous(q)) r = soft_mul_exact(x.hi, x.lo, c.hi, c.lo, up);
  SoftNum n;
  n.hi = (uint32_t)(r >> 32);
  n.lo = (uint32_t)r;
  n.se = x.se + c.de - (up ? SOFT_BIAS : SOFT_BIAS + (1u << 20));
  return n;
}

// x / b for a divisor record with its top bit set (b: its value, read only
// where the rounding is in doubt)
template <class B>
SOFT_HD SoftNum soft_div(const SoftNum& x, const SoftRec& d, B b) {
  const uint64_t q1 = soft_core(x.hi, x.lo, d.hi, d.lo);
  bool up = (int64_t)q1 < 0;
  const uint64_t q = up ? q1 : q1 + q1;
  uint64_t r = (q + 0x400u) & ~(uint64_t)0x7ff;
  if (soft_ambiguous(q)) r = soft_div_exact(x.hi, x.lo, q1, b(), up);
  SoftNum n;
  n.hi = (uint32_t)(r >> 32);
  n.lo = (uint32_t)r;
  n.se = x.se + d.de - (up ? SOFT_BIAS : SOFT_BIAS + (1u << 20));
  return n;
}

SOFT_HD double soft_join(const SoftNum& n) {
  return soft_double(((n.hi >> 11) & 0xfffffu) | n.se, (n.lo >> 11) | (n.hi << 21));
}

// the sign of a record's operand, in the top bit
SOFT_HD uint32_t soft_sign(const SoftRec& c) { return c.de; }

// record of a divisor (div) or factor; idx: where the kernels find its value
inline SoftRec soft_record(double v, bool div, uint32_t idx) {
  SoftRec r{0, 0, 0, idx};
  const uint64_t u = soft_bits(v);
  const uint32_t sign = (uint32_t)(u >> 63) << 31;
  const int ex = (int)((u >> 52) & 0x7ff);
  r.de = sign;
  if (ex < 1023 - SOFT_REC_EXP || ex > 1023 + SOFT_REC_EXP || (div && sign)) return r;  // zero, subnormal, extreme: FP64 path
  const uint64_t m = (u & ((1ull << 52) - 1)) | (1ull << 52);
  uint64_t f;
  if (div) {
    const unsigned __int128 q = ((unsigned __int128)1 << 116) / m;  // 2^64 * 2^52 / m, in (2^63, 2^64]
    f = q >> 64 ? ~0ull : (uint64_t)q;
    r.de = SOFT_BIAS + ((uint32_t)(1023 - ex) << 20);
  } else {
    f = m << 11;
    r.de = SOFT_BIAS + sign + ((uint32_t)(ex - 1022) << 20);
  }
  r.hi = (uint32_t)(f >> 32);
  r.lo = (uint32_t)f;
  return r;
}

}  // namespace phono
