// IEEE double addition, multiplication and fused multiply-add (round to nearest even) on the
// integer pipes.
//
// GB300 issues FP64 instructions at 1.6 lanes per clock and SM (5.0e11 per second measured;
// conversions 5.9e11, comparisons 5.0e11), so the FP64 kernels of this library are bounded by
// their FP64 instruction count while most issue slots stay empty. The functions below compute
// some of such a kernel's operations from 32- and 64-bit integer instructions (about 30 for an
// addition, 40 for a product, 50 for a fused multiply-add), beside the FP64 instructions that
// remain. Where they report true the result is the correctly rounded one, bit for bit; operands
// outside the ranges that each one names (zeros, subnormal numbers, infinities, NaN, results
// near the ends of the exponent range, sums with cancellation) report false, the value is then
// meaningless, and the caller (s64_add, s64_mul, ... below) branches to the hardware's instruction,
// operation by operation: where the ranges hold in a whole warp no FP64 instruction is issued, a
// predicated one would still take its slot of the pipe.
#pragma once
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define S64_HD __host__ __device__ __forceinline__
#else
#define S64_HD inline
#endif

namespace soft64 {

S64_HD uint64_t bits(double x)
{
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t b;
  std::memcpy(&b, &x, 8);
  return b;
#endif
}

S64_HD double value(uint32_t hi, uint32_t lo)
{
#ifdef __CUDA_ARCH__
  return __hiloint2double((int)hi, (int)lo);
#else
  const uint64_t b = ((uint64_t)hi << 32) | lo;
  double x;
  std::memcpy(&x, &b, 8);
  return x;
#endif
}

S64_HD int leading_zeros(uint32_t x)
{
#ifdef __CUDA_ARCH__
  return __clz((int)x);
#else
  return x ? __builtin_clz(x) : 32;
#endif
}

// a factor taken apart once: significand with the leading one at bit 63, exponent field, sign.
// A factor that is not a normal number gets an exponent that no range test below accepts.
struct Factor {
  uint64_t m;
  int e;
  uint32_t h; // high word (its sign bit is used)
};

S64_HD Factor factor(double x)
{
  const uint64_t X = bits(x);
  Factor f;
  f.h = (uint32_t)(X >> 32);
  f.e = (int)((f.h >> 20) & 0x7ffu);
  f.m = ((X & 0x000fffffffffffffULL) | 0x0010000000000000ULL) << 11;
  if ((unsigned)(f.e - 1) > 2045u) f.e = 1 << 20;
  return f;
}

// sign (bit 31), exponent field e of the leading one at bit 63 of m, 64-bit significand m with
// a sticky bit 0: rounded to 53 bits, ties to even. A carry out of the significand moves to the
// exponent (m = 2^64 counts twice the leading one).
S64_HD double round_pack(uint32_t sign, int e, uint64_t m)
{
  const uint64_t r     = m + 0x3ffu + (((uint32_t)m >> 11) & 1u);
  const uint32_t carry = r < m ? 1u : 0u;
  const uint64_t q     = r >> 11; // with the leading one at bit 52
  const uint32_t hi    = (uint32_t)(q >> 32) + ((uint32_t)(e - 1) << 20) + (carry << 21);
  return value(hi | (sign & 0x80000000u), (uint32_t)q);
}

// high 64 bits of a product of two 64-bit significands, with a nonzero low half kept in *rest
S64_HD uint64_t mul_high(uint64_t a, uint64_t b, uint32_t* mid, uint32_t* low)
{
  const uint32_t a0 = (uint32_t)a, a1 = (uint32_t)(a >> 32), b0 = (uint32_t)b, b1 = (uint32_t)(b >> 32);
  const uint64_t t0 = (uint64_t)a0 * b0;
  const uint64_t t1 = (uint64_t)a1 * b0 + (uint32_t)(t0 >> 32);
  const uint64_t t2 = (uint64_t)a0 * b1 + (uint32_t)t1;
  *mid              = (uint32_t)t2; // bits 32 .. 63
  *low              = (uint32_t)t0; // bits 0 .. 31
  return (uint64_t)a1 * b1 + (uint32_t)(t1 >> 32) + (uint32_t)(t2 >> 32);
}

// a + b: normal operands of one sign whose exponents differ by at most 10
S64_HD bool add(double a, double b, double* s)
{
  const uint64_t A = bits(a), B = bits(b);
  const uint32_t ah = (uint32_t)(A >> 32), bh = (uint32_t)(B >> 32);
  const int ea = (int)((ah >> 20) & 0x7ffu), eb = (int)((bh >> 20) & 0x7ffu);
  const int d  = ea - eb;
  if ((int32_t)(ah ^ bh) < 0 || (unsigned)(d + 10) > 20u || (unsigned)(ea - 11) > 2020u) return false;
  // significands with the leading one at bit 62: the 10 bits below the last place hold the
  // shifted part, nothing is lost
  const uint64_t ma = ((A & 0x000fffffffffffffULL) | 0x0010000000000000ULL) << 10;
  const uint64_t mb = ((B & 0x000fffffffffffffULL) | 0x0010000000000000ULL) << 10;
  const int da = d < 0 ? -d : 0, db = d > 0 ? d : 0;
  const uint64_t m = (ma >> da) + (mb >> db); // leading one at bit 62 or 63
  const int up     = (int)((uint32_t)(~(uint32_t)(m >> 32)) >> 31);
  *s               = round_pack(ah, ea + da + 1 - up, m << up);
  return true;
}

// f * b: normal operands, normal product
S64_HD bool mul(const Factor& f, double b, double* p)
{
  const uint64_t B  = bits(b);
  const uint32_t bh = (uint32_t)(B >> 32);
  const int eb      = (int)((bh >> 20) & 0x7ffu);
  const int e       = f.e + eb - 1022; // exponent field of bit 127 of the product
  if ((unsigned)(eb - 1) > 2045u || (unsigned)(e - 3) > 2040u) return false;
  const uint64_t mb = ((B & 0x000fffffffffffffULL) | 0x0010000000000000ULL) << 11;
  uint32_t mid, low;
  uint64_t m   = mul_high(f.m, mb, &mid, &low);
  const int up = (int)((uint32_t)(~(uint32_t)(m >> 32)) >> 31);
  m            = (m << up) | ((mid >> 31) & (uint32_t)up);
  m |= ((mid << up) | low) ? 1u : 0u;
  *p = round_pack(f.h ^ bh, e - up, m);
  return true;
}

// fma(f, b, c): normal operands with |f b| < |c| / 2 (exponents at least three apart)
S64_HD bool fma_small(const Factor& f, double b, double c, double* r)
{
  const uint64_t B = bits(b), C = bits(c);
  const uint32_t bh = (uint32_t)(B >> 32), ch = (uint32_t)(C >> 32);
  const int eb = (int)((bh >> 20) & 0x7ffu), ec = (int)((ch >> 20) & 0x7ffu);
  const int d   = ec + 1023 - (f.e + eb); // bit 63 of the product's significand relative to c's
  if (d < 3 || (unsigned)(eb - 1) > 2045u || (unsigned)(ec - 8) > 2030u) return false;
  const uint64_t mb = ((B & 0x000fffffffffffffULL) | 0x0010000000000000ULL) << 11;
  const uint64_t mc = ((C & 0x000fffffffffffffULL) | 0x0010000000000000ULL) << 10; // leading one at bit 62
  uint32_t mid, low;
  const uint64_t m = mul_high(f.m, mb, &mid, &low);
  // aligned to c and rounded to odd: a nonzero part below bit 0 is kept as a set bit 0
  const int sh        = d > 63 ? 63 : d;
  const uint64_t out  = m << (64 - sh);
  const uint32_t rest = mid | low | (uint32_t)out | (uint32_t)(out >> 32);
  const uint64_t p    = (m >> sh) | (rest ? 1u : 0u);
  const uint64_t s    = (int32_t)(f.h ^ bh ^ ch) < 0 ? mc - p : mc + p; // leading one at bit 61 .. 63
  const int n         = leading_zeros((uint32_t)(s >> 32));
  *r                  = round_pack(ch, ec + 1 - n, s << n);
  return true;
}

S64_HD uint32_t bits32(float x)
{
#ifdef __CUDA_ARCH__
  return (uint32_t)__float_as_int(x);
#else
  uint32_t b;
  std::memcpy(&b, &x, 4);
  return b;
#endif
}

// (double)x: a normal x
S64_HD bool from_float(float x, double* d)
{
  const uint32_t b = bits32(x);
  if (((b >> 23) & 0xffu) - 1u > 253u) return false;
  *d = value((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + (896u << 20)), b << 29);
  return true;
}

// (float)x, ties to even: x in the float format's normal range (a round up past it gives
// infinity, as the conversion does)
S64_HD bool to_float(double x, float* f)
{
  const uint64_t B  = bits(x);
  const uint32_t hi = (uint32_t)(B >> 32), lo = (uint32_t)B;
  if (((hi >> 20) & 0x7ffu) - 897u > 253u) return false;
  uint32_t v = (((hi & 0x7fffffffu) - (896u << 20)) << 3) | (lo >> 29);
  v += ((lo & 0x1fffffffu) + 0x0fffffffu + (v & 1u)) >> 29;
  v |= hi & 0x80000000u;
#ifdef __CUDA_ARCH__
  *f = __int_as_float((int)v);
#else
  std::memcpy(f, &v, 4);
#endif
  return true;
}

} // namespace soft64

#ifdef __CUDACC__
// the same with the hardware's instruction where the integer form does not apply
__device__ __forceinline__ double s64_add(double a, double b)
{
  double s;
  if (soft64::add(a, b, &s)) return s;
  return __dadd_rn(a, b);
}
__device__ __forceinline__ double s64_mul(const soft64::Factor& f, double a, double b)
{
  double p;
  if (soft64::mul(f, b, &p)) return p;
  return __dmul_rn(a, b);
}
__device__ __forceinline__ double s64_mul(double a, double b) { return s64_mul(soft64::factor(a), a, b); }
__device__ __forceinline__ double s64_fma_small(const soft64::Factor& f, double a, double b, double c)
{
  double r;
  if (soft64::fma_small(f, b, c, &r)) return r;
  return __fma_rn(a, b, c);
}
__device__ __forceinline__ double s64_fma_small(double a, double b, double c)
{
  return s64_fma_small(soft64::factor(a), a, b, c);
}
__device__ __forceinline__ double s64_from_float(float x)
{
  double d;
  if (soft64::from_float(x, &d)) return d;
  return (double)x;
}
__device__ __forceinline__ float s64_to_float(double x)
{
  float f;
  if (soft64::to_float(x, &f)) return f;
  return __double2float_rn(x);
}
// SOFT false: the FP64 instruction (kernels that latency bounds, see their rules)
template <bool SOFT>
__device__ __forceinline__ double s64_add(double a, double b)
{
  return SOFT ? s64_add(a, b) : __dadd_rn(a, b);
}
template <bool SOFT>
__device__ __forceinline__ double s64_mul(const soft64::Factor& f, double a, double b)
{
  return SOFT ? s64_mul(f, a, b) : __dmul_rn(a, b);
}
template <bool SOFT>
__device__ __forceinline__ double s64_mul(double a, double b)
{
  return SOFT ? s64_mul(a, b) : __dmul_rn(a, b);
}
template <bool SOFT>
__device__ __forceinline__ double s64_fma_small(const soft64::Factor& f, double a, double b, double c)
{
  return SOFT ? s64_fma_small(f, a, b, c) : __fma_rn(a, b, c);
}
#endif
