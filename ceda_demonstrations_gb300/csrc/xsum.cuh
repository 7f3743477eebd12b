// Exact, order-independent accumulation of doubles (host + device).
//
// Every term x is truncated toward zero to a multiple of 2^-160 and added exactly into
// ten signed 64-bit limbs, limb k carrying 32-bit digits of weight 2^(32k-160). A term
// touches at most three limbs and never propagates a carry, so per-thread accumulators,
// warp shuffles, block trees and global atomics can combine partial sums in any order and
// the total is the same integer. The result is that integer rounded once to the nearest
// double. Terms with |x| >= 2^128 (or inf) set the overflow flag, NaN sets the NaN flag.
// Up to 2^31 terms fit without limb overflow.
//
// This replaces the order-dependent allreduce of the reference's NVECTOR reductions
// (gkeyll_diffusion/src/nvector_gkylzero.c:234-404): the value a reduction returns here is
// independent of the grid shape, the SM count and the kernel that produced the terms.
#pragma once
#include <cstdint>
#include <cstring>

#include "soft64.cuh"

#ifdef __CUDACC__
#define XS_HD __host__ __device__ __forceinline__
#else
#define XS_HD inline
#endif

namespace xsum {

constexpr int NL = 10;
constexpr unsigned FLAG_NAN = 1u, FLAG_OVF = 2u;

struct Limbs {
  long long l[NL];
};

XS_HD void zero(Limbs& a)
{
#pragma unroll
  for (int k = 0; k < NL; ++k) a.l[k] = 0;
}

XS_HD unsigned long long bits_of(double x)
{
#ifdef __CUDA_ARCH__
  return (unsigned long long)__double_as_longlong(x);
#else
  unsigned long long b;
  std::memcpy(&b, &x, 8);
  return b;
#endif
}

XS_HD void add(Limbs& a, double x, unsigned& flags)
{
  unsigned long long b = bits_of(x);
  const bool neg       = (b >> 63) != 0;
  const int e          = (int)((b >> 52) & 0x7ff);
  unsigned long long m = b & ((1ULL << 52) - 1);
  if (e == 0x7ff)
  {
    flags |= m ? FLAG_NAN : FLAG_OVF;
    return;
  }
  int exp2;
  if (e == 0) exp2 = -1074;
  else
  {
    m |= (1ULL << 52);
    exp2 = e - 1075;
  }
  if (exp2 > 75)
  { // |x| >= 2^128
    flags |= FLAG_OVF;
    return;
  }
  int sh = exp2 + 160;
  if (sh < 0)
  {
    m  = (sh <= -64) ? 0ULL : (m >> (-sh));
    sh = 0;
  }
  const int k  = sh >> 5; // 0 .. 7 (sh <= 235)
  const int bs = sh & 31;
  // v = m << bs spans up to 85 bits: digits d0 | d1 | d2
  const unsigned long long lo = m << bs;
  const unsigned long long hi = bs ? (m >> (64 - bs)) : 0ULL;
  long long d0                = (long long)(lo & 0xffffffffULL);
  long long d1                = (long long)(lo >> 32);
  long long d2                = (long long)hi;
  if (neg)
  {
    d0 = -d0;
    d1 = -d1;
    d2 = -d2;
  }
  // three adds into limbs k, k+1, k+2; one branch per term (the terms of one warp usually
  // share k) instead of a select on every limb
  switch (k)
  {
#define XS_CASE(K)                                                                                                   \
  case K:                                                                                                            \
    a.l[K] += d0;                                                                                                    \
    a.l[K + 1] += d1;                                                                                                \
    a.l[K + 2] += d2;                                                                                                \
    break;
    XS_CASE(0)
    XS_CASE(1)
    XS_CASE(2)
    XS_CASE(3)
    XS_CASE(4)
    XS_CASE(5)
    XS_CASE(6)
    XS_CASE(7)
#undef XS_CASE
  default: break;
  }
}

XS_HD void merge(Limbs& a, const Limbs& b)
{
#pragma unroll
  for (int k = 0; k < NL; ++k) a.l[k] += b.l[k];
}

XS_HD double from_bits(unsigned long long b)
{
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)b);
#else
  double x;
  std::memcpy(&x, &b, 8);
  return x;
#endif
}

// Normalise the limbs into a two's-complement integer of 32-bit digits and round it to the
// nearest double (ties to even). Integer arithmetic only, so host and device produce the
// same bits; no array is indexed by a computed value, so the device keeps it in registers (one
// thread runs this at the end of every reduction).
XS_HD double finalize(const long long* limbs, unsigned flags)
{
  if (flags & FLAG_NAN) return from_bits(0x7ff8000000000000ULL);
  if (flags & FLAG_OVF) return from_bits(0x7ff0000000000000ULL);
  constexpr int ND = NL + 1; // digit NL holds the sign extension
  unsigned int dg[ND];
  long long carry = 0;
#pragma unroll
  for (int k = 0; k < NL; ++k)
  {
    const long long v = limbs[k] + carry;
    dg[k]             = (unsigned int)(v & 0xffffffffLL);
    carry             = v >> 32; // arithmetic shift: floor division by 2^32
  }
  const bool negative = carry < 0;
  dg[NL]              = (unsigned int)(carry & 0xffffffffLL);
  if (negative)
  { // magnitude = two's-complement negation
    unsigned long long c = 1;
#pragma unroll
    for (int k = 0; k < ND; ++k)
    {
      const unsigned long long s = (unsigned long long)(unsigned int)(~dg[k]) + c;
      dg[k]                      = (unsigned int)s;
      c                          = s >> 32;
    }
  }
  // the three highest digits from the leading nonzero one, and whether anything lies below
  int top = -1;
  unsigned int w2 = 0, w1 = 0, w0 = 0, below = 0;
#pragma unroll
  for (int k = ND - 1; k >= 0; --k)
  {
    if (top < 0)
    {
      w2  = dg[k];
      top = w2 ? k : -1;
    }
    else if (top - k == 1) w1 = dg[k];
    else if (top - k == 2) w0 = dg[k];
    else below |= dg[k];
  }
  if (top < 0) return 0.0;
  // leading one to bit 63, the rest as a sticky bit
  const int lz               = soft64::leading_zeros(w2);
  const unsigned long long m = ((((unsigned long long)w2 << 32) | w1) << lz) | (((unsigned long long)w0 << lz) >> 32);
  below |= w0 << lz;
  const int e = 1023 - 160 + 32 * top + 31 - lz; // exponent field of the leading one
  return soft64::round_pack(negative ? 0x80000000u : 0u, e, m | (below ? 1u : 0u));
}

} // namespace xsum
