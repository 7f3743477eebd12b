// Compares soft64.cuh with the host's IEEE arithmetic: prints the handled and the wrong results
// of additions, products and fused multiply-adds over seeded operands.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "soft64.cuh"

static double make(uint64_t sign_frac, int e)
{
  e               = e < 0 ? 0 : (e > 2047 ? 2047 : e);
  const uint64_t b = (sign_frac & 0x800fffffffffffffULL) | ((uint64_t)e << 52);
  double x;
  std::memcpy(&x, &b, 8);
  return x;
}

int main(int argc, char** argv)
{
  const long n = argc > 1 ? std::atol(argv[1]) : 1000000;
  std::mt19937_64 r(argc > 2 ? std::strtoull(argv[2], nullptr, 10) : 1);
  long handled[3] = {0, 0, 0}, wrong = 0;
  for (long i = 0; i < n; ++i)
  {
    uint64_t f[3] = {r(), r(), r()};
    // significands with long runs of zeros or ones at the end: ties and carries
    for (int k = 0; k < 3; ++k)
      if ((i >> (2 * k)) & 1)
      {
        const uint64_t low = (1ULL << (r() % 53)) - 1;
        f[k] = ((i >> (2 * k)) & 2) ? (f[k] | low) : (f[k] & ~low);
      }
    const bool any = (i % 5) == 0; // the whole exponent range, its ends among it
    const int ea = any ? (int)(r() % 2048) : 1023 + (int)(r() % 41) - 20;
    const int eb = ea + (int)(r() % 27) - 13;
    const int ec = any && (i & 1) ? (int)(r() % 2048) : ea + eb - 1023 + (int)(r() % 90) - 5;
    const double a = make(f[0], ea), b = make(f[1], eb), c = make(f[2], ec);
    double s;
    auto check = [&](int op, bool ok, double want) {
      if (!ok) return;
      ++handled[op];
      if (soft64::bits(s) != soft64::bits(want) && wrong++ < 5) std::printf("op %d: %a %a %a: %a, not %a\n", op, a, b, c, s, want);
    };
    check(0, soft64::add(a, b, &s), a + b);
    check(1, soft64::mul(soft64::factor(a), b, &s), a * b);
    check(2, soft64::fma_small(soft64::factor(a), b, c, &s), std::fma(a, b, c));
  }
  // conversions: every handled float exactly, doubles around the floats' ties and range ends
  long conv = 0;
  for (long i = 0; i < n; ++i)
  {
    const uint32_t u = (uint32_t)r();
    float x, y;
    std::memcpy(&x, &u, 4);
    double s;
    if (soft64::from_float(x, &s) && ++conv && soft64::bits(s) != soft64::bits((double)x)) ++wrong;
    const uint64_t low[] = {0, 0x10000000u, 0x0fffffffu, 0x10000001u, r() & 0x1fffffffu};
    const double d = make((r() & ~0x1fffffffULL) | low[i % 5], 890 + (int)(r() % 270));
    const float want = (float)d;
    if (soft64::to_float(d, &y) && ++conv && soft64::bits32(y) != soft64::bits32(want)) ++wrong;
  }
  if (conv < n) ++wrong; // most of them are handled
  // operands that no function may take: zeros, subnormals, infinities, NaN
  const double odd[] = {0.0, -0.0, 4.9e-324, -2.2e-308, INFINITY, -INFINITY, NAN};
  double s;
  float g;
  for (double x : odd)
    wrong += soft64::from_float((float)x, &s) + soft64::to_float(x, &g) + soft64::to_float(1e39, &g) +
             soft64::to_float(1e-39, &g) + soft64::add(x, 1.0, &s) + soft64::add(1.0, x, &s) + soft64::add(x, x, &s) +
             soft64::mul(soft64::factor(x), 1.0, &s) + soft64::mul(soft64::factor(1.0), x, &s) +
             soft64::fma_small(soft64::factor(x), 1e-3, 1.0, &s) + soft64::fma_small(soft64::factor(1e-3), x, 1.0, &s) +
             soft64::fma_small(soft64::factor(1e-3), 1.0, x, &s);
  std::printf("handled %ld %ld %ld wrong %ld\n", handled[0], handled[1], handled[2], wrong);
  return wrong != 0;
}
