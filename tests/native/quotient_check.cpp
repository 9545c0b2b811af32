// refined_quotient against the division of IEEE 754, with reciprocals that are off by a unit either way.
#include "quotient.cuh"
#include <cstdint>
#include <cstdio>
#include <cstring>

static uint32_t bits(float f) { uint32_t u; std::memcpy(&u, &f, 4); return u; }

int main() {
  uint64_t s = 88172645463325252ull;
  auto next = [&] { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return static_cast<uint32_t>(s >> 16); };
  long wrong = 0, small_wrong = 0, n = 0;
  double worst = 0;
  auto check = [&](float x, float d) {
    const float want = x / d, r0 = 1.f / d;
    const float rs[3] = {r0, nextafterf(r0, 0.f), nextafterf(r0, 2.f)};
    for (float r : rs) {
      const float got = blitz::refined_quotient(x, d, r);
      ++n;
      if (bits(got) == bits(want)) continue;
      if (want != 0.f && fabsf(want) < 0x1p-100f) {
        ++small_wrong;
        const double off = fabs((double)got - (double)want) / fabs((double)want);
        if (fabsf(want) >= 0x1p-126f && off > worst) worst = off;
        continue;
      }
      if (++wrong < 10) std::printf("%a / %a: %a, not %a\n", x, d, got, want);
    }
  };
  // what SiLU divides: x / (1 + e^-x)
  for (int i = 0; i < 1500000; ++i) {
    const float u = static_cast<float>(next()) * 0x1p-32f;
    const float x = (i & 1 ? 174.f : 12.f) * (u - 0.5f);
    check(x, 1.f + expf(-x));
  }
  // any numerator and denominator of the range
  for (int i = 0; i < 500000; ++i) {
    uint32_t a = next(), b = next();
    float x, d;
    std::memcpy(&x, &a, 4);
    b = 0x3f800000u + b % (0x7e3c0000u - 0x3f800000u);
    std::memcpy(&d, &b, 4);
    if (fabsf(x) < 8e37f && d < 8e37f) check(x, d);
  }
  const float zeros[] = {0.f, -0.f, 1e-45f, -1e-45f};
  for (float x : zeros) check(x, 2.f);
  check(0.f, 1.f);
  check(-0.f, 1.f);
  std::printf("%ld quotients, %ld differ, %ld of those below 2^-100 (normal ones by at most %g)\n", n, wrong, small_wrong, worst);
  return wrong != 0 || worst > 0x1p-22;
}
