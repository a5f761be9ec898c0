/* The quotients of the one-launch pressure solve (plume_b200/csrc/cluster_solve.cu, quotient and reciprocal),
 * restated with the same float and double operations, checked against IEEE x / d for divisors spread over the
 * couplings' sums and cell volumes: x of random bit patterns, around each divisor's multiples of halfway points,
 * zeros, infinities and NaN. The reciprocal starts from a float off by up to a few ulps, as the device's
 * approximate one may be. Prints mismatches among normal quotients (and zeros, infinities and NaN), mismatches
 * among subnormal quotients, and the number checked. */
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

static uint64_t state = 0x9e3779b97f4a7c15ull;
static uint32_t next32(void) {
  state ^= state << 13;
  state ^= state >> 7;
  state ^= state << 17;
  return (uint32_t)(state >> 32);
}
static float from_bits(uint32_t b) {
  float x;
  memcpy(&x, &b, 4);
  return x;
}
static uint32_t to_bits(float x) {
  uint32_t b;
  memcpy(&b, &x, 4);
  return b;
}

static double reciprocal(float d, int ulps) {
  const double x = (double)d;
  double y = (double)from_bits(to_bits(1.0f / d) + (uint32_t)ulps);
  y = fma(y, fma(-x, y, 1.0), y);
  return fma(y, fma(-x, y, 1.0), y);
}

static uint64_t bad = 0, bad_subnormal = 0, checked = 0;

static void check(float x, float d, double inv) {
  volatile float vx = x, vd = d;
  const float want = vx / vd, got = (float)((double)x * inv);
  checked++;
  if (to_bits(want) == to_bits(got) || (isnan(want) && isnan(got))) return;
  if (want != 0.0f && fabsf(want) < 0x1p-126f) bad_subnormal++;
  else bad++;
}

int main(void) {
  for (int n = 0; n < 4000; ++n) {
    const float fixed[] = {1.0f, 2.0f, 3.0f, 4.0f, 5.0f, 6.0f, 4.6666665f, 5.3333335f, 6.9411764f, 1.0f / 3.0f};
    const float d = n < 10 ? fixed[n] : from_bits((uint32_t)(110 + next32() % 26) << 23 | (next32() & 0x7fffffu));
    const double inv = reciprocal(d, (int)(next32() % 7) - 3);
    for (int k = 0; k < 20000; ++k) {
      check(from_bits(next32()), d, inv);
      /* near a midpoint between two floats: x = the float nearest d * (m + 1/2 ulp) */
      const float m = from_bits((uint32_t)(60 + next32() % 130) << 23 | (next32() & 0x7fffffu));
      const double half = ((double)m + (double)from_bits(to_bits(m) + 1)) / 2;
      check((float)(half * (double)d), d, inv);
    }
    check(0.0f, d, inv);
    check(-0.0f, d, inv);
    check(INFINITY, d, inv);
    check(-INFINITY, d, inv);
    check(NAN, d, inv);
    check(0x1.fffffep+127f, d, inv);
  }
  printf("%llu %llu %llu\n", (unsigned long long)bad, (unsigned long long)bad_subnormal, (unsigned long long)checked);
  return 0;
}
