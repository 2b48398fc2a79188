// Host build of fpconv::split_a checked against the FP64 arithmetic it
// stands for: random entries of every magnitude, entries at and next to the
// midpoints of the 64-grid and of both fp16 roundings, the clamp, special
// values.  Prints "ok <count>" or the first mismatch.
#include <stdint.h>
#include <stdio.h>
#include <cmath>
#include <random>

#include "fpconv.cuh"

using namespace lime::fpconv;

static uint16_t hb(__half h) { return __half_as_ushort(h); }
static bool same(uint16_t a, uint16_t b, bool zeros) {
  return a == b || (zeros && !((a | b) & 0x7fff));
}

static int check(double x) {
  float v0;
  __half h1, h2;
  split_a(x, v0, h1, h2);
  const double kq = std::fmin(std::fmax(std::rint(x * (1.0 / 64.0)), -127.0), 127.0);
  const double r1 = x - kq * 64.0;
  const __half e1 = __double2half(r1);
  const __half e2 = __double2half(r1 - (double)__half2float(e1));
  if (std::isnan(x) || std::isinf(x)) return std::isfinite(__half2float(h1)) ? 1 : 0;
  if (bits32(v0) != bits32((float)(kq * 64.0)) || !same(hb(h1), hb(e1), false) || !same(hb(h2), hb(e2), true)) {
    printf("mismatch x=%.17g (%016llx): %g %04x %04x, expected %g %04x %04x\n", x, (unsigned long long)bits64(x), v0,
           hb(h1), hb(h2), kq * 64.0, hb(e1), hb(e2));
    return 1;
  }
  return 0;
}

int main() {
  std::mt19937_64 g(7);
  long count = 0;
  for (int i = 0; i < 4000000; ++i, ++count) {
    const uint64_t m = g();
    double x = from_bits64((m & 0x800FFFFFFFFFFFFFull) | ((uint64_t)(1023 - 30 + g() % 43) << 52));
    const int kind = i % 5;
    if (kind) {
      // 64 k + an odd multiple of a power of two (the midpoints), moved by a few last places or a tiny amount
      const double k = 64.0 * ((int)(g() % 257) - 128);
      const double q = std::ldexp((double)(2 * (g() % 4096) + 1), -(int)(g() % 26));
      x = k + (m >> 63 ? -q : q);
      if (kind >= 2) x += std::ldexp((double)(2 * (g() % 2048) + 1), -26 + (int)(g() % 12)) * (m & 1 ? 1 : -1);
      if (kind >= 3) x = from_bits64(bits64(x) + (int64_t)(g() % 9) - 4);
      if (kind == 4) x += std::ldexp(1.0, -20 - (int)(g() % 30)) * (m & 2 ? 1 : -1);
      if (!(std::fabs(x) < 8192.0)) continue;
    }
    if (check(x)) return 1;
  }
  const double special[] = {0.0, -0.0, 32.0, -32.0, 96.0, 8191.999999999999, -8191.999999999999, 8128.0, 8160.0,
                            0x1p-25, -0x1p-25, 0x1.8p-25, 0x1p-24, 0x1.8p-24, 0x1p-26, 4.9e-324, -1e-310, 0x1p-14,
                            0x1.ffffffffffffep-15, INFINITY, -INFINITY, NAN};
  for (double x : special) {
    if (check(x)) return 1;
    ++count;
  }
  printf("ok %ld\n", count);
  return 0;
}
