// The system-matrix kernels' quotient (div_rcp in csrc/kernels_sm.cu): one
// correction of the product with the rounded reciprocal, against the division.
// Random significands, and those next to powers of two, to each other and to the
// extremes.  Prints the number of pairs that differ.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>

static float of(uint32_t bits) {
  float f;
  std::memcpy(&f, &bits, 4);
  return f;
}

static long check(uint32_t ma, uint32_t mb, int ea, int eb) {
  const float a = of((uint32_t(127 + ea) << 23) | (ma & 0x7fffff)), b = of((uint32_t(127 + eb) << 23) | (mb & 0x7fffff));
  const float y = 1.0f / b, q = a * y;
  const float r = std::fmaf(-q, b, a);
  return std::fmaf(r, y, q) != a / b;
}

int main() {
  uint64_t s = 0x9e3779b97f4a7c15ull;
  auto rnd = [&] {
    s ^= s << 13;
    s ^= s >> 7;
    s ^= s << 17;
    return uint32_t(s >> 20);
  };
  long wrong = 0;
  for (int i = 0; i < (1 << 24); i++) wrong += check(rnd(), rnd(), int(rnd() % 60) - 30, int(rnd() % 60) - 30);
  for (uint32_t near = 0; near < 2048; near++)
    for (int i = 0; i < 512; i++) {
      const uint32_t m = rnd();
      wrong += check(m, near, 0, 0) + check(m, 0x7fffff - near, 0, 0);          // b next to a power of two
      wrong += check(near, m, 0, 0) + check(0x7fffff - near, m, 0, 0);          // a next to one
      wrong += check(m, m + near, 0, 0) + check(m, m - near, 0, 0);             // a next to b
    }
  std::printf("%ld\n", wrong);
  return 0;
}
