// fpi::to_float_rn against the host's conversion: random bit patterns, values
// around every float rounding boundary and the ends of the float range.
#include <cstdio>
#include "../../sdem_gb300/csrc/fp64_int.cuh"

static uint64_t state = 88172645463325252ull;
static uint64_t next() {
  state ^= state << 13; state ^= state >> 7; state ^= state << 17;
  return state;
}
static long bad = 0;
static void check(uint64_t u) {
  const double x = fpi::from_bits(u);
  const float want = (float)x, got = fpi::to_float_rn(x);
  if (want != want ? got == got : fpi::fbits(want) != fpi::fbits(got)) {
    if (bad++ < 5) std::printf("%016llx: %08x, not %08x\n", (unsigned long long)u, fpi::fbits(got), fpi::fbits(want));
  }
}
int main() {
  for (long i = 0; i < 20000000; i++) check(next());
  for (long i = 0; i < 20000000; i++) {   // float range; ties and their neighbours
    const uint64_t e = 860 + next() % 320, m = next() & fpi::kMant;
    const uint64_t u = (next() & fpi::kSign) | e << 52 | m;
    check(u);
    const uint64_t tie = (u & ~0x1FFFFFFFull) | 0x10000000ull;
    check(tie); check(tie - 1); check(tie + 1); check(u | 0x1FFFFFFFull); check(u & ~0x1FFFFFFFull);
  }
  const uint64_t ends[] = {0, fpi::kSign, 0x7FF0000000000000ull, 0x7FF8000000000000ull, 1, 0x47EFFFFFE0000000ull,
                           0x47EFFFFFF0000000ull, 0x47EFFFFFEFFFFFFFull, 0x3810000000000000ull, 0x380FFFFFFFFFFFFFull};
  for (uint64_t u : ends) { check(u); check(u ^ fpi::kSign); }
  std::printf("%ld mismatches\n", bad);
  return bad != 0;
}
