// Host build of the quotient from a reciprocal (tealeaf_ref_gb300/csrc/tl_fp64emu.cuh), checked against
// the FPU's division on seeded operands: exponents over the whole range (subnormals, zeros, infinities
// and NaNs among them), numerators near the subnormal range, divisors with all-ones and near-zero
// significands and a close to b.  Usage: quotient_host N SEED; prints the mismatch count.
#include "tl_fp64emu.cuh"

#include <cstdio>
#include <cstdlib>
#include <random>

using namespace tl::emu;

int main(int argc, char** argv) {
  const long n = argc > 1 ? atol(argv[1]) : 1000000;
  std::mt19937_64 rng(argc > 2 ? atol(argv[2]) : 1);
  long bad = 0;
  for (long i = 0; i < n; ++i) {
    uint64_t ma = rng(), mb = rng();
    if (i % 4 == 1) mb |= FRAC ^ (rng() & 0xff);
    if (i % 4 == 2) mb &= 0xff;
    if (i % 4 == 3) ma = (ma & 0xffffffffull) | (mb & 0xfffff00000000ull);
    uint64_t ea = rng() % 2048, eb = rng() % 2048;
    if (i & 8) ea = rng() % 400, eb = 290 + rng() % 600;  // small numerators
    if (i & 16) ea = eb > 1000 ? eb : eb + rng() % 60;    // quotients near one
    const double a = from_bits((rng() & SIGN) | ea << 52 | (ma & FRAC)), b = from_bits(eb << 52 | (mb & FRAC));
    const double q = quotient(a, b, 1.0 / b), want = a / b;
    if (bits(q) != bits(want) && !(std::isnan(q) && std::isnan(want))) ++bad;
  }
  printf("mismatch %ld\n", bad);
  return bad != 0;
}
