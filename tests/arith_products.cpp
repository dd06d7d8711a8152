// Host check of the recursions' products against exact 128-bit arithmetic (compiled and run by
// test_arith_products_cpu.py; the host forms run the same reductions as the device's):
//   mulw(a, w)        congruent to a w and at most 2^61 + 2^47 - 1, for any 64-bit a, w < q;
//   mulw_digit(a, w)  the same for any 32-bit a;
//   red60(x)          congruent to x and below 2^60 + 2^18, canon(x) its residue, any x;
//   acc_fold          congruent to the accumulated sum and below 2^60 + 2^37, any 128-bit sum;
//   the transforms' units stay within the bounds their passes state.
#include <cstdio>
#include <cstdlib>

#include "ig_arith.cuh"

using namespace ig;

static u64 rng_state = 0x9E3779B97F4A7C15ULL;
static u64 next() {
  rng_state ^= rng_state << 13;
  rng_state ^= rng_state >> 7;
  rng_state ^= rng_state << 17;
  return rng_state;
}
static u64 mulmod(u64 a, u64 b) { return (u64)((u128)a * b % Q); }
static int fails = 0;
static void fail(const char* what, unsigned long long a, unsigned long long b) {
  if (fails++ < 5) std::printf("FAIL %s: %llx %llx\n", what, a, b);
}

int main(int argc, char** argv) {
  const long n = argc > 1 ? std::atol(argv[1]) : 1000000;
  const u64 PROD = (1ULL << 61) + (1ULL << 47) - 1, TWO = PROD;  // the passes' "2+"
  const u64 edges[] = {0, 1, Q - 1, Q, Q + 1, 2 * Q - 1, (1ULL << 60) - 1, 1ULL << 60, 15 * Q, 0xFFFFFFFFULL,
                       0xFFFFFFFF00000000ULL, ~0ULL, ~0ULL - Q};
  const int ne = sizeof edges / sizeof *edges;
  const u64 wedges[] = {0, 1, Q - 1, Q / 2, 0xFFFFFFFFULL, 0x0FFFFFFF00000000ULL};
  for (long i = 0; i < n; i++) {
    const u64 w = i < 6 * ne ? wedges[i / ne] : next() % Q;
    const u64 a = i < 6 * ne ? edges[i % ne] : next();
    const Tw t = make_tw(w);
    const u64 v = mulw(a, t);
    if (v > PROD || v % Q != mulmod(a % Q, w)) fail("mulw", a, w);
    const u32 d = (u32)(i & 1 ? a : a >> 44);
    const u64 vd = mulw_digit(d, t);
    if (vd > PROD || vd % Q != mulmod(d, w)) fail("mulw_digit", d, w);
    if (red60(a) >= (1ULL << 60) + (1ULL << 18) || red60(a) % Q != a % Q) fail("red60", a, 0);
    if (canon(a) != a % Q) fail("canon", a, 0);
    const u64 nearq = (i % 15 + 1) * Q + (u64)(i % 7) - 3;
    if (canon(nearq) != nearq % Q) fail("canon near a multiple", nearq, 0);

    // Sums: the words of the largest link (two of 15q, one just above q), then any 128 bits.
    Acc s{0, 0, 0, 0};
    u128 want = 0;
    for (int k = 0; k < 4; k++) {
      const u64 x = i == 0 ? 15 * Q : next() % (15 * Q), y = i == 0 ? Q - 1 : next() % Q;
      mac(s, x, y);
      mac(s, y, y);
      want += (u128)x * y + (u128)y * y;
    }
    u64 f = acc_fold(s);
    if (f >= (1ULL << 60) + (1ULL << 37) || f % Q != (u64)(want % Q)) fail("acc_fold", f, 0);
    Acc r{(u32)next(), (u32)next(), (u32)next(), (u32)next()};
    if (i == 1) r = Acc{~0u, ~0u, ~0u, ~0u};
    const u128 rv = ((u128)(((u64)r.r3 << 32) | r.r2) << 64) | (((u64)r.r1 << 32) | r.r0);
    f = acc_fold(r);
    if (f >= (1ULL << 60) + (1ULL << 37) || f % Q != (u64)(rv % Q)) fail("acc_fold any", f, 0);

    // Inverse unit on words up to 2+: no sum passes 64 bits, differences stay positive.
    const bool top = i & 1;
    u64 x[4];
    for (auto& e : x) e = top ? TWO : next() % (TWO + 1);
    if (top) x[i >> 1 & 3] = 0;
    const u128 s01 = (u128)x[0] + x[1], s23 = (u128)x[2] + x[3];
    if ((s01 + s23) >> 64) fail("inverse sum", x[0], x[1]);
    if (x[0] > x[1] + 3 * Q || (u64)s01 > (u64)s23 + 5 * Q) fail("inverse difference", x[0], x[1]);
    if ((u128)x[1] + 3 * (u128)Q >> 64 || s23 + 5 * (u128)Q >> 64) fail("inverse offset", x[0], x[1]);
    // Forward units: a product is at most 3q, and 9q in, or a reduced word in, leaves room for two.
    if (PROD > 3 * Q || (u128)9 * Q + (1 << 21) + 6 * (u128)Q >> 64) fail("forward growth", 0, 0);
  }
  if (fails) return 1;
  std::printf("ok\n");
  return 0;
}
