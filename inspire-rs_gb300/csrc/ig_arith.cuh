// Exact arithmetic shared by the device kernels and the host-side set-up code.
//
// Modulus: q = 2^60 - 2^14 + 1 (DEFAULT_Q of the reference, src/math/mod_q.rs:7), the
// only ciphertext modulus of the d2048 parameter sets the respond path serves.
//
// Three exact product forms are used:
//   * by a fixed factor w held as a Tw (w and w 2^32 mod q): transform twiddles and scalar
//     constants (mulw), left in [0, 2q + 2^47).
//   * sums of full products folded at 2^60 (Acc): the recursions' products of two values
//     in standard form, left in [0, q + 2^37).
//   * Montgomery (a * b * 2^-64 mod q, canonical): products of a value in standard form with
//     an operand stored pre-multiplied by 2^64 ("R-form").
// In R-form: the packing store, the client's secret, NoPacking's query and the Galois keys until they
// are folded. In standard form, scaled once: the key rows of masks and seats (k_key_rows), the
// folded Galois keys and, in the links, `a`, whose factor takes a store word's 2^-64.
// NTT-domain values that vary per query stay in standard form.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define IG_HD __host__ __device__ __forceinline__
#else
#define IG_HD inline
#endif

namespace ig {

typedef uint64_t u64;
typedef uint32_t u32;
typedef unsigned __int128 u128;
typedef int64_t i64;

static constexpr u64 Q = 1152921504606830593ULL;  // 2^60 - 2^14 + 1
// -q^-1 mod 2^64
static constexpr u64 QINV_NEG = []() constexpr {
  u64 y = 1;
  for (int i = 1; i < 64; i++) y |= (y * Q) & (1ULL << i);
  return (u64)0 - y;
}();

IG_HD u64 mulhi(u64 a, u64 b) {
#ifdef __CUDA_ARCH__
  return __umul64hi(a, b);
#else
  return (u64)(((u128)a * b) >> 64);
#endif
}

IG_HD u64 csub(u64 x) { return x >= Q ? x - Q : x; }
IG_HD u64 addq(u64 a, u64 b) { return csub(a + b); }
IG_HD u64 subq(u64 a, u64 b) { return a >= b ? a - b : a + Q - b; }
IG_HD u64 negq(u64 a) { return a == 0 ? 0 : Q - a; }

// a * b * 2^-64 mod q for a, b < q.
IG_HD u64 mont(u64 a, u64 b) {
  u64 lo = a * b;
  u64 hi = mulhi(a, b);
  u64 m = lo * QINV_NEG;
  // (a*b + m*q) / 2^64; the low halves sum to 0 mod 2^64, carrying 1 unless both are 0.
  u64 t = hi + mulhi(m, Q) + (lo != 0 ? 1 : 0);
  return csub(t);
}

IG_HD u128 wide(u64 a, u64 b) { return (u128)a * b; }

// c + a * b with the 64-bit accumulation inside the wide multiply. nvcc splits mad.wide.u32 into
// a multiply and a 64-bit add; the lo/hi pair with a carry stays one instruction (a register
// probe: 4.3 against 5.3 cycles a warp, 1.4 against 2.6 instructions).
IG_HD u64 mad_wide(u32 a, u32 b, u64 c) {
#ifdef __CUDA_ARCH__
  u32 l = (u32)c, h = (u32)(c >> 32);
  asm("mad.lo.cc.u32 %0,%2,%3,%0; madc.hi.u32 %1,%2,%3,%1;" : "+r"(l), "+r"(h) : "r"(a), "r"(b));
  return ((u64)h << 32) | l;
#else
  return (u64)a * b + c;
#endif
}

// A fixed factor w < q as 32-bit words, w = h 2^32 + l, beside w2 = w 2^32 mod q.
struct alignas(16) Tw {
  u32 l, h, l2, h2;
};
static constexpr u64 MASK60 = (1ULL << 60) - 1, MASK61 = (1ULL << 61) - 1;
inline Tw make_tw(u64 w) {  // host
  const u64 w2 = (u64)(((u128)w << 32) % Q);
  return Tw{(u32)w, (u32)(w >> 32), (u32)w2, (u32)(w2 >> 32)};
}

// a * w mod q in [0, 2^61 + 2^47), just above 2q, for any 64-bit a. With a = ah 2^32 + al,
// P = al w + ah w2 is below 2^93 and congruent to a w: w2 takes the place of half of the full
// product. 2^61 = 2 (2^14 - 1) mod q, so the 32 bits above bit 61 come back as one more wide
// multiply. Five wide multiplies (20 cycles a warp of the heavy pipe), where a Shoup product takes
// three wide, two high and four low ones (28), and no companion word: a register-only butterfly
// takes 28 to 31 cycles a warp instead of 45.
IG_HD u64 mulw(u64 a, const Tw& t) {
  const u32 ah = (u32)(a >> 32), al = (u32)a;
#ifdef __CUDA_ARCH__
  u32 p0, p1, p2;
  asm("{.reg .u32 b0, b1; .reg .u64 A, B;\n"
      " mul.wide.u32 A, %3, %5; mov.b64 {%0, %1}, A;\n"
      " mul.wide.u32 B, %3, %6; mov.b64 {b0, b1}, B;\n"
      " mad.lo.cc.u32 b0, %4, %8, b0; madc.hi.u32 b1, %4, %8, b1;\n"
      " mad.lo.cc.u32 %0, %4, %7, %0; madc.hi.cc.u32 %1, %4, %7, %1; addc.u32 b1, b1, 0;\n"
      " add.cc.u32 %1, %1, b0; addc.u32 %2, b1, 0;}"
      : "=&r"(p0), "=&r"(p1), "=&r"(p2)
      : "r"(al), "r"(ah), "r"(t.l), "r"(t.h), "r"(t.l2), "r"(t.h2));
  return mad_wide(__funnelshift_l(p1, p2, 3), 32766u, ((u64)(p1 & 0x1fffffffu) << 32) | p0);
#else
  const u64 w = ((u64)t.h << 32) | t.l, w2 = ((u64)t.h2 << 32) | t.l2;
  const u128 P = (u128)al * w + (u128)ah * w2;
  return (u64)(P & MASK61) + (u64)(u32)(P >> 61) * 32766u;
#endif
}

// The same for a 32-bit a (a gadget digit): three wide multiplies.
IG_HD u64 mulw_digit(u32 a, const Tw& t) {
  const u64 lo = (u64)a * t.l;
  const u64 hi = mad_wide(a, t.h, lo >> 32);
  return mad_wide((u32)(hi >> 29), 32766u, (((u64)((u32)hi & 0x1fffffffu)) << 32) | (u32)lo);
}

// x mod q in [0, 2^60 + 2^18) for any 64-bit x: 2^60 = 2^14 - 1 (mod q).
IG_HD u64 red60(u64 x) {
  const u32 h = (u32)(x >> 32);
  return mad_wide(h >> 28, 16383u, ((u64)(h & 0x0fffffffu) << 32) | (u32)x);
}
// x mod q, canonical, for any 64-bit x. r = red60(x) is at or above q exactly when r + 2^14 - 1
// reaches 2^60, and its low 60 bits are then r - q.
IG_HD u64 canon(u64 x) {
  const u64 r = red60(x), u = r + 16383u;
  return u >> 60 ? u & MASK60 : r;
}

// A 128-bit sum of products of 64-bit words, as four words: mac adds a * b (four wide multiplies
// with their carries), acc_fold gives the sum mod q.
struct Acc {
  u32 r0, r1, r2, r3;
};
IG_HD Acc acc_from(u64 x) { return Acc{(u32)x, (u32)(x >> 32), 0, 0}; }
IG_HD void mac(Acc& s, u64 a, u64 b) {
#ifdef __CUDA_ARCH__
  asm("mad.lo.cc.u32 %0,%4,%6,%0; madc.hi.cc.u32 %1,%4,%6,%1; madc.lo.cc.u32 %2,%5,%7,%2; madc.hi.u32 %3,%5,%7,%3;\n"
      "mad.lo.cc.u32 %1,%4,%7,%1; madc.hi.cc.u32 %2,%4,%7,%2; addc.u32 %3,%3,0;\n"
      "mad.lo.cc.u32 %1,%5,%6,%1; madc.hi.cc.u32 %2,%5,%6,%2; addc.u32 %3,%3,0;"
      : "+r"(s.r0), "+r"(s.r1), "+r"(s.r2), "+r"(s.r3)
      : "r"((u32)a), "r"((u32)(a >> 32)), "r"((u32)b), "r"((u32)(b >> 32)));
#else
  u128 v = ((u128)(((u64)s.r3 << 32) | s.r2) << 64) | (((u64)s.r1 << 32) | s.r0);
  v += (u128)a * b;
  s = Acc{(u32)v, (u32)(v >> 32), (u32)(v >> 64), (u32)(v >> 96)};
#endif
}
// The sum mod q in [0, 2^60 + 2^37), for any sum below 2^128: 2^64 = 2^18 - 16 brings the two high
// words down to 83 bits, 2^60 = 2^14 - 1 the rest. Three wide multiplies, where a Montgomery
// reduction takes five wide, two low ones and its conditional subtractions.
IG_HD u64 acc_fold(const Acc& s) {
  const u64 p0 = mad_wide(s.r2, 262128u, (u64)s.r0);
  const u64 p1 = mad_wide(s.r3, 262128u, (u64)s.r1 + (p0 >> 32));
  return mad_wide((u32)(p1 >> 28), 16383u, ((p1 & 0x0fffffffu) << 32) | (u32)p0);
}
IG_HD u64 mulq(u64 a, u64 b) {
  Acc s{0, 0, 0, 0};
  mac(s, a, b);
  return acc_fold(s);
}

// x mod q for any 128-bit x, using 2^60 == 2^14 - 1 (mod q).
IG_HD u64 reduce128(u128 x) {
  const u128 M60 = (((u128)1) << 60) - 1;
  x = (x >> 60) * ((((u128)1) << 14) - 1) + (x & M60);  // < 2^83
  x = (x >> 60) * ((((u128)1) << 14) - 1) + (x & M60);  // < 2^61
  u64 r = (u64)x;
  r = csub(r);
  return csub(r);
}

// ChaCha20 block (RFC 7539 quarter rounds, 64-bit counter in words 12-13 and 64-bit
// stream id in words 14-15), the keystream rand_chacha's ChaCha20Rng draws from.
IG_HD u32 rotl(u32 x, int r) { return (x << r) | (x >> (32 - r)); }

IG_HD void chacha20_block(const u32 key[8], u64 counter, u64 stream, u32 out[16]) {
  u32 s[16] = {0x61707865u, 0x3320646eu, 0x79622d32u, 0x6b206574u, key[0], key[1], key[2], key[3],
               key[4], key[5], key[6], key[7], (u32)counter, (u32)(counter >> 32), (u32)stream,
               (u32)(stream >> 32)};
  u32 x[16];
#pragma unroll
  for (int i = 0; i < 16; i++) x[i] = s[i];
#define IG_QR(a, b, c, d)                      \
  x[a] += x[b]; x[d] = rotl(x[d] ^ x[a], 16); \
  x[c] += x[d]; x[b] = rotl(x[b] ^ x[c], 12); \
  x[a] += x[b]; x[d] = rotl(x[d] ^ x[a], 8);  \
  x[c] += x[d]; x[b] = rotl(x[b] ^ x[c], 7);
#pragma unroll
  for (int i = 0; i < 10; i++) {
    IG_QR(0, 4, 8, 12) IG_QR(1, 5, 9, 13) IG_QR(2, 6, 10, 14) IG_QR(3, 7, 11, 15)
    IG_QR(0, 5, 10, 15) IG_QR(1, 6, 11, 12) IG_QR(2, 7, 8, 13) IG_QR(3, 4, 9, 14)
  }
#undef IG_QR
#pragma unroll
  for (int i = 0; i < 16; i++) out[i] = x[i] + s[i];
}

// rand 0.8 gen_range(0..q) acceptance for u64: v * q = hi:lo, accept when lo <= zone,
// zone = (q << clz(q)) - 1.
static constexpr u64 RANGE_ZONE = (Q << 4) - 1;

// ------------------------------------------------------------------------------------
// Shoup products and the Montgomery reduction of sums that the recursions took before mulw and Acc: no kernel calls them,
// tests/arith_bounds.cpp checks their bounds.

// q held in a register the compiler cannot see through, so est * q issues as an integer
// multiply (FMA pipe) rather than shifts and adds (ALU pipe).
IG_HD u64 q_opaque() {
#ifdef __CUDA_ARCH__
  u64 r;
  asm("mov.b64 %0, %1;" : "=l"(r) : "l"(Q));
  return r;
#else
  return Q;
#endif
}

IG_HD u32 mulhi32(u32 a, u32 b) {
#ifdef __CUDA_ARCH__
  return __umulhi(a, b);
#else
  return (u32)(((u64)a * b) >> 32);
#endif
}

// a * w mod q up to three q: in [0, 4q) for any a < 2^64. The quotient estimate takes the
// high word of a * w' from three of its four 32-bit partial products: the high one whole
// and the high halves of the two middle ones; the low one is dropped. The three dropped
// fractions are each below one unit, so the estimate undershoots floor(a w' / 2^64) by
// at most 2, and a w - est q exceeds the exact Shoup remainder (below 2q) by at most 2q.
IG_HD u64 shoup_lazy4(u64 a, u64 w, u64 wp) {
  const u32 ah = (u32)(a >> 32), al = (u32)a, wh = (u32)(wp >> 32), wl = (u32)wp;
  const u64 est = (u64)ah * wh + mulhi32(ah, wl) + mulhi32(al, wh);
  return a * w - est * q_opaque();
}

// a * w mod q up to three q for a below 2^32 (a gadget digit). The quotient estimate is
// floor(a wh / 2^32), wh the high word of w'; the exact floor(a w' / 2^64) adds a wl / 2^64
// (below one unit, wl the low word) to a wh / 2^32, so the estimate undershoots it by at
// most 1 and a w - est q lies in [0, 3q).
IG_HD u64 shoup_digit(u32 a, u64 w, u64 wp) {
  const u64 est = mulhi32(a, (u32)(wp >> 32));
  return (u64)a * w - est * q_opaque();
}

// x - 2q when x >= 2q.
IG_HD u64 csub2(u64 x) { return x >= 2 * Q ? x - 2 * Q : x; }
// x - 4q when x >= 4q.
IG_HD u64 csub4(u64 x) { return x >= 4 * Q ? x - 4 * Q : x; }

// Montgomery reduction of a 128-bit sum of products, x * 2^-64 mod q for x < 2q * 2^64 (sums of products whose factors
// run up to 8q, such as transforms kept below 8q times words below q): the quotient lands below 3q.
IG_HD u64 redc_wide(u128 x) {
  const u64 lo = (u64)x, hi = (u64)(x >> 64);
  const u64 m = lo * QINV_NEG;
  return csub(csub2(hi + mulhi(m, Q) + (lo != 0 ? 1 : 0)));
}

// Shoup companion floor(w * 2^64 / q).
IG_HD u64 shoup_companion(u64 w) { return (u64)(((u128)w << 64) / Q); }

}  // namespace ig
